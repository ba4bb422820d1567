"""Workloads by which the speed of the framework is measured, with their inputs, results in 64 bits and tolerances.

Training: the MNIST-shaped classifier, GPT-2 small and Llama-7B layers through ``Trainer.step``, and attention by itself
with the options that a transformer block turns on.  Serving: the INT4 Llama engine (prompts, the verify pass and the
draft pass of speculative decoding, sampling), and the layer-stack engine (Surelorn decoding, Nufalorn prompts, a mixture
of experts).  One pass is one call that a user makes; decode passes of the INT4 engine are CUDA-graph replays of
``LlamaInt4Engine.forward``, which is how ``SpeculativeDecoder`` runs them.
"""
import copy
import functools
import math

import torch

BF, F32, F64 = torch.bfloat16, torch.float32, torch.float64
SCALE = 65536.0                          # loss scale at the start of training
GPT2 = dict(vocab=50304, layers=12, width=768, heads=12, ff=3072, context=2048)
LLAMA = dict(vocab=32000, layers=2, width=4096, heads=32, kv_heads=8, ff=11008, context=4096)   # two layers of the 7B shape
SURELORN = dict(vocab=32000, width=2048, layers=4, heads=16, dim=128, q_rank=768, kv_rank=512, ff=5632)
NUFALORN = dict(vocab=32000, width=2048, heads=16, kv_heads=4, dim=128, ff=5632, rank=32, kinds=("gla", "attention", "hgrn2", "gla"),
                block=4096, base=5e5, mult=0.8, cap=40.0, eps=1e-5, tau=8.0)
EXPERTS = dict(width=2048, experts=64, top=6, ff=1408, shared=2816, groups=8, keep=4, eps=1e-6)
TABLE = 16.0                             # token table of the served Llama: a layer adds about a tenth to the stream
EPS = 1e-5                               # norms of GPT-2 and Llama


def listed():
    return [
        # one optimizer step of the 784-512-512-10 classifier at its benchmark's batch: small kernels, launches count
        {"name": "mlp_step", "kind": "mlp", "batch": 256},
        # the headline training step: GPT-2 small, global batch 64 x 2048
        {"name": "gpt2_step", "kind": "gpt2", "batch": 64, "seq": 2048},
        # the same model fine-tuned on short odd-length text: a few thousand tokens a step, no size a multiple of a tile
        {"name": "gpt2_step_ragged", "kind": "gpt2", "batch": 5, "seq": 1111},
        # a pipeline stage of the 7B configuration: layers of width 4096 with grouped queries, micro-batch 1 x 4096
        {"name": "llama_step", "kind": "llama", "batch": 1, "seq": 4096},
        # attention of a block with a sliding window and position biases, forward and backward, odd length
        {"name": "attention_window", "kind": "attention", "batch": 2, "seq": 3001, "heads": 32, "kv_heads": 8, "dim": 128, "causal": True,
         "window": 1024, "alibi": True},
        # serving: 16 prompts of 512 tokens into the INT4 cache
        {"name": "int4_prompt", "kind": "int4_prompt", "batch": 16, "seq": 511},
        # the verify pass of speculative decoding: 16 sequences, 4 drafted tokens and the last one
        {"name": "int4_verify", "kind": "int4_decode", "batch": 16, "history": 640, "tokens": 5},
        # one drafted token for each of the 16 sequences (the draft model has two layers of this width)
        {"name": "int4_draft", "kind": "int4_decode", "batch": 16, "history": 640, "tokens": 1},
        # the distributions and tokens of a verify pass: temperature 0.8, top-k 50, top-p 0.9
        {"name": "sample_verify", "kind": "sample", "rows": 80, "vocab": 32000, "temperature": 0.8, "top_k": 50, "top_p": 0.9},
        # one decode step of 32 running requests of different lengths
        {"name": "surelorn_decode", "kind": "surelorn_decode", "batch": 32, "context": 1000},
        # two prompts of different lengths arriving together
        {"name": "nufalorn_prompt", "kind": "nufalorn_prompt", "batch": 2, "seq": 1900},
        # a mixture-of-experts layer over one step's prompt tokens
        {"name": "experts_prompt", "kind": "experts", "tokens": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mlp", "gpt2", "llama", "attention", "int4_prompt", "int4_decode", "int4_decode", "sample", "surelorn_decode", "nufalorn_prompt", "experts"])
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 32, 4096)}
    if kind == "gpt2":
        seq = _log(rng, 128, 2048)
        return {"kind": kind, "batch": max(1, _log(rng, 512, 32768) // seq), "seq": seq}
    if kind == "llama":
        return {"kind": kind, "batch": 1, "seq": _log(rng, 256, 4096)}
    if kind == "attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (12, 12, 64), (16, 4, 128), (8, 1, 64)])
        return {"kind": kind, "batch": rng.randint(1, 3), "seq": _log(rng, 130, 4096), "heads": heads, "kv_heads": kv_heads, "dim": dim,
                "causal": rng.random() < 0.8, "window": rng.choice([-1, -1, 255, 1024]), "alibi": rng.random() < 0.3}
    if kind == "int4_prompt":
        return {"kind": kind, "batch": rng.randint(1, 16), "seq": _log(rng, 32, 512)}
    if kind == "int4_decode":
        return {"kind": kind, "batch": rng.randint(1, 16), "history": _log(rng, 16, 2000), "tokens": rng.choice([1, 1, 3, 5, 8])}
    if kind == "sample":
        k, p = rng.choice([(50, 0.9), (50, 1.0), (0, 0.9), (200, 0.95), (1, 1.0)])
        return {"kind": kind, "rows": rng.randint(1, 128), "vocab": rng.choice([32000, 50304, 50257]), "temperature": rng.choice([0.7, 0.8, 1.0]), "top_k": k, "top_p": p}
    if kind == "surelorn_decode":
        return {"kind": kind, "batch": rng.randint(1, 64), "context": _log(rng, 100, 2000)}
    if kind == "nufalorn_prompt":
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": _log(rng, 64, 2048)}
    return {"kind": kind, "tokens": _log(rng, 32, 4096)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _ids(g, vocab, *shape):
    return torch.randint(0, vocab, shape, generator=g, device="cuda")


def _gpt2_shapes(m):
    W, F = m["width"], m["ff"]
    out = [("wte", (m["vocab"], W)), ("wpe", (m["context"], W))]
    for i in range(m["layers"]):
        out += [(f"{i}.norm1.w", (W,)), (f"{i}.norm1.b", (W,)), (f"{i}.qkv.w", (3 * W, W)), (f"{i}.qkv.b", (3 * W,)), (f"{i}.proj.w", (W, W)), (f"{i}.proj.b", (W,)),
                (f"{i}.norm2.w", (W,)), (f"{i}.norm2.b", (W,)), (f"{i}.up.w", (F, W)), (f"{i}.up.b", (F,)), (f"{i}.down.w", (W, F)), (f"{i}.down.b", (W,))]
    return out + [("norm.w", (W,)), ("norm.b", (W,))]


def _llama_shapes(m):
    W, F, D = m["width"], m["ff"], m["width"] // m["heads"]
    out = [("wte", (m["vocab"], W))]
    for i in range(m["layers"]):
        out += [(f"{i}.norm1.w", (W,)), (f"{i}.qkv.w", ((m["heads"] + 2 * m["kv_heads"]) * D, W)), (f"{i}.proj.w", (W, W)),
                (f"{i}.norm2.w", (W,)), (f"{i}.gate_up.w", (2 * F, W)), (f"{i}.down.w", (W, F))]
    return out + [("norm.w", (W,)), ("head.w", (m["vocab"], W))]


def _mlp_shapes():
    dims = (784, 512, 512, 10)
    return [p for i, (a, b) in enumerate(zip(dims, dims[1:])) for p in ((f"{i}.w", (b, a)), (f"{i}.b", (b,)))]


def _weights(shapes, g, table=0.02):
    """bf16 values as training meets them: matrices N(0, 0.02) (the classifier's N(0, 2 / in)), norm weights around 1, biases around 0.
    table: standard deviation of the token table."""
    out = {}
    for name, shape in shapes:
        std = table if name == "wte" else 0.02 if shape[-1] not in (784, 512) else (2.0 / shape[-1]) ** 0.5
        t = _randn(g, *shape, std=0.02 if len(shape) == 1 else std, dtype=F32)
        out[name] = (t + 1.0 if "norm" in name and name.endswith(".w") else t).to(BF)
    return out


@functools.lru_cache(maxsize=None)
def _template(kind):
    """The model without values (its own initial weights are drawn on the host, which takes seconds at these sizes)."""
    if kind == "mlp":
        from cogito_b200.models.mlp import MLPClassifier
        return MLPClassifier(784, (512, 512), 10, device="meta", dtype=BF)
    if kind == "gpt2":
        from cogito_b200.models.gpt2 import GPT2 as Model, GPT2Config
        m = GPT2
        return Model(GPT2Config(m["vocab"], m["layers"], m["width"], m["heads"], m["ff"], m["context"], norm_eps=EPS), device="meta", dtype=BF)
    from cogito_b200.models.llama import Llama, LlamaConfig
    m = LLAMA
    return Llama(LlamaConfig(m["vocab"], m["layers"], m["width"], m["heads"], m["kv_heads"], m["ff"], m["context"], norm_eps=EPS), device="meta", dtype=BF)


def _model(kind, weights):
    model = copy.deepcopy(_template(kind)).to_empty(device="cuda")
    params = list(model.parameters())
    assert [tuple(p.shape) for p in params] == [tuple(w.shape) for w in weights.values()]
    with torch.no_grad():
        for p, w in zip(params, weights.values()):
            p.copy_(w)
    return model


SHAPES = {"mlp": _mlp_shapes, "gpt2": lambda: _gpt2_shapes(GPT2), "llama": lambda: _llama_shapes(LLAMA)}
RATE = {"mlp": 1e-3, "gpt2": 3e-4, "llama": 3e-4}


def _batch(case, g):
    if case["kind"] == "mlp":
        return torch.rand(case["batch"], 784, generator=g, device="cuda"), torch.randint(0, 10, (case["batch"],), generator=g, device="cuda")
    vocab = (GPT2 if case["kind"] == "gpt2" else LLAMA)["vocab"]
    return _ids(g, vocab, case["batch"], case["seq"]), _ids(g, vocab, case["batch"], case["seq"])


def _attention_inputs(case, g):
    B, T, H, G, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim"))
    return [_randn(g, B, T, h, D) for h in (H, G, G, H)]


def _surelorn_tensors(g):
    m = SURELORN
    W, H, d = m["width"], m["heads"], m["dim"]
    out = {}
    mat = lambda name, o, i: out.update({name: _randn(g, o, i, std=i ** -0.5)})
    vec = lambda name, n: out.update({name: _randn(g, n, std=0.1, dtype=F32).add_(1.0).to(BF)})
    out["embed"] = _randn(g, m["vocab"], W)
    for i in range(m["layers"]):
        p = f"l{i}."
        vec(p + "norm1", W), vec(p + "norm2", W), vec(p + "mix.dq.norm", m["q_rank"]), vec(p + "mix.dkv.norm", m["kv_rank"])
        mat(p + "mix.dq", m["q_rank"], W), mat(p + "mix.uq", H * d, m["q_rank"]), mat(p + "mix.dkv", m["kv_rank"], W)
        mat(p + "mix.uk", H * d, m["kv_rank"]), mat(p + "mix.uv", H * d, m["kv_rank"]), mat(p + "mix.o", W, H * d)
        mat(p + "mlp.gate", m["ff"], W), mat(p + "mlp.up", m["ff"], W), mat(p + "mlp.down", W, m["ff"])
    vec("final.norm", W), mat("head", m["vocab"], W)
    return out


def _nufalorn_tensors(g):
    m = NUFALORN
    W, H, d, G = m["width"], m["heads"], m["dim"], m["kv_heads"]
    out = {}
    mat = lambda name, o, i: out.update({name: _randn(g, o, i, std=i ** -0.5)})
    vec = lambda name, n, std=0.2, mean=0.0: out.update({name: (_randn(g, n, std=std, dtype=F32) + mean).to(BF)})
    out["embed"] = _randn(g, m["vocab"], W)
    for i, kind in enumerate(m["kinds"]):
        p = f"l{i}."
        vec(p + "norm1", W), vec(p + "norm2", W)
        mat(p + "mix.q", H * d, W), mat(p + "mix.o", W, H * d)
        mat(p + "mix.v", (G if kind == "attention" else H) * d, W)
        if kind != "hgrn2":
            mat(p + "mix.k", (G if kind == "attention" else H) * d, W)
        if kind != "attention":
            vec(p + "mix.norm", d, mean=1.0)
        if kind == "gla":
            mat(p + "mix.g", H * d, W), mat(p + "mix.a1", m["rank"], W), mat(p + "mix.a2", H * d, m["rank"]), vec(p + "mix.a2.b", H * d, 2.0, 2.0)
        if kind == "hgrn2":
            mat(p + "mix.f", H * d, W), vec(p + "mix.f.b", H * d, 2.0, 2.0)
            out[p + "mix.lower"] = (0.9 * torch.rand(H * d, generator=g, device="cuda")).to(BF)
        mat(p + "mlp.gate", m["ff"], W), mat(p + "mlp.up", m["ff"], W), mat(p + "mlp.down", W, m["ff"])
    vec("final.norm", W), mat("head", m["vocab"], W)
    return out


def _expert_inputs(case, g):
    m, t = EXPERTS, {}
    W, F = m["width"], m["ff"]
    for e in range(m["experts"]):
        t[f"e{e}.gate"], t[f"e{e}.up"], t[f"e{e}.down"] = _randn(g, F, W, std=W ** -0.5), _randn(g, F, W, std=W ** -0.5), _randn(g, W, F, std=F ** -0.5)
    t["router"], t["correction"] = _randn(g, m["experts"], W, std=W ** -0.5), _randn(g, m["experts"], std=0.02)
    t["shared.gate"], t["shared.up"], t["shared.down"] = (_randn(g, *s, std=s[1] ** -0.5) for s in ((m["shared"], W), (m["shared"], W), (W, m["shared"])))
    x, w = _randn(g, case["tokens"], W, dtype=F32), _randn(g, W, std=0.1, dtype=F32) + 1.0
    return t, x, w


def _contexts(case, g):
    """Token lists of the running requests: up to a quarter shorter than the longest."""
    C = case["context"]
    return [_ids(g, SURELORN["vocab"], C - (C // 4) * i // max(1, case["batch"] - 1)).tolist() for i in range(case["batch"])]


def _prompts(case, g):
    return [_ids(g, NUFALORN["vocab"], case["seq"] - (case["seq"] // 5) * i // max(1, case["batch"] - 1)).tolist() for i in range(case["batch"])]


def _served_weights(g):
    """As a trained model has them: the tokens carry most of the residual stream, so that the rounding to 4 bits is not amplified from layer to layer."""
    return _weights(_llama_shapes(LLAMA), g, table=TABLE)


def _int4_engine(case, g, room):
    from cogito_b200.serve.engine import LlamaInt4Engine
    return LlamaInt4Engine(_model("llama", _served_weights(g)), case["batch"], max_seq_len=room)


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in SHAPES:
        from cogito_b200.optim.fused import FusedAdam, GradScaler
        from cogito_b200.train import Trainer
        model = _model(kind, _weights(SHAPES[kind](), g))
        opt = FusedAdam(model.parameters(), lr=RATE[kind], scaler=GradScaler("cuda", init_scale=SCALE))
        x, y = _batch(case, g)
        return {"kind": kind, "trainer": Trainer(model, opt), "opt": opt, "x": x, "y": y}
    if kind == "attention":
        from cogito_b200.ops.attention import alibi_slopes
        q, k, v, do = _attention_inputs(case, g)
        return {"kind": kind, "q": q.requires_grad_(), "k": k.requires_grad_(), "v": v.requires_grad_(), "do": do, "causal": case["causal"],
                "window": case["window"], "alibi": alibi_slopes(case["heads"], "cuda") if case["alibi"] else None}
    if kind == "int4_prompt":
        engine = _int4_engine(case, g, case["seq"] + 257)
        return {"kind": kind, "engine": engine, "ids": _ids(g, LLAMA["vocab"], case["batch"], case["seq"])}
    if kind == "int4_decode":
        engine = _int4_engine(case, g, case["history"] + 257)
        engine.forward(_ids(g, LLAMA["vocab"], case["batch"], case["history"]), commit=True)
        tokens = _ids(g, LLAMA["vocab"], case["batch"], case["tokens"])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                engine.forward(tokens)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            logits = engine.forward(tokens)
        return {"kind": kind, "engine": engine, "graph": graph, "tokens": tokens, "logits": logits}
    if kind == "sample":
        return {"kind": kind, "logits": _randn(g, case["rows"], case["vocab"], std=2.0, dtype=F32), "step": torch.tensor([seed], device="cuda"),
                "how": {k: case[k] for k in ("temperature", "top_k", "top_p")}}
    if kind == "surelorn_decode":
        from cogito_b200.models.surelorn import Surelorn, SurelornConfig
        from cogito_b200.serve.stack import StackEngine
        m = SURELORN
        mixer = {"heads": m["heads"], "dim": m["dim"], "vdim": m["dim"], "q_rank": m["q_rank"], "kv_rank": m["kv_rank"], "scale": m["dim"] ** -0.5}
        layer = {"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": m["ff"]}}
        cfg = SurelornConfig.from_dict({"vocab": m["vocab"], "width": m["width"], "embedding": {"scale": m["width"] ** 0.5}, "norm": {"eps": 1e-6},
                                        "layers": [layer] * m["layers"]})
        engine = StackEngine(Surelorn(cfg, _surelorn_tensors(g), "cuda", BF), case["batch"], case["context"] + 256, pool_tokens=case["batch"] * (case["context"] + 64))
        contexts = _contexts(case, g)
        for c in contexts:
            engine.step([(engine.open(), c, [])])
        slots = sorted(engine.cached, key=lambda s: -engine.cached[s])
        tokens = _ids(g, m["vocab"], case["batch"]).tolist()
        state = {"kind": kind, "engine": engine, "entries": [(s, [t], [0]) for s, t in zip(slots, tokens)], "cached": dict(engine.cached)}
        run(state)                       # the engine keeps a decode graph by batch size: a serving program has it
        return state
    if kind == "nufalorn_prompt":
        from cogito_b200.models.nufalorn import Nufalorn, NufalornConfig
        from cogito_b200.serve.stack import StackEngine
        m = NUFALORN
        H, d = m["heads"], m["dim"]
        mixers = {"attention": {"heads": H, "kv_heads": m["kv_heads"], "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": m["block"]}, "rot": {"base": m["base"], "dims": d}},
                  "hgrn2": {"heads": H, "dim": d, "vdim": d}, "gla": {"heads": H, "dim": d, "vdim": d, "tau": m["tau"], "a_rank": m["rank"]}}
        cfg = NufalornConfig.from_dict({"vocab": m["vocab"], "width": m["width"], "residual_mult": m["mult"], "logit_softcap": m["cap"], "norm": {"eps": m["eps"]},
                                        "layers": [{"type": k, "mixer": mixers[k], "mlp": {"kind": "dense", "ff": m["ff"]}} for k in m["kinds"]]})
        engine = StackEngine(Nufalorn(cfg, _nufalorn_tensors(g), "cuda", BF), case["batch"], case["seq"] + 256, pool_tokens=case["batch"] * (case["seq"] + 64))
        return {"kind": kind, "engine": engine, "prompts": _prompts(case, g)}
    from cogito_b200.nn.moe import MixtureOfExperts, MoESpec
    m = EXPERTS
    t, x, w = _expert_inputs(case, g)
    spec = MoESpec(m["ff"], m["experts"], m["top"], groups=m["groups"], keep=m["keep"], shared_ff=m["shared"])
    return {"kind": kind, "layer": MixtureOfExperts(spec, t, "cuda", BF), "x": x, "h": x.to(BF), "w": w}


def run(state):
    kind = state["kind"]
    if kind in SHAPES:
        loss = state["trainer"].step(state["x"], state["y"])
        return {"loss": loss, "gradients": state["opt"].grad, "weights": state["opt"].fp.flat}
    if kind == "attention":
        from cogito_b200.ops.attention import flash_attention
        q, k, v = state["q"], state["k"], state["v"]
        o = flash_attention(q, k, v, causal=state["causal"], window=state["window"], alibi=state["alibi"])
        return (o.detach(),) + torch.autograd.grad(o, (q, k, v), state["do"])
    if kind == "int4_prompt":
        state["engine"].reset()
        return state["engine"].forward(state["ids"], commit=True)
    if kind == "int4_decode":
        state["graph"].replay()
        return state["logits"]
    if kind == "sample":
        from cogito_b200.serve.sampling import sample
        return sample(state["logits"], seed=7, step=state["step"], return_probs=True, **state["how"])
    if kind == "surelorn_decode":
        logits = state["engine"].step(state["entries"])
        state["engine"].cached.update(state["cached"])          # the step's tokens are taken back
        return logits
    if kind == "nufalorn_prompt":
        engine = state["engine"]
        slots = [engine.open() for _ in state["prompts"]]
        logits = engine.step([(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])
        for s in slots:
            engine.close(s)
        return logits
    from cogito_b200.ops.stream import stream_update
    with torch.no_grad():
        y, pairs = state["layer"].branch(state["h"])
        return stream_update(state["x"], y, state["w"], EXPERTS["eps"], BF, **pairs), state["x"]


# ------------------------------------------------------------------ work
def _pairs(T, causal, window):
    """Query-key pairs that see each other."""
    if window < 0:
        return T * (T + 1) // 2 if causal else T * T
    w = min(window, T - 1)
    half = T * (w + 1) - w * (w + 1) // 2
    return half if causal else 2 * half - T


def work(case):
    kind = case["kind"]
    if kind in SHAPES:
        sizes = {n: math.prod(s) for n, s in SHAPES[kind]()}
        total = sum(sizes.values())
        rows = case["batch"] * case.get("seq", 1)
        used = total - (0 if kind == "mlp" else sum(v for n, v in sizes.items() if n == "wpe" or (n == "wte" and kind == "llama")))   # the tied table is the head
        flops = 6.0 * rows * used
        if kind != "mlp":
            m = GPT2 if kind == "gpt2" else LLAMA
            flops += 12.0 * m["layers"] * m["width"] * case["batch"] * _pairs(case["seq"], True, -1)
        return {"bytes": 30.0 * total + rows * (16 if kind != "mlp" else 784 * 4 + 8), "flops": flops}
    if kind == "attention":
        B, T, H, G, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim"))
        return {"bytes": 2.0 * B * T * D * (4 * H + 4 * G), "flops": 14.0 * D * B * H * _pairs(T, case["causal"], case["window"])}
    if kind in ("int4_prompt", "int4_decode"):
        m = LLAMA
        weights = sum(math.prod(s) for n, s in _llama_shapes(m) if n.endswith(".w") and len(s) == 2)
        B, new, past = case["batch"], case.get("seq", case.get("tokens")), case.get("history", 0)
        rows, D = B * new, m["width"] // m["heads"]
        kv = m["layers"] * 2 * m["kv_heads"] * D * (0.5 + 4 / 32)
        flops = 2.0 * rows * weights + 4.0 * m["layers"] * m["width"] * B * (new * past + _pairs(new, True, -1))
        return {"bytes": weights * (0.5 + 4 / 128) + B * (past + new) * kv + rows * (2 * m["width"] + 4 * m["vocab"]), "flops": flops}
    if kind == "sample":
        return {"bytes": 8.0 * case["rows"] * case["vocab"], "flops": 4.0 * case["rows"] * case["vocab"]}
    if kind == "surelorn_decode":
        m = SURELORN
        W, H, d = m["width"], m["heads"], m["dim"]
        layer = W * (m["q_rank"] + m["kv_rank"] + H * d + 3 * m["ff"]) + H * d * (m["q_rank"] + 2 * m["kv_rank"])
        weights = m["layers"] * layer + m["vocab"] * W
        context = sum(case["context"] - (case["context"] // 4) * i // max(1, case["batch"] - 1) + 1 for i in range(case["batch"]))
        return {"bytes": 2.0 * weights + 2.0 * m["layers"] * m["kv_rank"] * context + case["batch"] * (2 * W + 4 * m["vocab"]),
                "flops": 2.0 * case["batch"] * weights + 4.0 * m["layers"] * context * H * m["kv_rank"]}
    if kind == "nufalorn_prompt":
        m = NUFALORN
        W, H, d, G = m["width"], m["heads"], m["dim"], m["kv_heads"]
        lengths = [case["seq"] - (case["seq"] // 5) * i // max(1, case["batch"] - 1) for i in range(case["batch"])]
        per = {"attention": W * (2 * H + 2 * G) * d, "hgrn2": W * 4 * H * d, "gla": W * (5 * H * d + m["rank"]) + m["rank"] * H * d}
        layers = sum(per[k] + 3 * W * m["ff"] for k in m["kinds"])
        n, flops = sum(lengths), 2.0 * case["batch"] * W * m["vocab"]
        flops += 2.0 * n * layers + sum(4.0 * H * d * _pairs(t, True, -1) for t in lengths) * m["kinds"].count("attention")
        flops += 4.0 * n * H * d * d * (len(m["kinds"]) - m["kinds"].count("attention"))
        return {"bytes": 2.0 * (layers + m["vocab"] * W) + 2.0 * n * W + 4.0 * case["batch"] * m["vocab"], "flops": flops}
    m, n = EXPERTS, case["tokens"]
    used = min(m["experts"], n * m["top"])
    return {"bytes": 2.0 * m["width"] * (3 * used * m["ff"] + 3 * m["shared"] + m["experts"]) + n * m["width"] * 12,
            "flops": 2.0 * n * m["width"] * (3 * m["top"] * m["ff"] + 3 * m["shared"] + m["experts"])}


# ------------------------------------------------------------------ results in 64 bits
def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope(x, base):
    """[.., T, D]: element i turns with element i + D / 2 by position * base^(-2 i / D)."""
    T, D = x.shape[-2:]
    a = torch.arange(T, device=x.device, dtype=F64)[:, None] * base ** (-torch.arange(D // 2, device=x.device, dtype=F64) * 2 / D)
    u, v = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _softmax_attention(q, k, v, scale, first=0):
    """q [.., t, D] at positions first.., k and v [.., T, D]: causal."""
    s = q @ k.transpose(-1, -2) * scale
    hide = torch.arange(k.shape[-2], device=q.device)[None] > first + torch.arange(q.shape[-2], device=q.device)[:, None]
    return torch.softmax(s.masked_fill(hide, float("-inf")), -1) @ v


def _linear(x, w, i, name):
    y = x @ w[f"{i}.{name}.w"].T
    return y + w[f"{i}.{name}.b"] if f"{i}.{name}.b" in w else y


def _gpt2_loss(w, ids, targets):
    m, F = GPT2, torch.nn.functional
    H, W = m["heads"], m["width"]
    T = ids.shape[0]
    x = w["wte"][ids] + w["wpe"][:T]
    for i in range(m["layers"]):
        h = F.layer_norm(x, (W,), w[f"{i}.norm1.w"], w[f"{i}.norm1.b"], EPS)
        q, k, v = _linear(h, w, i, "qkv").view(T, 3, H, W // H).permute(1, 2, 0, 3)
        x = x + _linear(_softmax_attention(q, k, v, (W // H) ** -0.5).transpose(0, 1).reshape(T, W), w, i, "proj")
        h = F.layer_norm(x, (W,), w[f"{i}.norm2.w"], w[f"{i}.norm2.b"], EPS)
        x = x + _linear(F.gelu(_linear(h, w, i, "up"), approximate="tanh"), w, i, "down")
    logits = F.layer_norm(x, (W,), w["norm.w"], w["norm.b"], EPS) @ w["wte"].T
    return F.cross_entropy(logits, targets, reduction="sum")


def _llama_hidden(w, ids, cached=None, first=0):
    """ids [T]; cached: what keys and values become in the cache; first: rows before it only serve as history."""
    m, F = LLAMA, torch.nn.functional
    H, G, W, T = m["heads"], m["kv_heads"], m["width"], ids.shape[0]
    D = W // H
    x = w["wte"][ids]
    for i in range(m["layers"]):
        qkv = _linear(_rms(x, w[f"{i}.norm1.w"], EPS), w, i, "qkv").view(T, H + 2 * G, D).transpose(0, 1)
        qk = _rope(qkv[:H + G], 10000.0)
        q, k, v = qk[:H], qk[H:], qkv[H + G:]
        if cached is not None:
            k, v = cached(k), cached(v)
        o = _softmax_attention(q, k.repeat_interleave(H // G, 0), v.repeat_interleave(H // G, 0), D ** -0.5)
        x = x + _linear(o.transpose(0, 1).reshape(T, W), w, i, "proj")
        gate, up = _linear(_rms(x, w[f"{i}.norm2.w"], EPS), w, i, "gate_up").chunk(2, -1)
        x = x + _linear(F.silu(gate) * up, w, i, "down")
    return _rms(x[first:], w["norm.w"], EPS)


def _llama_loss(w, ids, targets):
    return torch.nn.functional.cross_entropy(_llama_hidden(w, ids) @ w["head.w"].T, targets, reduction="sum")


def _mlp_loss(w, x, targets):
    h = x.to(BF).double()
    for i in range(3):
        h = h @ w[f"{i}.w"].T + w[f"{i}.b"]
        h = torch.relu(h) if i < 2 else h
    return torch.nn.functional.cross_entropy(h, targets, reduction="sum")


def _flat(values):
    """One vector, every tensor padded to a multiple of 8 values."""
    return torch.cat([torch.nn.functional.pad(t.reshape(-1), (0, -t.numel() % 8)) for t in values])


def _exact_step(case, g):
    kind = case["kind"]
    w = {n: t.double().requires_grad_() for n, t in _weights(SHAPES[kind](), g).items()}
    x, y = _batch(case, g)
    parts = [(x, y)] if kind == "mlp" else list(zip(x, y))
    loss_of = {"mlp": _mlp_loss, "gpt2": _gpt2_loss, "llama": _llama_loss}[kind]
    total = 0.0
    for a, b in parts:
        loss = loss_of(w, a, b) / y.numel()
        loss.backward()
        total += float(loss.detach())
    grads = [t.grad if t.grad is not None else torch.zeros_like(t) for t in w.values()]
    flat, p = _flat(grads), _flat([t.detach() for t in w.values()])
    return {"loss": torch.tensor(total, dtype=F64), "gradients": flat * SCALE, "weights": p - RATE[kind] * flat / (flat.abs() + 1e-8)}


def _exact_attention(case, g):
    q, k, v, do = (t.double() for t in _attention_inputs(case, g))
    B, T, H, G, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "dim"))
    at = torch.arange(T, device="cuda")
    far = at[None] - at[:, None]
    hide = (far > 0) if case["causal"] else torch.zeros_like(far, dtype=torch.bool)
    if case["window"] >= 0:
        hide = hide | (far.abs() > case["window"])
    o, dq, dk, dv = (torch.zeros_like(t) for t in (q, q, k, v))
    for b in range(B):
        for h in range(H):
            i, s = h // (H // G), D ** -0.5
            score = q[b, :, h] @ k[b, :, i].T * s
            if case["alibi"]:
                score = score + 2.0 ** (-8.0 * (h + 1) / H) * far
            p = torch.softmax(score.masked_fill_(hide, float("-inf")), -1)
            o[b, :, h] = p @ v[b, :, i]
            dv[b, :, i] += p.T @ do[b, :, h]
            ds = p * (do[b, :, h] @ v[b, :, i].T - (do[b, :, h] * o[b, :, h]).sum(-1, keepdim=True))
            dq[b, :, h] = ds @ k[b, :, i] * s
            dk[b, :, i] += ds.T @ q[b, :, h] * s
    return o, dq, dk, dv


def _int4(t, group):
    """fp32 values as groups of ``group`` consecutive ones become in 4 bits: absmax / 7, halves away from zero."""
    f = t.float().reshape(-1, group)
    top = f.abs().amax(1, keepdim=True)
    s = torch.where(top < 1e-10, torch.ones_like(top), top / 7.0)
    q = (f / s).abs().add(0.5).floor().mul((f / s).sign()).clamp(-8, 7)
    return (q * s).double().view(t.shape)


def _exact_int4(case, g):
    raw = _served_weights(g)
    w = {n: _int4(t.T.contiguous(), 128).T if n.endswith(".w") and t.dim() == 2 else t.double() for n, t in raw.items()}
    if case["kind"] == "int4_prompt":
        ids, first = _ids(g, LLAMA["vocab"], case["batch"], case["seq"]), 0
    else:
        history = _ids(g, LLAMA["vocab"], case["batch"], case["history"])
        ids, first = torch.cat([history, _ids(g, LLAMA["vocab"], case["batch"], case["tokens"])], 1), case["history"]
    cached = lambda t: _int4(t.to(BF), 32)
    return torch.stack([(_llama_hidden(w, row, cached, first) @ w["head.w"].T).to(F32 if first == 0 else F64) for row in ids])


def _exact_sample(case, g):
    x = _randn(g, case["rows"], case["vocab"], std=2.0, dtype=F32).double() / case["temperature"]
    k = min(case["top_k"] or 1024, 1024, case["vocab"])
    order = torch.argsort(-x, dim=-1, stable=True)[:, :k]
    p = torch.softmax(x.gather(1, order), -1)
    if case["top_p"] < 1:
        p = p * ((p.cumsum(-1) - p) < case["top_p"])
    return None, torch.zeros_like(x).scatter_(1, order, p / p.sum(-1, keepdim=True))


def _exact_surelorn(case, g):
    m = SURELORN
    W, H, d = m["width"], m["heads"], m["dim"]
    w = {n: t.double() for n, t in _surelorn_tensors(g).items()}
    contexts = _contexts(case, g)
    tokens = _ids(g, m["vocab"], case["batch"]).tolist()
    out = []
    for c, t in zip(contexts, tokens):
        ids = torch.tensor(c + [t], device="cuda")
        T = len(ids)
        turn = torch.arange(T, device="cuda", dtype=F64)[:, None] * 10000.0 ** (-2.0 * torch.arange(W // 2, device="cuda", dtype=F64) / W)
        x = w["embed"][ids] * W ** 0.5 + torch.stack([turn.sin(), turn.cos()], -1).view(T, W)
        for i in range(m["layers"]):
            p = f"l{i}.mix."
            q = (_rms(x @ w[p + "dq"].T, w[p + "dq.norm"], 1e-6) @ w[p + "uq"].T).view(T, H, d).transpose(0, 1)
            lat = _rms(x @ w[p + "dkv"].T, w[p + "dkv.norm"], 1e-6)
            k, v = ((lat @ w[p + n].T).view(T, H, d).transpose(0, 1) for n in ("uk", "uv"))
            o = _softmax_attention(q, k, v, d ** -0.5).transpose(0, 1).reshape(T, H * d)
            x = x + _rms(o @ w[p + "o"].T, w[f"l{i}.norm1"], 1e-6)
            p = f"l{i}.mlp."
            x = x + _rms((torch.nn.functional.silu(x @ w[p + "gate"].T) * (x @ w[p + "up"].T)) @ w[p + "down"].T, w[f"l{i}.norm2"], 1e-6)
        out.append(_rms(x[-1], w["final.norm"], 1e-6) @ w["head"].T)
    return torch.stack(out)


def _turn(x, base, sign=1):
    """[T, .., D]: elements 2 i and 2 i + 1 are a plane turned by position * base^(-2 i / D)."""
    T, D = x.shape[0], x.shape[-1]
    a = sign * torch.arange(T, device="cuda", dtype=F64)[:, None] * base ** (-2.0 * torch.arange(D // 2, device="cuda", dtype=F64) / D)
    a = a.view((T,) + (1,) * (x.dim() - 2) + (D // 2,))
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1).flatten(-2)


def _recurrence(q, k, v, a):
    """S <- diag(a) S + k v^T, o = S^T q; everything [T, H, d]."""
    S, out = torch.zeros(q.shape[1], q.shape[2], v.shape[2], device="cuda", dtype=F64), []
    for t in range(q.shape[0]):
        S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return torch.stack(out)


def _exact_nufalorn(case, g):
    m, F = NUFALORN, torch.nn.functional
    H, d, G, eps = m["heads"], m["dim"], m["kv_heads"], m["eps"]
    w = {n: t.double() for n, t in _nufalorn_tensors(g).items()}
    out = []
    for prompt in _prompts(case, g):
        T = len(prompt)
        x = w["embed"][torch.tensor(prompt, device="cuda")]
        for i, kind in enumerate(m["kinds"]):
            t = {n[len(f"l{i}.mix."):]: v for n, v in w.items() if n.startswith(f"l{i}.mix.")}
            h = _rms(x, 1 + w[f"l{i}.norm1"], eps)
            part = lambda n: (h @ t[n].T).view(T, -1, d)
            if kind == "attention":
                q, k, v = _turn(part("q"), m["base"]), _turn(part("k"), m["base"]), _turn(_rms(part("v"), 1.0, eps), m["base"])
                q, k, v = (z.repeat_interleave(H // z.shape[1], 1).transpose(0, 1) for z in (q, k, v))
                s = (q @ k.transpose(1, 2) * d ** -0.5).masked_fill(torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1), float("-inf"))
                p = torch.softmax(F.pad(s, (0, 1)), -1)[..., :T]             # one more score of 0: the sink
                y = _turn((p @ v).transpose(0, 1), m["base"], -1).reshape(T, H * d)
            elif kind == "hgrn2":
                f = t["lower"] + (1 - t["lower"]) * torch.sigmoid(h @ t["f"].T + t["f.b"])
                f = f.view(T, H, d)
                y = (_rms(_recurrence(F.silu(part("q")), 1 - f, part("v"), f), t["norm"], eps)).reshape(T, H * d)
            else:
                a = torch.sigmoid((h @ t["a1"].T) @ t["a2"].T + t["a2.b"]) ** (1 / m["tau"])
                o = _recurrence(part("q") * d ** -0.5, part("k"), part("v"), a.view(T, H, d))
                y = _rms(o, t["norm"], eps).reshape(T, H * d) * F.silu(h @ t["g"].T)
            h = _rms(x, 1 + w[f"l{i}.norm2"], eps)
            p = f"l{i}.mlp."
            x = x + m["mult"] * (y @ t["o"].T + (torch.relu(h @ w[p + "gate"].T) * (h @ w[p + "up"].T)) @ w[p + "down"].T)
        logits = _rms(x[-1], 1 + w["final.norm"], eps) @ w["head"].T
        out.append(m["cap"] * torch.tanh(logits / m["cap"]))
    return torch.stack(out)


def _exact_experts(case, g):
    m, F = EXPERTS, torch.nn.functional
    t, x, w = _expert_inputs(case, g)
    t, h = {n: v.double() for n, v in t.items()}, x.to(BF).double()
    gated = lambda z, p: (F.silu(z @ t[p + "gate"].T) * (z @ t[p + "up"].T)) @ t[p + "down"].T
    s = torch.softmax(h @ t["router"].T, -1)
    choice = s + t["correction"]
    per = m["experts"] // m["groups"]
    kept = choice.view(-1, m["groups"], per).amax(-1).topk(m["keep"])[1]
    allowed = torch.zeros(len(h), m["groups"], dtype=torch.bool, device="cuda").scatter_(1, kept, True).repeat_interleave(per, 1)
    picked = choice.masked_fill(~allowed, float("-inf")).topk(m["top"])[1]
    weight = s.gather(1, picked)
    weight = weight / weight.sum(-1, keepdim=True)
    y = gated(h, "shared.")
    for e in range(m["experts"]):
        row, at = (picked == e).nonzero(as_tuple=True)
        y[row] += weight[row, at, None] * gated(h[row], f"e{e}.")
    x = x.double() + _rms(y, w.double(), m["eps"])
    return x, x


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in SHAPES:
        return _exact_step(case, g)
    with torch.no_grad():
        return {"attention": _exact_attention, "int4_prompt": _exact_int4, "int4_decode": _exact_int4, "sample": _exact_sample, "surelorn_decode": _exact_surelorn,
                "nufalorn_prompt": _exact_nufalorn, "experts": _exact_experts}[kind](case, g)


def tolerance(case):
    """About four times the error against ``exact`` as measured: bf16 operands with fp32 sums; in training, gradients through all layers; with the INT4
    cache, values next to a rounding boundary of 4 bits; sampling is fp32 throughout."""
    kind = case["kind"]
    if kind in SHAPES:
        return {"rel": 0.03, "max": 0.9}
    if kind == "sample":
        return {"rel": 1e-5, "max": 1e-3, "differ": 0.01}
    return {"rel": {"attention": 0.012, "surelorn_decode": 0.008, "nufalorn_prompt": 0.022, "experts": 0.012}.get(kind, 0.03), "max": 0.9}
