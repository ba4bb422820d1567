"""Norm, loss, elementwise, reduction, embedding and optimizer kernels against
PyTorch fp32 on a B200."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def relerr(x, ref):
    x, ref = x.float().cpu(), ref.float().cpu()
    return ((x - ref).abs().max() / (ref.abs().max() + 1e-6)).item()


@pytest.mark.parametrize("B,T,H,D", [(1, 1, 1, 16), (3, 7, 5, 64), (2, 33, 3, 128), (1, 5, 2, 48)])
@pytest.mark.parametrize("backward", [False, True])
def test_rope_by_eight_pairs(B, T, H, D, backward):
    from cogito_b200.ops import misc as M
    torch.manual_seed(T)
    cos, sin = M.rope_tables(40, D, 10000.0, DEV)
    packed = torch.randn(B, T, H + 2, D, device=DEV, dtype=torch.bfloat16)
    pos = torch.randint(-2, 45, (B, T), dtype=torch.int32, device=DEV)                   # clamped to the table
    for how in ({"pos_offset": 4}, {"positions": pos}):
        got, ref = packed.clone(), packed.cpu()
        M.rope_apply_(got[:, :, 1:1 + H], cos, sin, backward=backward, **how)
        how = {k: v.cpu() if isinstance(v, torch.Tensor) else v for k, v in how.items()}
        M.rope_apply_(ref[:, :, 1:1 + H], cos.cpu(), sin.cpu(), backward=backward, **how)
        assert relerr(got, ref) < 2 ** -8 and torch.equal(got[:, :, 0].cpu(), packed[:, :, 0].cpu()) and torch.equal(got[:, :, -1].cpu(), packed[:, :, -1].cpu())


# both sides of the line between the backward kernels: narrow rows and small products, element by element; the others by rows
@pytest.mark.parametrize("rows,H", [(1, 8), (1100, 120), (1024, 128), (1023, 128), (513, 256), (129, 1016)])
def test_swiglu_backward_on_both_sides_of_its_line(rows, H):
    from cogito_b200.ops import _lib
    L = _lib.lib()
    torch.manual_seed(H)
    x, dy = torch.randn(rows, 2 * H, device=DEV).bfloat16(), torch.randn(rows, H, device=DEV).bfloat16()
    got, ref, xf, dyf = torch.empty_like(x), torch.empty(rows, 2 * H, device=DEV), x.float(), dy.float()
    _lib.check(L.cgk_swiglu_backward(1, x.data_ptr(), dy.data_ptr(), got.data_ptr(), rows, H, _lib.stream_ptr()))
    _lib.check(L.cgk_swiglu_backward(0, xf.data_ptr(), dyf.data_ptr(), ref.data_ptr(), rows, H, _lib.stream_ptr()))
    assert torch.equal(got, ref.bfloat16())


# the vectorised bf16 kernels divide without a branch: every bf16 gate (infinities, NaN, zeros of both signs, denormals) rounds to what
# the fp32 kernels' division rounds to
@pytest.mark.parametrize("draw", range(3))
def test_swiglu_over_all_bf16_gates_has_the_bits_of_the_division(draw):
    from cogito_b200.ops import _lib
    L, H = _lib.lib(), 65536
    g = torch.arange(H, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    torch.manual_seed(draw)
    one = torch.ones(H, device=DEV, dtype=torch.bfloat16)
    up, dy = (one, one) if draw == 0 else (torch.randn(H, device=DEV).bfloat16() for _ in range(2))
    rows = 2                                                  # the backward kernel by rows starts at 128 K elements
    x, dy = torch.cat([g, up]).repeat(rows, 1), dy.repeat(rows, 1)
    got, dgot = torch.empty(rows, H, device=DEV, dtype=torch.bfloat16), torch.empty(rows, 2 * H, device=DEV, dtype=torch.bfloat16)
    ref, dref, xf, dyf = torch.empty(rows, H, device=DEV), torch.empty(rows, 2 * H, device=DEV), x.float(), dy.float()
    _lib.check(L.cgk_swiglu_forward(1, x.data_ptr(), got.data_ptr(), rows, H, _lib.stream_ptr()))
    _lib.check(L.cgk_swiglu_forward(0, xf.data_ptr(), ref.data_ptr(), rows, H, _lib.stream_ptr()))
    _lib.check(L.cgk_swiglu_backward(1, x.data_ptr(), dy.data_ptr(), dgot.data_ptr(), rows, H, _lib.stream_ptr()))
    _lib.check(L.cgk_swiglu_backward(0, xf.data_ptr(), dyf.data_ptr(), dref.data_ptr(), rows, H, _lib.stream_ptr()))
    for a, b in ((got, ref.bfloat16()), (dgot, dref.bfloat16())):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.view(torch.int16)[~a.isnan()], b.view(torch.int16)[~b.isnan()])


# rows of more than 1024 elements take a CTA each: the smallest and largest, a width that fills no whole warp, more rows than CTAs
@pytest.mark.parametrize("rows,D", [(1, 1032), (5, 8192), (700, 1608), (1300, 2048)])
@pytest.mark.parametrize("rms", [False, True])
def test_wide_norm_against_64_bits(rows, D, rms):
    from cogito_b200.ops import norm as N
    torch.manual_seed(rows)
    x, r, dy = (torch.randn(rows, D, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    g = (torch.randn(D, device=DEV) * 0.1 + 1).bfloat16()
    b = None if rms else torch.randn(D, device=DEV).bfloat16()
    y, s, mean, rstd = N.norm_forward_raw(x, g, b, 1e-5, rms, r, True)
    assert torch.equal(s, (x.float() + r.float()).bfloat16())
    dx, dg, db = N.norm_backward_raw(dy, s, g, mean, rstd, rms, r)
    sd, gd = s.double(), g.double()
    m = 0.0 if rms else sd.mean(-1, keepdim=True)
    rs = ((sd - m).pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt()
    h, t = (sd - m) * rs, dy.double() * gd
    s1 = 0.0 if rms else t.mean(-1, keepdim=True)
    rel = lambda u, v: ((u.double() - v).norm() / v.norm()).item()
    # bf16 results of fp32 arithmetic: 2^-9 at most, half that on average; fp32 column sums of `rows` terms
    assert rel(y, h * gd + (0.0 if rms else b.double())) < 2 ** -9 * 1.1
    assert rel(dx, rs * (t - s1 - h * (t * h).mean(-1, keepdim=True)) + r.double()) < 2 ** -9 * 1.1
    assert rel(dg, (dy.double() * h).sum(0)) < 2e-6 and (rms or rel(db, dy.double().sum(0)) < 2e-6)
    if rms:
        u = x.clone()
        assert torch.equal(N.add_rms_norm_(u, r, g, 1e-5), y) and torch.equal(u, s)


# a row's result does not depend on how many rows the call has: few rows take a CTA each, many a warp each
@pytest.mark.parametrize("D", [1032, 1608, 2048, 4096, 8192])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("with_res", [False, True])
def test_wide_norm_has_the_same_bits_for_few_rows_and_for_many(D, rms, with_res):
    from cogito_b200.ops import norm as N
    torch.manual_seed(D)
    few, many = 592, 2560                                     # four rows per SM of 148, and more than that
    x = torch.randn(many, D, device=DEV, dtype=torch.bfloat16) * 3 + 0.5
    r = torch.randn(many, D, device=DEV, dtype=torch.bfloat16) if with_res else None
    g = (torch.randn(D, device=DEV) * 0.1 + 1).bfloat16()
    b = None if rms else torch.randn(D, device=DEV).bfloat16()
    whole = N.norm_forward_raw(x, g, b, 1e-5, rms, r, True)
    for part in (slice(0, few), slice(few, few + 1), slice(many - 37, many)):
        got = N.norm_forward_raw(x[part], g, b, 1e-5, rms, None if r is None else r[part], True)
        for u, v in zip(got, whole):
            assert (u is None) == (v is None) and (u is None or torch.equal(u, v[part]))


# one element per access below 80 K elements or off a 16-byte boundary, four above
@pytest.mark.parametrize("n", [1, 1000, 81919, 81920, 81923, 200001])
@pytest.mark.parametrize("shift", [0, 1])
def test_adam_step_by_one_and_by_four(n, shift):
    from cogito_b200.ops import _lib
    torch.manual_seed(n)
    p, m, v, g = (torch.rand(n + 4, device=DEV)[shift:shift + n] for _ in range(4))
    p16 = torch.empty(n + 4, device=DEV, dtype=torch.bfloat16)[shift:shift + n]
    lr, b1, b2, eps, wd = 1e-2, 0.9, 0.99, 1e-8, 0.1
    pd, md, vd, gd = (t.double() for t in (p, m, v, g))
    md, vd = b1 * md + (1 - b1) * gd, b2 * vd + (1 - b2) * gd * gd
    pd = pd * (1 - lr * wd) - lr * (md / (1 - b1)) / ((vd / (1 - b2)).sqrt() + eps)
    _lib.check(_lib.lib().cgk_adam_step(p.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(), p16.data_ptr(), n, lr, b1, b2, eps, wd, 0.0, None, _lib.stream_ptr()))
    # a handful of fp32 roundings each; 1 - b2 and 1 - b1 are fp32 differences of rounded constants: 2^-24 / 0.01 at most
    for got, ref in ((m, md), (v, vd), (p, pd)):
        assert ((got.double() - ref).abs() <= ref.abs() * 1e-5 + 1e-6).all()
    assert torch.equal(p16, p.bfloat16())


@pytest.mark.parametrize("D", [768, 1608, 4096])
def test_norm_backward_takes_scratch_on_any_boundary(D):
    from cogito_b200.ops import _lib
    L, rows = _lib.lib(), 70
    torch.manual_seed(D)
    x, dy = (torch.randn(rows, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    g, mean, rstd = torch.ones(D, device=DEV, dtype=torch.bfloat16), torch.zeros(rows, device=DEV), torch.ones(rows, device=DEV)
    n, results = L.cgk_norm_backward_scratch_elems(rows, D), []
    for shift in (0, 1, 2, 3):
        scratch, dx, dg, db = torch.empty(n + 4, device=DEV), torch.empty_like(x), torch.empty(D, device=DEV), torch.empty(D, device=DEV)
        _lib.check(L.cgk_norm_backward(dy.data_ptr(), x.data_ptr(), g.data_ptr(), mean.data_ptr(), rstd.data_ptr(), None, dx.data_ptr(), dg.data_ptr(),
                                       db.data_ptr(), scratch[shift:].data_ptr(), rows, D, 0, 0, _lib.stream_ptr()))
        results.append((dx, dg, db))
    assert all(torch.equal(a, b) for r in results[1:] for a, b in zip(r, results[0]))


def test_add_rms_norm_refuses_other_shapes_and_takes_any_alignment():
    from cogito_b200.ops import norm as N
    torch.manual_seed(3)
    for dev in ("cpu", DEV):
        x, y, g = (torch.randn(*s, device=dev).bfloat16() for s in ((3, 2, 64), (6, 64), (64,)))
        before = x.clone()
        for bad_y, bad_g in ((y[:5], g), (torch.cat([y, y]), g), (y, g[:56]), (y, torch.cat([g, g]))):
            with pytest.raises((ValueError, RuntimeError)):
                N.add_rms_norm_(x, bad_y, bad_g, 1e-5)
            assert torch.equal(x, before)
        want_x = before + y.view_as(x)
        want = N.rms_norm(want_x, g, 1e-5)
        shifted = torch.cat([y.new_zeros(4), y.reshape(-1)])[4:].view(6, 64)           # contiguous, 8 bytes off a 16-byte boundary
        wide = torch.cat([y, y], 1)[:, :64].reshape(3, 2, 64).transpose(0, 1).contiguous().transpose(0, 1)     # not contiguous
        for form in (y, shifted, wide):
            u = before.clone()
            assert torch.equal(N.add_rms_norm_(u, form, g, 1e-5), want) and torch.equal(u, want_x)
        gp = g.clone().requires_grad_()
        u = before.clone()
        N.add_rms_norm_(u, y, gp, 1e-5).float().sum().backward()                       # a weight that autograd follows has its gradient
        assert gp.grad is not None and gp.grad.float().abs().sum() > 0


@pytest.mark.parametrize("rows,D", [(64, 768), (33, 128), (1000, 4096), (7, 8)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("with_res", [False, True])
def test_norm_forward_backward(rows, D, rms, with_res):
    from cogito_b200.ops import norm as N
    torch.manual_seed(0)
    x = torch.randn(rows, D, device=DEV, dtype=torch.bfloat16)
    r = torch.randn(rows, D, device=DEV, dtype=torch.bfloat16) if with_res else None
    g = (torch.randn(D, device=DEV) * 0.1 + 1).to(torch.bfloat16)
    b = None if rms else (torch.randn(D, device=DEV) * 0.1).to(torch.bfloat16)
    xs = [t.clone().requires_grad_(True) for t in (x, g)] + ([b.clone().requires_grad_(True)] if b is not None else [])
    rg = r.clone().requires_grad_(True) if with_res else None
    out = N.rms_norm(xs[0], xs[1], 1e-5, rg) if rms else N.layer_norm(xs[0], xs[1], xs[2], 1e-5, rg)
    y, s = out if with_res else (out, None)
    # fp32 oracle
    xf = x.float().requires_grad_(True)
    rf = r.float().requires_grad_(True) if with_res else None
    gf = g.float().requires_grad_(True)
    bf = b.float().requires_grad_(True) if b is not None else None
    sf = xf + rf if with_res else xf
    if with_res:
        sf = sf.detach().to(torch.bfloat16).float() + (sf - sf.detach())   # the kernel rounds the sum to bf16
    if rms:
        yf = sf * torch.rsqrt((sf * sf).mean(-1, keepdim=True) + 1e-5) * gf
    else:
        yf = torch.nn.functional.layer_norm(sf, (D,), gf, bf, 1e-5)
    assert relerr(y, yf) < 2e-2
    dy = torch.randn_like(y)
    ds = torch.randn_like(y) if with_res else None
    if with_res:
        torch.autograd.backward([y, s], [dy, ds])
        torch.autograd.backward([yf, sf], [dy.float(), ds.float()])
    else:
        y.backward(dy)
        yf.backward(dy.float())
    assert relerr(xs[0].grad, xf.grad) < 3e-2
    assert relerr(xs[1].grad, gf.grad) < 3e-2
    if b is not None:
        assert relerr(xs[2].grad, bf.grad) < 3e-2
    if with_res:
        assert relerr(rg.grad, rf.grad) < 3e-2


@pytest.mark.parametrize("R,V", [(64, 50304), (33, 32000), (5, 1000), (16, 10)])
def test_fused_cross_entropy(R, V):
    from cogito_b200.ops.loss import cross_entropy
    torch.manual_seed(0)
    logits = (torch.randn(R, V, device=DEV) * 2).to(torch.bfloat16)
    tg = torch.randint(0, V, (R,), device=DEV)
    tg[0] = -100
    ref_in = logits.float().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(ref_in, tg, ignore_index=-100)
    ref.backward()
    x = logits.clone().requires_grad_(True)
    y = x * 1.0
    loss = cross_entropy(y, tg, grad_scale=4.0)
    loss.backward()
    assert abs(float(loss) - float(ref)) < 2e-2 * max(1.0, abs(float(ref)))
    assert relerr(x.grad, ref_in.grad * 4.0) < 3e-2
    # device-resident scale
    x2 = logits.clone().requires_grad_(True)
    loss2 = cross_entropy(x2 * 1.0, tg, grad_scale=torch.tensor([4.0], device=DEV))
    loss2.backward()
    assert relerr(x2.grad, ref_in.grad * 4.0) < 3e-2


def test_ce_stats_and_backward_split():
    import ctypes
    from cogito_b200.ops import _lib
    torch.manual_seed(0)
    R, V = 40, 4096
    logits = torch.randn(R, V, device=DEV).to(torch.bfloat16)
    tg = torch.randint(0, V, (R,), device=DEV)
    L = _lib.lib()
    halves = []
    for s in range(2):
        sh = logits[:, s * V // 2:(s + 1) * V // 2].contiguous()
        mx, sm, tl = (torch.empty(R, device=DEV) for _ in range(3))
        _lib.check(L.cgk_ce_stats(sh.data_ptr(), tg.data_ptr(), s * V // 2, mx.data_ptr(), sm.data_ptr(),
                                  tl.data_ptr(), R, V // 2, V // 2, _lib.stream_ptr()))
        halves.append((sh, mx, sm, tl))
    gmax = torch.maximum(halves[0][1], halves[1][1])
    gsum = sum(h[2] * torch.exp(h[1] - gmax) for h in halves)
    lse = gmax + torch.log(gsum)
    tgt = halves[0][3] + halves[1][3]
    ref = torch.nn.functional.cross_entropy(logits.float(), tg, reduction="none")
    assert relerr(lse - tgt, ref) < 1e-2
    probs = torch.softmax(logits.float(), -1)
    probs[torch.arange(R), tg] -= 1
    for s, (sh, *_rest) in enumerate(halves):
        d = torch.empty_like(sh)
        _lib.check(L.cgk_ce_backward(sh.data_ptr(), tg.data_ptr(), s * V // 2, lse.data_ptr(), d.data_ptr(), R,
                                     V // 2, V // 2, 1.0, None, -100, _lib.stream_ptr()))
        assert relerr(d, probs[:, s * V // 2:(s + 1) * V // 2]) < 2e-2


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_elementwise_and_broadcast(dtype):
    from cogito_b200.ops import functional as F
    torch.manual_seed(0)
    a = torch.randn(5, 1, 33, device=DEV).to(dtype)
    b = torch.randn(1, 7, 33, device=DEV).to(dtype)
    for op, fn in [("add", torch.add), ("sub", torch.sub), ("mul", torch.mul), ("div", torch.div)]:
        bb = b + 3 if op == "div" else b
        assert relerr(F.binary(op, a, bb), fn(a.float(), bb.float())) < 2e-2
    big = torch.randn(1 << 16, device=DEV).to(dtype)
    assert relerr(F.binary("add", big, big), big.float() * 2) < 1e-2
    x = torch.rand(1000, device=DEV).to(dtype) + 0.5
    for op, fn in [("exp", torch.exp), ("log", torch.log), ("sqrt", torch.sqrt), ("tanh", torch.tanh),
                   ("sigmoid", torch.sigmoid), ("relu", torch.relu), ("rsqrt", torch.rsqrt),
                   ("gelu", lambda t: torch.nn.functional.gelu(t, approximate="tanh")),
                   ("silu", torch.nn.functional.silu)]:
        assert relerr(F.unary(op, x), fn(x.float())) < 2e-2, op
        xr = x.float().clone().detach().requires_grad_(True)
        fn(xr).sum().backward()
        dy = torch.ones_like(x)
        assert relerr(F.unary_backward(op, x, dy), xr.grad) < 3e-2, op
    assert relerr(F.unary("pow", x, 3.0), x.float() ** 3) < 2e-2


def test_large_elementwise_beyond_16M_elements():
    """The reference's grid cap (65535 blocks, no stride loop) breaks above 16.7 M elements."""
    from cogito_b200.ops import functional as F
    n = (1 << 24) + 12345
    a = torch.ones(n, device=DEV)
    out = F.binary("add", a, a)
    assert float(out.min()) == 2.0 and float(out[-1]) == 2.0


def test_reductions():
    from cogito_b200.ops import functional as F
    torch.manual_seed(0)
    x = torch.randn(6, 50, 9, device=DEV)
    for op, fn in [("sum", torch.sum), ("mean", torch.mean)]:
        assert relerr(F.reduce(op, x), fn(x).reshape(1)) < 1e-4
        for d in range(3):
            assert relerr(F.reduce(op, x, d), fn(x, d)) < 1e-4
    assert relerr(F.reduce("max", x, 1), x.max(1).values) == 0
    assert relerr(F.reduce("min", x), x.min().reshape(1)) == 0
    m = torch.randn(777, 100, device=DEV).to(torch.bfloat16)
    assert relerr(F.colsum(m), m.float().sum(0)) < 1e-3


def test_embedding_swiglu_dropout():
    from cogito_b200.ops import misc as M
    torch.manual_seed(0)
    V, D, B, T = 100, 64, 3, 17
    wte = torch.randn(V, D, device=DEV).to(torch.bfloat16).requires_grad_(True)
    wpe = torch.randn(32, D, device=DEV).to(torch.bfloat16).requires_grad_(True)
    ids = torch.randint(0, V, (B, T), device=DEV)
    out = M.embedding(ids, wte, wpe)
    ref = wte.float()[ids] + wpe.float()[:T][None]
    assert relerr(out, ref) < 1e-2
    g = torch.randn_like(out)
    out.backward(g)
    rw = torch.zeros(V, D, device=DEV).index_add_(0, ids.reshape(-1), g.float().reshape(-1, D))
    assert relerr(wte.grad, rw) < 2e-2
    assert relerr(wpe.grad[:T], g.float().sum(0)) < 2e-2
    x = torch.randn(9, 2 * 40, device=DEV).to(torch.bfloat16).requires_grad_(True)
    y = M.swiglu(x)
    xf = x.detach().float().requires_grad_(True)
    yf = torch.nn.functional.silu(xf[:, :40]) * xf[:, 40:]
    assert relerr(y, yf) < 2e-2
    gy = torch.randn_like(y)
    y.backward(gy)
    yf.backward(gy.float())
    assert relerr(x.grad, xf.grad) < 3e-2
    z = torch.ones(100000, device=DEV)
    d = M.dropout(z, 0.25, True, seed=7)
    kept = (d != 0).float().mean().item()
    assert abs(kept - 0.75) < 0.01 and abs(float(d.max()) - 1 / 0.75) < 1e-5
    assert torch.equal(d, M.dropout(z, 0.25, True, seed=7))


def test_fused_adam_and_scaler_match_cpu_rule():
    from cogito_b200.optim.fused import FusedAdam, GradScaler
    torch.manual_seed(0)
    w_g = torch.nn.Parameter(torch.randn(300, 17, device=DEV).to(torch.bfloat16))
    w_c = torch.nn.Parameter(w_g.detach().float().cpu().clone())
    og = FusedAdam([w_g], lr=1e-2, weight_decay=0.1, scaler=GradScaler(DEV, enabled=True, init_scale=1024.0))
    oc = FusedAdam([w_c], lr=1e-2, weight_decay=0.1, scaler=GradScaler("cpu", enabled=True, init_scale=1024.0))
    for step in range(4):
        g = torch.randn(300, 17)
        if step == 2:
            g[0, 0] = float("inf")          # overflow: both must skip and halve the scale
        og.zero_grad(); oc.zero_grad()
        w_g.main_grad.copy_((g * og.scaler.sync()["scale"]).to(DEV))
        w_c.main_grad.copy_(g * oc.scaler.scale)
        og.step(); oc.step()
    sg, sc = og.scaler.sync(), oc.scaler.sync()
    assert sg["scale"] == sc["scale"] == 512.0 and sg["skipped"] == sc["skipped"] == 1 and sg["step"] == sc["step"] == 3
    assert relerr(og.master, oc.fp.flat) < 1e-5
    assert relerr(w_g, w_c) < 1e-2


def test_fused_sgd_nesterov_matches_torch():
    from cogito_b200.optim.fused import FusedSGD
    torch.manual_seed(0)
    w = torch.nn.Parameter(torch.randn(1000, device=DEV))
    wt = torch.nn.Parameter(w.detach().clone())
    o = FusedSGD([w], lr=0.1, momentum=0.9, weight_decay=0.01, nesterov=True, master_weights=False)
    ot = torch.optim.SGD([wt], lr=0.1, momentum=0.9, weight_decay=0.01, nesterov=True)
    for _ in range(5):
        g = torch.randn(1000, device=DEV)
        o.zero_grad(); w.main_grad.copy_(g); o.step()
        wt.grad = g.clone(); ot.step()
    assert relerr(w, wt) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_softmax_dropout_residual_kernel(dtype):
    """One row kernel for softmax -> multiply -> add, against the three separate steps."""
    from cogito_b200.ops.misc import _dropout_apply, softmax_dropout_residual
    torch.manual_seed(0)
    tol = 1e-5 if dtype == torch.float32 else 2e-2
    x = torch.randn(37, 4, 1000, device="cuda").to(dtype).requires_grad_(True)
    res = torch.randn(37, 4, 1000, device="cuda").to(dtype).requires_grad_(True)
    mul = ((torch.rand(37, 4, 1000, device="cuda") > 0.3).float() / 0.7).to(dtype)
    out = softmax_dropout_residual(x, res, mul=mul)
    ref = torch.softmax(x.float(), -1) * mul.float() + res.float()
    assert (out.float() - ref).abs().max() < tol
    g = torch.randn_like(out)
    gx, gr = torch.autograd.grad(out, (x, res), g)
    rx, rr = torch.autograd.grad(ref, (x, res), g.float())
    assert (gx.float() - rx.float()).abs().max() < tol * max(1.0, float(rx.abs().max())) and torch.equal(gr, g)
    # generated mask = the mask of the stand-alone dropout kernel for the same seed
    y = softmax_dropout_residual(x.detach(), res.detach(), p=0.2, seed=77)
    s = torch.softmax(x.detach().float(), -1)
    sep = _dropout_apply(s, 0.2, 77) + res.detach().float()
    assert (y.float() - sep).abs().max() < tol
    x2 = x.detach().clone().requires_grad_(True)
    y2 = softmax_dropout_residual(x2, None, p=0.2, seed=77)
    (g2,) = torch.autograd.grad(y2, x2, g)
    xs = x.detach().float().requires_grad_(True)
    keep = _dropout_apply(torch.ones_like(xs), 0.2, 77)          # the mask itself, scaled by 1 / (1 - p)
    (r2,) = torch.autograd.grad(torch.softmax(xs, -1) * keep, xs, g.float())
    assert (g2.float() - r2).abs().max() < tol * max(1.0, float(r2.abs().max()))
