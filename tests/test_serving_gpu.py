"""Serving kernels on the GPU against their host restatements (fp32 PyTorch / the C library)."""
import copy
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from cogito_b200.models.llama import Llama, LlamaConfig
from cogito_b200.ops import _lib
from cogito_b200.quant.int4 import Int4Linear, dequantize_int4, quantize_int4
from cogito_b200.serve.engine import LlamaInt4Engine, SpeculativeDecoder
from cogito_b200.serve.kv_cache import PagedKVCacheInt4
from cogito_b200.serve.sampling import filtered_probs, sample, spec_accept, tree_attention_mask
from cogito_b200.utils import rng

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROOT = Path(__file__).resolve().parent.parent


def test_int4_quantize_dequantize_bit_exact_with_host():
    torch.manual_seed(0)
    x = torch.randn(64, 384) * 2
    x[0, :4] = torch.tensor([0.5, 1.5, -0.5, -2.5]) * (x[0, :128].abs().max() / 7)
    pc, sc = quantize_int4(x, 128)
    pg, sg = quantize_int4(x.to(DEV), 128)
    assert torch.equal(pg.cpu(), pc) and torch.equal(sg.cpu(), sc)
    assert torch.equal(dequantize_int4(pg, sg, x.numel(), 128).cpu(), dequantize_int4(pc, sc, x.numel(), 128))
    assert torch.equal(dequantize_int4(pg, sg, x.numel(), 128, torch.bfloat16).cpu(),
                       dequantize_int4(pc, sc, x.numel(), 128).bfloat16())


@pytest.mark.parametrize("M,K,N,group,splits", [(16, 512, 256, 128, 0), (80, 1024, 384, 128, 2), (5, 256, 128, 64, 1),
                                                (130, 512, 256, 128, 0), (1, 4096, 512, 128, 0)])
@pytest.mark.parametrize("kernel", ["wb", "wa"])
def test_int4_gemm_matches_dequantised_product(M, K, N, group, splits, kernel):
    torch.manual_seed(M + K)
    w = torch.randn(N, K) * 0.05
    bias = torch.randn(N) * 0.1
    lin = Int4Linear(w, bias, group).to(DEV)
    lin.kernel = kernel
    x = (torch.randn(M, K) + 0.5).bfloat16()                # a DC offset exercises the row-sum correction of "wa"
    got = lin(x.to(DEV), splits=splits).float().cpu()
    # oracle: the same packed weights, dequantised on the host, fp32 product
    wt = dequantize_int4(lin.packed.cpu(), lin.scales.cpu(), K * N, group).view(K, N)
    ref = x.float() @ wt + lin.bias.float().cpu()
    err = (got - ref).abs().max().item()
    assert err <= 2e-2 * ref.abs().max().item() + 1e-2, err
    _lib.assert_device_ok()


# the line of steps is cut into equal pieces: fewer steps than CTAs (one tile), pieces inside a tile, over several tiles, an odd
# number of steps per tile, every number of X chunks per thread, two row tiles
@pytest.mark.parametrize("M,K,N", [(1, 128, 128), (16, 384, 128), (16, 11008, 640), (17, 128 * 29, 1280), (48, 256, 12800), (80, 4096, 6144),
                                   (96, 640, 8192), (128, 1408, 4096), (150, 512, 1024)])
@pytest.mark.parametrize("kernel", ["wa", "wb"])
def test_int4_gemm_pieces_of_the_weight_stream(M, K, N, kernel):
    torch.manual_seed(M + K)
    lin = Int4Linear(torch.randn(N, K) * 0.05, torch.randn(N) * 0.1, 128).to(DEV)
    lin.kernel = kernel
    x = (torch.randn(M, K) + 0.5).bfloat16().to(DEV)
    ref = x.double() @ lin.dequantized().double() + lin.bias.double()
    for _ in range(2):                                        # the scratch is left zero for the next call
        # one operand is scaled and rounded to bf16 once per element (wb: its scale before that), the sums are fp32: 2^-8 of the
        # terms' norm at most, and the result's rounding
        err = (lin(x).double() - ref).norm() / ref.norm()
        assert err < 2 ** -7, err
    _lib.assert_device_ok()


# few rows: 8, 16 and 32 columns of MMAs, one unit of 64 k per warp and fewer, clusters of eight down to two and pieces of the line,
# an fp32 result; rows of X and of the output that lie further apart than they are long are the C entry's
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 31, 33, 65])
@pytest.mark.parametrize("K,N", [(128, 256), (512, 128), (1024, 640), (4096, 2176), (1664, 6144), (1152, 9600)])
def test_int4_gemm_few_rows(M, K, N):
    torch.manual_seed(M + K)
    lin = Int4Linear(torch.randn(N, K) * 0.05, torch.randn(N) * 0.1, 128).to(DEV)
    lin.kernel = "wa"
    x = (torch.randn(M, K) + 0.5).bfloat16().to(DEV)
    ref = x.double() @ lin.dequantized().double() + lin.bias.double()
    full = lin(x, f32=True)
    assert full.dtype == torch.float32
    # x' is rounded to bf16 once per element (2^-9 of the terms' norm), sums are fp32 with terms 17 times as large as the weights
    assert ((full.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    assert torch.equal(full.bfloat16(), lin(x)) and torch.equal(full, lin(x, f32=True))
    _lib.assert_device_ok()


# an fp32 result of "wb": whole tiles and parts of tiles, rows that end inside a warp, an odd number of steps for the two converting groups
@pytest.mark.parametrize("M,K,N,group", [(33, 128, 128, 64), (80, 384, 22016, 128), (97, 4096, 640, 128), (130, 1152, 19072, 64)])
def test_int4_gemm_in_fp32_by_row_tiles(M, K, N, group):
    torch.manual_seed(M + K)
    lin = Int4Linear(torch.randn(N, K) * 0.05, torch.randn(N) * 0.1, group).to(DEV)
    lin.kernel = "wb"
    x = torch.randn(M, K).bfloat16().to(DEV)
    ref = x.double() @ lin.dequantized().double() + lin.bias.double()
    full = lin(x, f32=True)
    # scale, then weight rounded to bf16 (2^-9 of the terms' norm each), fp32 sums
    assert full.dtype == torch.float32 and ((full.double() - ref).norm() / ref.norm()).item() < 2 ** -7
    assert torch.equal(full.bfloat16(), lin(x)) and torch.equal(full, lin(x, f32=True))
    _lib.assert_device_ok()


# left-over tiles in pieces of their own (uneven ones too), in equal pieces of their line, whole, and one of a single step; rows about a multiple of 16
@pytest.mark.parametrize("K,N", [(1152, 6144), (1408, 4096), (5504, 4096), (256, 11264), (128, 640)])
@pytest.mark.parametrize("M", [47, 48, 113, 129])
def test_int4_gemm_by_ways_to_deal_tiles(M, K, N):
    torch.manual_seed(M + K)
    lin = Int4Linear(torch.randn(N, K) * 0.05, torch.randn(N) * 0.1, 64).to(DEV)
    lin.kernel = "wb"
    x = torch.randn(M, K).bfloat16().to(DEV)
    ref = x.double() @ lin.dequantized().double() + lin.bias.double()
    # scale, then weight rounded to bf16 (2^-9 of the terms' norm each), fp32 sums; a bf16 result 2^-9 of its own
    got = lin(x, f32=True)
    assert ((got.double() - ref).norm() / ref.norm()).item() < 2 ** -7 and torch.equal(got.bfloat16(), lin(x))
    _lib.assert_device_ok()


# the reordered weights hold every nibble (q + 8) and scale where the products read it, also from packed weights off a word's boundary
@pytest.mark.parametrize("wa,offset", [(True, 0), (True, 1), (True, 2), (False, 0), (False, 4)])
@pytest.mark.parametrize("K,N", [(64, 128), (192, 384)])
def test_int4_tiles_hold_the_packed_weights(wa, offset, K, N):
    torch.manual_seed(K)
    L, group = _lib.lib(), 128
    room = torch.randint(0, 256, (K * N // 2 + 16,), dtype=torch.uint8, device=DEV)
    packed, scales = room[offset:offset + K * N // 2], torch.rand(K * N // group, device=DEV)
    tiles = torch.zeros((L.cgk_int4_wa_tiles_bytes if wa else L.cgk_int4_tiles_bytes)(K, N), dtype=torch.uint8, device=DEV)
    _lib.check((L.cgk_int4_wa_tile_weights if wa else L.cgk_int4_tile_weights)(packed.data_ptr(), scales.data_ptr(), K, N, group, tiles.data_ptr(), _lib.stream_ptr()))
    byte = packed.cpu().view(K, N // 2)
    u = torch.stack([byte & 0xF, byte >> 4], -1).view(K, N).int() ^ 8                              # q + 8 of [k, n]
    s = scales.cpu().view(K, N // group).repeat_interleave(group, 1)
    step = 32 if wa else 64
    tiles = tiles.cpu().view(N // 128, K // step, -1)
    words = tiles[:, :, :step * 64].contiguous().view(torch.int32).long() & 0xFFFFFFFF
    got = torch.stack([(words >> (4 * e)) & 0xF for e in range(8)], -1).int()                    # [tile, step, word, nibble]
    u = u.view(K // step, step, N // 128, 128).permute(2, 0, 1, 3)                                 # [tile, step, k, column]
    i, e = torch.arange(got.shape[2])[:, None], torch.arange(8)[None]
    if wa:
        lane, r = (i & 127) >> 2, e & 3
        column, k = (2 * (i >> 7) + ((i & 3) >> 1)) * 16 + (lane >> 2) + (r & 1) * 8, (lane & 3) * 8 + (i & 1) * 4 + (r >> 1) * 2 + (e >> 2)
    else:
        column, k = ((i & 511) >> 2) + 0 * e, (i >> 9) * 32 + (i & 3) * 8 + 2 * (e & 3) + (e >> 2)
    assert torch.equal(got, u[:, :, k, column])
    s = s.view(K // step, step, N // 128, 128).permute(2, 0, 3, 1)                                 # [tile, step, column, k]
    if wa:
        assert torch.equal(tiles[:, :, 2048:].contiguous().view(torch.float32), s[:, :, 0])
    else:
        assert torch.equal(tiles[:, :, 4096:].contiguous().view(torch.bfloat16), torch.cat([s[:, :, 0], s[:, :, 64]], -1).bfloat16())
    _lib.assert_device_ok()


# the depth of the weight ring that the environment asks for is raised to the least that the two converting groups can share
@pytest.mark.parametrize("depth", ["1", "3", "7"])
def test_int4_gemm_with_a_short_weight_ring(depth):
    code = ("import torch\nfrom cogito_b200.quant.int4 import Int4Linear\nfrom cogito_b200.ops import _lib\ntorch.manual_seed(0)\n"
            "lin = Int4Linear(torch.randn(640, 2048) * 0.05, None, 64).to('cuda')\nlin.kernel = 'wb'\nx = torch.randn(48, 2048).bfloat16().to('cuda')\n"
            "y, ref = lin(x, f32=True).double(), x.double() @ lin.dequantized().double()\n_lib.assert_device_ok()\n"
            # scale, then weight rounded to bf16 (2^-9 of the terms' norm each), fp32 sums
            "assert (y - ref).norm() / ref.norm() < 2 ** -7\n")
    run = subprocess.run([sys.executable, "-c", code], env={**os.environ, "CGK_INT4_RAW_STAGES": depth}, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


@pytest.mark.parametrize("N", [256, 22016])
def test_int4_gemm_few_rows_strided(N):
    L, M, K = _lib.lib(), 19, 1024
    lin = _int4_layer(K, N)
    lin.kernel = "wa"
    wide = torch.randn(M, K + 24, device=DEV, dtype=torch.bfloat16)
    want, out = lin(wide[:, 8:8 + K].contiguous()), torch.full((M, N + 4), 7.0, device=DEV, dtype=torch.bfloat16)
    parts = torch.empty(L.cgk_int4_wa_gemm_parts_floats(M, N, K, 0), device=DEV)
    counters = torch.zeros(L.cgk_int4_gemm_counters(M, N), dtype=torch.int32, device=DEV)
    _lib.check(L.cgk_int4_wa_gemm_parts(wide[:, 8:].data_ptr(), K + 24, lin._tiles[True].data_ptr(), parts.data_ptr(), counters.data_ptr(), out.data_ptr(), N + 4,
                                        None, M, N, K, 0, _lib.stream_ptr()), "cgk_int4_wa_gemm_parts")
    assert torch.equal(out[:, :N], want) and (out[:, N:] == 7).all() and not counters.any()


# parts of a shared tile are summed in the order of the CTAs, not of their arrival: a call gives the same bits every time
@pytest.mark.parametrize("M,K,N", [(16, 11008, 4096), (16, 4096, 22016), (80, 4096, 6144), (80, 4096, 22016), (200, 1408, 4096)])
@pytest.mark.parametrize("kernel", ["wa", "wb"])
def test_int4_gemm_repeats_itself_to_the_bit(M, K, N, kernel):
    torch.manual_seed(M + K)
    lin = Int4Linear.from_packed(torch.randint(0, 256, (K * N // 2,), dtype=torch.uint8), torch.rand(K * N // 128) * 0.01, K, N).to(DEV)
    lin.kernel = kernel
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    first = lin(x)
    for _ in range(20):
        assert torch.equal(lin(x), first)
    _lib.assert_device_ok()


# without room for the weights in bf16 a prompt goes through the streaming kernel, as it did before there was a dense route
def test_int4_linear_many_rows_without_room_for_the_dense_weights(monkeypatch):
    torch.manual_seed(9)
    lin = Int4Linear(torch.randn(384, 256) * 0.05, torch.randn(384) * 0.1, 128).to(DEV)
    x = torch.randn(300, 256, device=DEV, dtype=torch.bfloat16)

    def no_room(self, dtype=torch.float32):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(Int4Linear, "dequantized", no_room)
    out = torch.empty(300, 384, device=DEV, dtype=torch.bfloat16)
    lin.kernel = "wb"
    want = lin(x)
    lin.kernel = "auto"
    assert torch.equal(lin(x), want) and torch.equal(lin(x, out=out), want) and torch.equal(out, want)
    assert torch.equal(lin.forward_f32(x), want.float())
    _lib.assert_device_ok()


def _int4_layer(K=1024, N=2304):
    g = torch.Generator().manual_seed(K + N)
    packed = torch.randint(0, 256, (K * N // 2,), dtype=torch.uint8, generator=g)
    return Int4Linear.from_packed(packed, torch.rand(K * N // 128, generator=g) * 0.01, K, N).to(DEV)


# A captured launch keeps the addresses it was given: a later call with more rows must leave them alone, whether the kernel ran
# before the capture or not.  Memory that such a call gave back would be handed out again and filled.
@pytest.mark.parametrize("rows", [4, 20, 80])
@pytest.mark.parametrize("warm", [False, True])
def test_int4_launch_captured_before_a_larger_call(rows, warm):
    torch.manual_seed(rows)
    x, larger, prompt = (torch.randn(n, 1024, device=DEV, dtype=torch.bfloat16) for n in (rows, 200, 300))
    want, want_larger = _int4_layer()(x), _int4_layer()(larger)
    lin = _int4_layer()
    lin(prompt)                                               # goes through the dense product: no workspace yet
    if warm:
        lin(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = lin(x)
    if not warm:
        assert torch.equal(lin(x), want)                      # the layer's own copy of the weights is there before any replay
    assert torch.equal(lin(larger), want_larger)
    junk = [torch.full((n,), 0x55555555, dtype=torch.int32, device=DEV) for n in (16, 64, 256, 1024, 1 << 14, 1 << 18, 1 << 20) for _ in range(4)]
    for _ in range(3):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
    assert torch.equal(lin(larger), want_larger) and torch.equal(lin(x), want)
    assert all((j == 0x55555555).all() for j in junk)
    _lib.assert_device_ok()


def test_int4_launches_captured_more_often_than_there_are_counters():
    x = torch.randn(16, 1024, device=DEV, dtype=torch.bfloat16)
    lin = _int4_layer()
    want, graphs = lin(x), []
    for _ in range(lin._counters.CAPTURES + 3):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = lin(x)
        graphs.append((graph, got))
    for graph, got in graphs:
        for _ in range(2):
            got.zero_()
            graph.replay()
            assert torch.equal(got, want)
    assert len(lin._counters.by_capture) == lin._counters.CAPTURES


# a layer's first call on one stream and the next on another, while the first stream is still busy
@pytest.mark.parametrize("captured", [False, True])
def test_int4_layer_first_used_on_a_busy_stream(captured):
    x = torch.randn(16, 1024, device=DEV, dtype=torch.bfloat16)
    want, lin, busy = _int4_layer()(x), _int4_layer(), torch.cuda.Stream()
    a = torch.randn(4096, 4096, device=DEV)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        for _ in range(20):
            a = a @ a * 1e-2
        first = lin(x)
    if captured:
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.stream(side):
            graph.capture_begin(capture_error_mode="thread_local")
            second = lin(x)
            graph.capture_end()
            graph.replay()
        side.synchronize()
    else:
        second = lin(x)
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want)
    assert torch.equal(copy.deepcopy(lin)(x), want) and torch.equal(lin(x), want)


# calls of one layer on two streams, eager and captured, run at the same time
@pytest.mark.parametrize("rows", [16, 20])
def test_int4_layer_on_two_streams(rows):
    torch.manual_seed(rows)
    lin = _int4_layer()
    xs = [torch.randn(rows, 1024, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    want = [lin(x) for x in xs]
    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    graphs = []
    for x in xs:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [lin(x) for _ in range(20)]
        graphs.append((graph, outs))
    torch.cuda.synchronize()
    eager = [[], []]
    for _ in range(20):
        for x, stream, keep in zip(xs, streams, eager):
            with torch.cuda.stream(stream):
                keep.append(lin(x))
    torch.cuda.synchronize()
    for (graph, _), stream in zip(graphs, streams):
        with torch.cuda.stream(stream):
            graph.replay()
    torch.cuda.synchronize()
    for w, a, (_, b) in zip(want, eager, graphs):
        assert all(torch.equal(y, w) for y in a + b)
    _lib.assert_device_ok()


# the entry points that take an accumulator instead of parts: same bits, accumulator and counters left zero
@pytest.mark.parametrize("M,K,N,splits", [(5, 512, 1024, 0), (40, 1024, 384, 4), (130, 384, 256, 3), (7, 256, 256, 1)])
@pytest.mark.parametrize("wa", [False, True])
def test_int4_gemm_entry_points_with_an_accumulator(M, K, N, splits, wa):
    torch.manual_seed(M)
    L = _lib.lib()
    lin = Int4Linear(torch.randn(N, K) * 0.05, torch.randn(N) * 0.1, 128).to(DEV)
    lin.kernel = "wa" if wa else "wb"
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    want = lin(x, splits=splits)
    acc = torch.zeros(M, N, device=DEV)
    counters = torch.zeros(L.cgk_int4_gemm_counters(M, N), dtype=torch.int32, device=DEV)
    run = L.cgk_int4_wa_gemm if wa else L.cgk_int4_gemm
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    args = lambda a, c, s: (x.data_ptr(), K, lin._tiles[wa].data_ptr(), a, c, out.data_ptr(), N, lin.bias.data_ptr(), M, N, K, s, _lib.stream_ptr())
    for _ in range(2):
        out.zero_()
        _lib.check(run(*args(acc.data_ptr(), counters.data_ptr(), splits)))
        assert torch.equal(out, want) and not acc.any() and not counters.any()
    _lib.check(run(*args(None, None, 0)))                     # whole tiles
    # the same terms in another order: fp32 sums of K products, then the rounding to bf16
    assert ((out.float() - want.float()).norm() / want.float().norm()).item() < 2 ** -8
    assert run(*args(None, None, 2)) < 0                      # parts without a place for them
    _lib.assert_device_ok()


@pytest.mark.parametrize("n,group", [(8, 8), (1024, 32), (8 * 1031, 8), (128 * 999, 128), (24 * 100, 24)])
def test_int4_dequantize_by_words(n, group):
    p, s = quantize_int4(torch.randn(n), group)
    got = dequantize_int4(p.to(DEV), s.to(DEV), n, group, torch.bfloat16).cpu()
    assert torch.equal(got, dequantize_int4(p, s, n, group).bfloat16())


@pytest.mark.parametrize("rows", [258, 513])
def test_int4_linear_many_rows_goes_through_the_dense_product(rows):
    torch.manual_seed(rows)
    lin = Int4Linear(torch.randn(384, 256) * 0.05, torch.randn(384) * 0.1, 128).to(DEV)
    x = torch.randn(3, rows // 3, 256, device=DEV, dtype=torch.bfloat16)
    ref = (x.double() @ lin.dequantized(torch.bfloat16).double() + lin.bias.double())
    assert ((lin(x).double() - ref).abs() <= ref.abs() * 2 ** -8 + 1e-4).all()          # bf16 result of fp32 sums
    assert ((lin.forward_f32(x).double() - ref).abs() <= 256 * 2 ** -24 * 8 + 1e-5).all()   # fp32 sums of 256 products
    out = torch.empty(x.shape[0] * x.shape[1], 384, device=DEV, dtype=torch.bfloat16)
    assert lin(x, out=out).data_ptr() == out.data_ptr() and torch.equal(out.view_as(lin(x)), lin(x))


@pytest.mark.parametrize("D,group,Hk,Hq,Tq", [(128, 32, 2, 8, 5), (64, 16, 1, 4, 1), (128, 128, 2, 2, 3),
                                                 (128, 64, 2, 16, 5), (128, 32, 1, 4, 40), (128, 16, 1, 2, 2)])
def test_kv_append_and_attention_match_host(D, group, Hk, Hq, Tq):
    torch.manual_seed(D + Tq)
    B, hist = 3, 150
    gpu = PagedKVCacheInt4(2, B, 256, Hk, D, group, page_size=16, device=DEV)
    cpu = PagedKVCacheInt4(2, B, 256, Hk, D, group, page_size=16)
    perm = torch.randperm(gpu.page_table.numel()).view_as(gpu.page_table).int()
    gpu.page_table.copy_(perm); cpu.page_table.copy_(perm)
    k, v = torch.randn(B, hist, Hk, D).bfloat16(), torch.randn(B, hist, Hk, D).bfloat16()
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(1, k.to(d), v.to(d))
        c.commit(torch.tensor([hist, hist - 7, hist - 33], dtype=torch.int32, device=d))
    assert torch.equal(gpu.k_pages[1].cpu(), cpu.k_pages[1]) and torch.equal(gpu.v_scales[1].cpu(), cpu.v_scales[1])
    kn, vn, q = (torch.randn(B, Tq, h, D).bfloat16() for h in (Hk, Hk, Hq))
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(1, kn.to(d), vn.to(d))
    for splits in (1, 4):
        got = gpu.attention(1, q.to(DEV), splits=splits).float().cpu()
        ref = cpu.attention(1, q.float())
        assert (got - ref).abs().max().item() < 2e-2
    _lib.assert_device_ok()


@pytest.mark.parametrize("D,group,Hk,T", [(128, 32, 2, 5), (64, 8, 3, 1), (128, 128, 1, 7), (64, 16, 1, 3), (64, 64, 5, 9)])
def test_kv_append_of_strided_rows(D, group, Hk, T):
    torch.manual_seed(D + T)
    B = 3
    one, two = (PagedKVCacheInt4(1, B, 64, Hk, D, group, page_size=16, device=DEV) for _ in range(2))
    lengths = torch.tensor([0, 11, 30], dtype=torch.int32, device=DEV)
    for c in (one, two):
        c.commit(lengths)
    qkv = torch.randn(B, T, 2 * Hk + 4, D, device=DEV).bfloat16()
    qkv[0, 0, 4] = 0.0                                         # a group of zeros has scale 1
    k, v = qkv[:, :, 4:4 + Hk], qkv[:, :, 4 + Hk:]
    one.append(0, k, v)
    kept = two.append_rows(0, k, v, want=True)
    for x, y in zip((one.k_pages, one.v_pages, one.k_scales, one.v_scales), (two.k_pages, two.v_pages, two.k_scales, two.v_scales)):
        assert torch.equal(x[0], y[0])
    for b in range(B):
        held = two.gather(0, b, int(lengths[b]) + T)
        for h, kt in zip(held, kept):
            assert torch.equal(h[int(lengths[b]):].bfloat16(), kt[b])
    assert two.append_rows(0, k[..., ::2], v[..., ::2]) is None
    _lib.assert_device_ok()


# up to 32 query rows per kv head: one and two row tiles with rows that are padding, a history of less than a block, of blocks that cross pages,
# of more blocks per warp than it holds pages for, more CTAs per head than blocks; rows read out of a packed projection
@pytest.mark.parametrize("group,page,Hk,Hq,Tq,hist", [(32, 64, 2, 2, 1, 0), (32, 16, 2, 8, 1, 15), (64, 20, 1, 8, 2, 150), (128, 48, 3, 12, 5, 333), (32, 64, 1, 4, 8, 4999),
                                                      (32, 64, 1, 17, 1, 2100), (64, 7, 2, 8, 8, 64)])
def test_kv_attention_of_few_rows(group, page, Hk, Hq, Tq, hist):
    torch.manual_seed(hist + Tq)
    B, D, room = 2, 128, hist + 64
    gpu = PagedKVCacheInt4(1, B, room, Hk, D, group, page_size=page, device=DEV)
    cpu = PagedKVCacheInt4(1, B, room, Hk, D, group, page_size=page)
    perm = torch.randperm(gpu.page_table.numel()).view_as(gpu.page_table).int()
    gpu.page_table.copy_(perm); cpu.page_table.copy_(perm)
    kn, vn = (torch.randn(B, Tq, Hk, D).bfloat16() for _ in range(2))
    packed = torch.randn(B, Tq, Hq + 3, D).bfloat16()
    k, v = (torch.randn(B, hist, Hk, D).bfloat16() for _ in range(2))
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        if hist:
            c.append(0, k.to(d), v.to(d))
            c.commit(torch.tensor([hist, hist // 3], dtype=torch.int32, device=d))
        c.append(0, kn.to(d), vn.to(d))
    ref, q = cpu.attention(0, packed[:, :, 2:2 + Hq].float()), packed.to(DEV)[:, :, 2:2 + Hq]
    for splits in (1, 3, 8, 0):
        got = gpu.attention(0, q, splits=splits)
        # K, V and P are rounded to bf16 (2^-9 each), the results as well
        assert ((got.float().cpu() - ref).norm() / ref.norm()).item() < 2 ** -7
        assert torch.equal(got, gpu.attention(0, q.contiguous(), splits=splits))
    _lib.assert_device_ok()


# a head's keys shared by up to 16 CTAs: parts that are all empty but one, a last block of few keys, histories of other lengths side by side,
# and more CTAs than there are rows to write
@pytest.mark.parametrize("Hk,Hq,Tq", [(1, 4, 1), (2, 8, 5), (1, 1, 1), (1, 32, 1)])
@pytest.mark.parametrize("hist", [0, 40, 1030, 4500])
def test_kv_attention_shared_by_many_ctas(Hk, Hq, Tq, hist):
    torch.manual_seed(hist + Hq)
    B, D = 2, 128
    gpu = PagedKVCacheInt4(1, B, hist + 64, Hk, D, 32, page_size=64, device=DEV)
    cpu = PagedKVCacheInt4(1, B, hist + 64, Hk, D, 32, page_size=64)
    kn, vn, q = (torch.randn(B, Tq, h, D).bfloat16() for h in (Hk, Hk, Hq))
    k, v = (torch.randn(B, hist, Hk, D).bfloat16() for _ in range(2))
    q[0] *= 4                                                  # a few keys hold the mass of one sequence
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        if hist:
            c.append(0, k.to(d), v.to(d))
            c.commit(torch.tensor([hist, hist // 5], dtype=torch.int32, device=d))
        c.append(0, kn.to(d), vn.to(d))
    ref, q = cpu.attention(0, q.float()), q.to(DEV)
    for splits in (5, 8, 12, 16, 40, 0):
        got = gpu.attention(0, q, splits=splits)
        # a score of the first sequence is a sum of products with deviation 4: rounding K to bf16 (2^-9 of each product at most) moves it,
        # and so its key's weight by that share, by 4 * 2^-9 = 2^-7 in the mean square; V, P and the results are rounded too (2^-9 each)
        assert ((got.float().cpu() - ref).norm() / ref.norm()).item() < 2 ** -6
        assert torch.equal(got, gpu.attention(0, q, splits=splits))
    _lib.assert_device_ok()


# contiguous queries whose strides or address the kernel cannot use as they are: a dimension of length 1 with the stride of another one, an odd place in a buffer
@pytest.mark.parametrize("B,Tq", [(2, 1), (1, 3)])
def test_kv_attention_of_contiguous_queries_with_unusual_strides(B, Tq):
    torch.manual_seed(B)
    Hk, Hq, D = 2, 8, 128
    cache = PagedKVCacheInt4(1, B, 64, Hk, D, 32, page_size=16, device=DEV)
    cache.append(0, *(torch.randn(B, 30, Hk, D, device=DEV).bfloat16() for _ in range(2)))
    cache.commit(27)
    q = torch.randn(B, Tq, Hq, D, device=DEV).bfloat16()
    want = cache.attention(0, q)
    if Tq == 1:
        odd = q[:, 0].unsqueeze(-1).permute(0, 3, 1, 2)         # 'b h d 1 -> b 1 h d'
        assert odd.is_contiguous() and odd.stride(1) == 1
    else:
        odd = torch.empty(q.numel() + 8, device=DEV, dtype=q.dtype)[1:q.numel() + 1].view_as(q).copy_(q)
        assert odd.is_contiguous() and odd.data_ptr() % 16
    assert torch.equal(cache.attention(0, odd), want)
    _lib.assert_device_ok()


# pools on smaller boundaries than the few-row kernel's copies: its rule leaves them to the kernels that read single scales, or words
@pytest.mark.parametrize("group", [32, 64, 128])
@pytest.mark.parametrize("pages,scales", [(0, 4), (0, 8), (8, 0), (4, 4)])
@pytest.mark.parametrize("Tq", [3, 5])
def test_kv_attention_of_pools_on_small_boundaries(group, pages, scales, Tq):
    torch.manual_seed(group + pages)
    B, hist, Hk, Hq, D = 2, 150, 2, 8, 128
    gpu = PagedKVCacheInt4(1, B, 256, Hk, D, group, page_size=16, device=DEV)
    cpu = PagedKVCacheInt4(1, B, 256, Hk, D, group, page_size=16)

    def moved(t, by):                                          # the same pool, `by` bytes off a boundary of 256
        room = torch.empty(t.numel() + 64, dtype=t.dtype, device=t.device)
        return room[by // t.element_size():][:t.numel()].view_as(t).copy_(t)
    for pools, by in ((gpu.k_pages, 0), (gpu.v_pages, pages), (gpu.k_scales, scales), (gpu.v_scales, scales)):
        pools[0] = moved(pools[0], by)
    k, v = (torch.randn(B, hist, Hk, D).bfloat16() for _ in range(2))
    kn, vn, q = (torch.randn(B, Tq, h, D).bfloat16() for h in (Hk, Hk, Hq))
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(0, k.to(d), v.to(d))
        c.commit(torch.tensor([hist, hist - 41], dtype=torch.int32, device=d))
        c.append(0, kn.to(d), vn.to(d))
    ref = cpu.attention(0, q.float())
    for splits in (1, 3, 0):
        got = gpu.attention(0, q.to(DEV), splits=splits).float().cpu()
        # K, V and P are rounded to bf16 (2^-9 each), the results as well
        assert ((got - ref).norm() / ref.norm()).item() < 2 ** -7
    _lib.assert_device_ok()


def test_kv_attention_long_history_many_key_blocks():
    torch.manual_seed(3)
    B, hist, Hk, Hq, D, Tq = 2, 700, 2, 8, 128, 5
    gpu = PagedKVCacheInt4(1, B, 1024, Hk, D, 32, page_size=32, device=DEV)
    cpu = PagedKVCacheInt4(1, B, 1024, Hk, D, 32, page_size=32)
    k, v = torch.randn(B, hist, Hk, D).bfloat16(), torch.randn(B, hist, Hk, D).bfloat16()
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(0, k.to(d), v.to(d))
        c.commit(torch.tensor([hist, hist - 301], dtype=torch.int32, device=d))
    kn, vn, q = (torch.randn(B, Tq, h, D).bfloat16() for h in (Hk, Hk, Hq))
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(0, kn.to(d), vn.to(d))
    ref = cpu.attention(0, q.float())
    for splits in (1, 3, 0):
        got = gpu.attention(0, q.to(DEV), splits=splits).float().cpu()
        assert (got - ref).abs().max().item() < 2e-2
    _lib.assert_device_ok()


# more than 32 rows per kv head: the tcgen05 kernel over many blocks of 128 keys, one and two passes over the rows
@pytest.mark.parametrize("Tq", [9, 20])
def test_kv_attention_of_more_rows_over_many_key_blocks(Tq):
    torch.manual_seed(Tq)
    B, hist, Hk, Hq, D = 2, 1500, 2, 8, 128
    gpu = PagedKVCacheInt4(1, B, 1600, Hk, D, 32, page_size=32, device=DEV)
    cpu = PagedKVCacheInt4(1, B, 1600, Hk, D, 32, page_size=32)
    k, v = (torch.randn(B, hist, Hk, D).bfloat16() for _ in range(2))
    kn, vn, q = (torch.randn(B, Tq, h, D).bfloat16() for h in (Hk, Hk, Hq))
    for c, d in ((gpu, DEV), (cpu, "cpu")):
        c.append(0, k.to(d), v.to(d))
        c.commit(torch.tensor([hist, hist - 801], dtype=torch.int32, device=d))
        c.append(0, kn.to(d), vn.to(d))
    ref = cpu.attention(0, q.float())
    for splits in (1, 3, 0):
        got = gpu.attention(0, q.to(DEV), splits=splits).float().cpu()
        # K, V and P are rounded to bf16 (2^-9 each), the results as well
        assert ((got - ref).norm() / ref.norm()).item() < 2 ** -7
    _lib.assert_device_ok()


def test_sampling_matches_filtered_distribution():
    torch.manual_seed(1)
    V, rows = 32000, 4
    logits = torch.randn(rows, V) * 3
    for temp, k, p in ((1.0, 50, 0.9), (0.7, 8, 1.0), (1.3, 0, 0.5), (0.0, 50, 0.9)):
        tok, probs = sample(logits.to(DEV), temp, k, p, seed=5, step=0, return_probs=True)
        ref = filtered_probs(logits, temp, k, p)
        assert torch.allclose(probs.cpu(), ref, atol=2e-5), (temp, k, p)
        assert (ref.gather(1, tok.cpu().long()[:, None]) > 0).all()
    counts = torch.zeros(rows, V)
    step = torch.zeros(1, dtype=torch.int64, device=DEV)
    lg = logits.to(DEV).bfloat16()
    ref = filtered_probs(lg.float().cpu(), 1.0, 8, 1.0)
    for i in range(1500):
        step.fill_(i)
        counts.scatter_add_(1, sample(lg, 1.0, 8, 1.0, seed=9, step=step).cpu().long()[:, None], torch.ones(rows, 1))
    assert (counts / 1500 - ref).abs().max().item() < 0.05
    # different rows and steps draw from different streams
    same = torch.zeros(64, 1000, device=DEV)
    toks = sample(same, 1.0, 0, 1.0, seed=1, step=3)
    assert toks.unique().numel() > 32


# 32 768 keys fit the registers, 81 920 registers and shared memory; up to 512 wanted values are found through the threads' maxima
@pytest.mark.parametrize("V", [1, 31, 1023, 1025, 32768, 32769, 50257, 81920, 81923])
@pytest.mark.parametrize("k", [1, 2, 33, 512, 513, 0])
def test_sampling_selection_at_its_edges(V, k):
    g = torch.Generator().manual_seed(V * 7 + k)
    spread = torch.randn(2, V, generator=g) * 3
    crowded = spread.clone()
    crowded[:, (torch.arange(V) % 1024) < 40] += 30.0          # 40 threads hold all large values: more than 1024 reach the bound at long rows
    for x in (spread, crowded):
        for t in (x, x.bfloat16()):
            if t.dtype != torch.float32 and (k == 0 or x is crowded):
                continue                                       # bf16 values tie at the threshold, where the general way takes any of them
            tok, probs = sample(t.to(DEV), 0.8, k, 0.9, seed=3, step=1, return_probs=True)
            ref = filtered_probs(t, 0.8, k, 0.9)
            # the kernel's sums of up to 1024 probabilities run in another order than the oracle's: a value whose mass ends
            # within 1024 * 2^-24 of the nucleus may be in or out, which moves every other value by at most its own mass
            edge = ((ref > 0) != (probs.cpu() > 0)).sum().item()
            assert edge <= 2 and (edge or torch.allclose(probs.cpu(), ref, atol=2e-5))
            assert (probs.cpu().gather(1, tok.cpu().long()[:, None]) > 0).all()


# the distribution may take the place of its logits: rows kept in registers, in shared memory too, and read again
@pytest.mark.parametrize("V", [1000, 32000, 50257, 90000])
@pytest.mark.parametrize("k", [50, 0])
def test_sampling_in_place(V, k):
    torch.manual_seed(V + k)
    x = torch.randn(5, V, device=DEV) * 3
    step = torch.tensor([2], device=DEV)
    want_tok, want = sample(x, 0.8, k, 0.9, seed=3, step=step, return_probs=True)
    tok = torch.empty(5, dtype=torch.int32, device=DEV)
    _lib.check(_lib.lib().cgk_sample(x.data_ptr(), 0, V, 5, V, 0.8, k, 0.9, 3, step.data_ptr(), tok.data_ptr(), x.data_ptr(), _lib.stream_ptr()))
    assert torch.equal(tok, want_tok) and torch.equal(x, want)


def test_sampling_takes_the_first_of_equal_values():
    x = torch.zeros(1, 1000)
    x[0, [5, 900, 17]] = 1.0
    _, probs = sample(x.to(DEV), 1.0, 4, 1.0, return_probs=True)
    assert probs[0].nonzero().view(-1).tolist() == [0, 5, 17, 900]


# logits are selected as they are and only the few near the bound are divided by the temperature: the tokens kept are those of the
# quotients, the first of equal ones, also where neighbours fall together (rounding, subnormal quotients, overflow) or are no numbers (of more than 1024 equal ones, any are kept)
@pytest.mark.parametrize("V", [33, 1000, 32000, 50257])
@pytest.mark.parametrize("temperature", [0.7, 1.0, 3.0, 1e-6, 1e6, 1e30, 1e-40])
@pytest.mark.parametrize("kind", ["normal", "neighbours", "zeros", "tiny", "huge", "negative", "nan"])
def test_sampling_keeps_the_largest_quotients(V, temperature, kind):
    g = torch.Generator().manual_seed(V)
    x = torch.randn(3, V, generator=g)
    if kind == "neighbours":                                   # 16 neighbouring floats, many times each
        x = (torch.randint(0, 16, (3, V), generator=g, dtype=torch.int32) + 0x40490000).view(torch.float32)
    elif kind == "zeros":
        x[:, 3:] = torch.where(torch.rand(3, V - 3, generator=g) < 0.5, 0.0, -1.0)
    elif kind == "tiny":
        x = x * 1e-39
    elif kind == "huge":
        x = x * 1e38
    elif kind == "negative":
        x = -x.abs() * 1e37
        x[:, ::3] = float("-inf")
    elif kind == "nan":
        x[:, V // 2], x[:, 1] = float("nan"), float("-inf")
    x = x.to(DEV)
    k, t = 9, torch.tensor(temperature, device=DEV)
    quotient = x / t
    if kind == "nan":                                          # no number comes behind all numbers
        quotient[:, V // 2] = float("-inf")
    if V > 1024 and any(int((q == q.sort(descending=True)[0][k - 1]).sum()) > 512 for q in quotient):
        pytest.skip("more equal values than are ranked")
    quotient = torch.where((quotient == 0) & quotient.signbit(), -1e-45, quotient)     # a negative zero comes behind the others
    order = torch.sort(quotient, dim=-1, descending=True, stable=True)[1][:, :k]
    _, probs = sample(x, temperature, k, 1.0, return_probs=True)
    for r in range(3):
        best = quotient[r, order[r, 0]]
        if not torch.isfinite(best):                           # a sum of infinities or NaN: no distribution to compare
            continue
        want = torch.softmax(quotient[r, order[r]].double(), 0)
        assert (probs[r].nonzero().view(-1).tolist() == sorted(order[r][want.float() > 0].tolist()))
        assert (probs[r, order[r]].double() - want).abs().max() < 1e-6
    _lib.assert_device_ok()


# as many wanted as there are, minus infinity among them: the bound's 20 bits lie below its key
def test_sampling_keeps_minus_infinity_when_all_are_wanted():
    x = torch.tensor([[1.0, float("-inf"), 3.0, float("-inf"), 2.0]])
    tok, probs = sample(x.to(DEV), 0.5, 5, 1.0, return_probs=True)
    assert torch.allclose(probs.cpu(), torch.softmax(x / 0.5, -1))


def test_spec_accept_rule_and_commit():
    B, g, V = 64, 4, 512
    torch.manual_seed(2)
    q = torch.softmax(torch.randn(B, g, V), -1)
    p = torch.softmax(torch.randn(B, g + 1, V), -1)
    draft = torch.multinomial(q.view(-1, V), 1).view(B, g).int()
    # identical distributions: everything is accepted and a bonus token follows
    lengths = torch.full((B,), 10, dtype=torch.int32, device=DEV)
    stats = torch.zeros(2, dtype=torch.int32, device=DEV)
    pp = torch.cat([q, p[:, -1:]], 1)
    n, out = spec_accept(draft.to(DEV), q.to(DEV), pp.to(DEV), seed=1, step=0, lengths=lengths, stats=stats)
    assert (n == g).all() and torch.equal(out[:, :g].cpu(), draft) and (lengths == 10 + g + 1).all()
    assert stats.tolist() == [B * g, B * g]
    # zero target probability on the drafted token: rejected at position 0, resampled where p > q
    p0 = p.clone()
    p0[torch.arange(B), 0, draft[:, 0].long()] = 0
    p0[:, 0] /= p0[:, 0].sum(-1, keepdim=True)
    n, out = spec_accept(draft.to(DEV), q.to(DEV), p0.to(DEV), seed=1, step=1)
    assert (n == 0).all()
    tok = out[:, 0].cpu().long()
    assert ((p0[torch.arange(B), 0, tok] - q[torch.arange(B), 0, tok]) > 0).all()
    # acceptance frequency = E[min(1, p/q)] at the first position
    trials, acc0 = 300, 0
    for s in range(trials):
        n, _ = spec_accept(draft.to(DEV), q.to(DEV), p.to(DEV), seed=3, step=s)
        acc0 += (n >= 1).float().mean().item()
    ratio = (p[torch.arange(B), 0, draft[:, 0].long()] / q[torch.arange(B), 0, draft[:, 0].long()]).clamp(max=1).mean().item()
    assert abs(acc0 / trials - ratio) < 0.04
    parents = torch.tensor([-1, 0, 0, 2, 1], dtype=torch.int32)
    assert torch.equal(tree_attention_mask(parents.to(DEV), 7).cpu(), tree_attention_mask(parents, 7))


def test_engine_and_speculative_decoding_on_gpu():
    rng.manual_seed(0)
    cfg = LlamaConfig(vocab_size=1024, n_layer=2, d_model=256, n_head=4, n_kv_head=2, d_ff=512, max_seq_len=256)
    target = Llama(cfg)
    B = 4
    cpu_engine = LlamaInt4Engine(target, B, 128)
    gpu_engine = LlamaInt4Engine(target.to(DEV).bfloat16(), B, 128)
    prompts = torch.randint(0, 1024, (B, 9))
    lc = cpu_engine.forward(prompts, commit=True)
    lg = gpu_engine.forward(prompts.to(DEV), commit=True).cpu()
    assert torch.nn.functional.cosine_similarity(lc.flatten(), lg.flatten(), dim=0) > 0.98
    draft_engine = LlamaInt4Engine(target, B, 128)          # same weights: all drafts accepted under greedy decoding
    sd = SpeculativeDecoder(draft_engine, gpu_engine, gamma=4, temperature=0.0)
    seqs, stats = sd.generate(prompts.to(DEV), 10)
    assert stats.acceptance_rate > 0.8 and all(len(s) >= 19 for s in seqs)   # < 1 only through bf16 near-ties
    _lib.assert_device_ok()


# the decoding step is captured after the first prompts; prompts of other lengths then run other kernels and larger ones
def test_speculative_decoding_over_prompts_of_other_lengths():
    rng.manual_seed(1)
    cfg = LlamaConfig(vocab_size=1024, n_layer=2, d_model=512, n_head=8, n_kv_head=4, d_ff=1024, max_seq_len=256)
    target, draft = Llama(cfg).to(DEV).bfloat16(), Llama(cfg).to(DEV).bfloat16()
    B = 4
    decoder = lambda: SpeculativeDecoder(LlamaInt4Engine(draft, B, 160), LlamaInt4Engine(target, B, 160), gamma=4, temperature=0.0)
    sd = decoder()
    for length in (100, 10, 40, 15, 100):                     # 396 rows through the dense product, 36 and 156 rows, 14 tokens over the cache
        prompts = torch.randint(0, 1024, (B, length), device=DEV)
        got, _ = sd.generate(prompts, 12)
        assert sd._graph is not None
        fresh = decoder()
        want, _ = fresh.generate(prompts, 12)
        fresh.close()
        assert got == want
    sd.close()
    _lib.assert_device_ok()


# a captured attention call gives the same after a later one that needs more (few rows: no scratch to keep)
def test_kv_attention_captured_before_a_larger_call():
    torch.manual_seed(5)
    B, Hk, Hq, D = 2, 2, 8, 128
    cache = PagedKVCacheInt4(1, B, 512, Hk, D, 32, page_size=64, device=DEV)
    cache.append(0, *(torch.randn(B, 420, Hk, D, device=DEV).bfloat16() for _ in range(2)))
    cache.commit(400)
    q, more = torch.randn(B, 1, Hq, D, device=DEV).bfloat16(), torch.randn(B, 20, Hq, D, device=DEV).bfloat16()
    want = cache.attention(0, q)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = cache.attention(0, q)
    cache.attention(0, more)
    junk = [torch.full((n,), 1e30, device=DEV) for n in (1 << 8, 1 << 12, 1 << 14, 1 << 16, 1 << 18) for _ in range(4)]
    for _ in range(2):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
    assert all((j == 1e30).all() for j in junk)
    _lib.assert_device_ok()


# more than 32 rows per kv head: a captured call keeps its scratch although a later call needs more
def test_kv_attention_of_more_rows_captured_before_a_larger_call():
    torch.manual_seed(6)
    B, Hk, Hq, D = 2, 2, 8, 128
    cache = PagedKVCacheInt4(1, B, 512, Hk, D, 32, page_size=64, device=DEV)
    cache.append(0, *(torch.randn(B, 420, Hk, D, device=DEV).bfloat16() for _ in range(2)))
    cache.commit(400)
    q, more = (torch.randn(B, t, Hq, D, device=DEV).bfloat16() for t in (9, 20))
    want = cache.attention(0, q)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = cache.attention(0, q)
    cache.attention(0, more)
    junk = [torch.full((n,), 1e30, device=DEV) for n in (1 << 8, 1 << 12, 1 << 14, 1 << 16, 1 << 18) for _ in range(4)]
    for _ in range(2):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
    assert all((j == 1e30).all() for j in junk)
    _lib.assert_device_ok()


# in a captured pass launches overlap their predecessors, in one launched eagerly they do not: the same bits.  4 rows take the
# warp-level products and one row tile of the cache attention, 20 the tcgen05 products and two
@pytest.mark.parametrize("tokens", [1, 5])
@torch.no_grad()
def test_int4_pass_captured_and_launched_eagerly(tokens):
    rng.manual_seed(2)
    cfg = LlamaConfig(vocab_size=1024, n_layer=6, d_model=1024, n_head=8, n_kv_head=2, d_ff=2048, max_seq_len=512)
    engine = LlamaInt4Engine(Llama(cfg).to(DEV).bfloat16(), 4, 512)
    engine.forward(torch.randint(0, 1024, (4, 333), device=DEV), commit=True)
    ids = torch.randint(0, 1024, (4, tokens), device=DEV)
    want = engine.forward(ids).clone()
    assert torch.equal(engine.forward(ids), want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = engine.forward(ids)
    for _ in range(20):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)
    _lib.assert_device_ok()
