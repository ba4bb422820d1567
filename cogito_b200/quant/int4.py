"""INT4 weight quantisation and the weight-only GEMM that consumes it.

Format (bit-exact with cg_quantize_int4, src/quantize/int4.c:10-59): flat groups of
``group`` consecutive elements of the row-major tensor, ``scale = absmax / 7`` (1 when below
1e-10), ``q = clamp(round(x / scale), -8, 7)`` with halves rounded away from zero, two values
per byte with the even index in the low nibble, fp32 scales.

``Int4Linear`` keeps the weight transposed, ``[in, out]`` like the reference's
``cg_matmul_int4`` operand (src/quantize/int4.c:90-114), so that the tcgen05 kernel streams
each weight row once; on CPU the same product is computed from the dequantised weight.
"""
from __future__ import annotations

import os
import threading

import torch

from ..ops import _lib


def _round_half_away(x: torch.Tensor) -> torch.Tensor:
    return torch.sign(x) * torch.floor(torch.abs(x) + 0.5)


def quantize_int4(x: torch.Tensor, group: int = 128):
    """Returns (packed uint8 [ceil(n/2)], scales fp32 [ceil(n/group)]) of the flattened tensor."""
    if group <= 0 or group % 2:
        raise ValueError("group must be a positive even number")
    flat = x.detach().reshape(-1).float().contiguous()
    n = flat.numel()
    groups = (n + group - 1) // group
    if flat.is_cuda:
        packed = torch.zeros((n + 1) // 2, dtype=torch.uint8, device=flat.device)
        scales = torch.empty(groups, dtype=torch.float32, device=flat.device)
        _lib.check(_lib.lib().cgk_int4_quantize(flat.data_ptr(), n, group, packed.data_ptr(), scales.data_ptr(),
                                                _lib.stream_ptr()), "cgk_int4_quantize")
        _lib.count_launch()
        return packed, scales
    pad = groups * group - n
    g = torch.nn.functional.pad(flat, (0, pad)).view(groups, group)
    amax = g.abs().amax(1)
    scales = torch.where(amax < 1e-10, torch.ones_like(amax), amax / 7.0)
    q = _round_half_away(g / scales[:, None]).clamp_(-8, 7).to(torch.int16).view(-1)[:n + (n & 1)]
    if q.numel() < n + (n & 1):
        q = torch.nn.functional.pad(q, (0, n + (n & 1) - q.numel()))
    q = q & 0xF
    packed = (q[0::2] | (q[1::2] << 4)).to(torch.uint8)
    return packed, scales


def dequantize_int4(packed: torch.Tensor, scales: torch.Tensor, n: int, group: int = 128,
                    dtype: torch.dtype = torch.float32) -> torch.Tensor:
    if packed.is_cuda:
        out = torch.empty(n, dtype=dtype, device=packed.device)
        f32 = out.data_ptr() if dtype == torch.float32 else None
        b16 = out.data_ptr() if dtype == torch.bfloat16 else None
        if f32 is None and b16 is None:
            raise ValueError("dtype must be float32 or bfloat16")
        _lib.check(_lib.lib().cgk_int4_dequantize(packed.data_ptr(), scales.data_ptr(), n, group, f32, b16,
                                                  _lib.stream_ptr()), "cgk_int4_dequantize")
        _lib.count_launch()
        return out
    b = packed.to(torch.int16)
    q = torch.stack([b & 0xF, b >> 4], 1).reshape(-1)[:n]
    q = torch.where(q >= 8, q - 16, q).float()
    idx = torch.arange(n) // group
    return (q * scales[idx]).to(dtype)


class _Counters:
    """Arrival counters of the tiles that several CTAs share.  Every launch finds its own zero and leaves them zero, so launches
    that may run at the same time need different ones: a set per stream, and one per stream of a graph capture, which is not
    replaced when a later call needs more (the graph keeps its address)."""
    CAPTURES = 32                          # sets for captures; a launch captured beyond that zeroes its own inside the graph

    def __init__(self):
        self.lock = threading.Lock()
        self.by_stream, self.by_capture = {}, {}
        self.spare = None                  # [CAPTURES, the most that one launch needs]

    def __deepcopy__(self, memo):
        return _Counters()

    def __reduce__(self):
        return (_Counters, ())

    def prepare(self, most: int, device):
        """The sets for captures (``most``: counters of the largest launch); the caller holds the lock."""
        if self.spare is None or self.spare.value.device != device:
            self.by_stream, self.by_capture = {}, {}
            self.spare = _lib.Made(lambda: torch.zeros(self.CAPTURES, most, dtype=torch.int32, device=device))

    def get(self, need: int, most: int, device) -> torch.Tensor:
        stream = _lib.stream_ptr()
        if not torch.cuda.is_current_stream_capturing():
            own = self.by_stream.get(stream)
            if own is None or own.numel() < need or own.device != device:    # an older set goes back to the allocator in the stream's order
                own = self.by_stream[stream] = torch.zeros(need, dtype=torch.int32, device=device)
            return own
        if need <= most:
            key = (_lib.lib().cgk_capture_id(stream), stream)
            with self.lock:
                self.prepare(most, device)
                if key not in self.by_capture and len(self.by_capture) < self.CAPTURES:
                    self.by_capture[key] = len(self.by_capture)
                if key in self.by_capture:
                    return self.spare.here()[self.by_capture[key]]
        return torch.zeros(need, dtype=torch.int32, device=device)


class Int4Linear(torch.nn.Module):
    """y = x @ W^T (+ bias) with W stored as packed INT4 of W^T ([in, out], groups along out)."""

    # Which kernel multiplies: "wb" makes the weights the A operand of tcgen05 MMAs (converted tile in tensor
    # memory, up to 128 token rows per instruction), "wa" makes them the A operand of warp-level MMAs, fed from registers (cost
    # follows the token count; needs group % 128 == 0).  "auto": "wa" up to 16 token rows, "wb" up to two row
    # tiles, and beyond that (prompts) the weights are dequantised to bf16 once per call for the dense GEMM: "wb" converts
    # every weight tile again for each row tile.  That copy (2 bytes per weight: 180 MB for 4096 x 22016, 262 MB for
    # 4096 x 32000) comes from the allocator for the time of the call, one layer's at a time; where there is no room for it,
    # "wb" takes the call.  Each of the two kernels has its own tile-major copy of the weights, made on
    # first use; both sum the parts of a shared tile in a fixed order, so a call gives the same bits every time.
    # Times (us, layers one after the other) for 4096 x 6144, 4096 x 4096, 4096 x 22016, 11008 x 4096, 4096 x 32000, 2048 x 11264:
    #   16 rows   "wa" 8.5 6.5 20.6 10.9 25.6 10.4      "wb" 9.5 8.4 21.9 14.2 30.0 9.3
    #   17 rows   "wa" 12.5 9.0 30.9 15.6 38.6 15.3     "wb" 9.8 8.7 22.3 14.6 30.1 9.4    (four columns of MMAs instead of two)
    #   32 rows   "wa" 12.8 9.1 31.4 15.6 39.4 15.5     "wb" 10.0 8.9 22.6 15.0 30.5 9.7
    #   80 rows                                         "wb" 11.4 10.3 25.0 17.5 33.7 11.4
    #   200 rows  "wb" 19.8 14.7 44.4 27.5 63.1 18.9    dense 31.4 26.5 104 61.1 131 32.7
    # The line to the dense GEMM stays where the weights would be rounded once more than there.
    FEW_ROWS, DENSE_ROWS = 16, 256
    kernel = os.environ.get("COGITO_INT4_KERNEL", "auto")

    def __init__(self, weight: torch.Tensor, bias: torch.Tensor | None = None, group: int = 128):
        super().__init__()
        out_f, in_f = weight.shape
        if out_f % group:
            raise ValueError(f"out_features {out_f} must be a multiple of the group size {group}")
        self.in_features, self.out_features, self.group = in_f, out_f, group
        packed, scales = quantize_int4(weight.detach().t().contiguous(), group)
        self.register_buffer("packed", packed)
        self.register_buffer("scales", scales)
        self.register_buffer("bias", None if bias is None else bias.detach().to(torch.bfloat16))
        self._counters = _Counters()
        self._tiles, self._tiled = {}, {}     # kernel kind -> tile-major weights, and their making until it is known to be over

    @classmethod
    def from_packed(cls, packed: torch.Tensor, scales: torch.Tensor, in_features: int, out_features: int, group: int = 128,
                    bias: torch.Tensor | None = None) -> "Int4Linear":
        """Wraps already quantised values (of W^T, [in, out] row-major, as ``quantize_int4`` returns them),
        e.g. read from a checkpoint; nothing is re-quantised."""
        if packed.numel() != (in_features * out_features + 1) // 2 or scales.numel() != (in_features * out_features + group - 1) // group:
            raise ValueError("packed / scales do not match the layer shape and group size")
        self = cls.__new__(cls)
        torch.nn.Module.__init__(self)
        self.in_features, self.out_features, self.group = in_features, out_features, group
        self.register_buffer("packed", packed.to(torch.uint8).contiguous())
        self.register_buffer("scales", scales.to(torch.float32).contiguous())
        self.register_buffer("bias", None if bias is None else bias.detach().to(torch.bfloat16))
        self._counters = _Counters()
        self._tiles, self._tiled = {}, {}
        return self

    @classmethod
    def from_linear(cls, lin, group: int = 128) -> "Int4Linear":
        return cls(lin.weight.data, getattr(lin, "bias", None), group)

    def dequantized(self, dtype=torch.float32) -> torch.Tensor:
        """W^T as [in, out]."""
        return dequantize_int4(self.packed, self.scales, self.in_features * self.out_features, self.group, dtype) \
            .view(self.in_features, self.out_features)

    def _tile(self, wa: bool, device) -> torch.Tensor:
        """One-time tile-major reordering of the same quantised values, and the counters that captured calls will need: made
        before anything is recorded, so that a graph neither repeats the work nor owns the memory."""
        L, K, N = _lib.lib(), self.in_features, self.out_features
        nbytes, tile = (L.cgk_int4_wa_tiles_bytes, L.cgk_int4_wa_tile_weights) if wa else (L.cgk_int4_tiles_bytes, L.cgk_int4_tile_weights)

        def make():
            tiles = torch.empty(nbytes(K, N), dtype=torch.uint8, device=device)
            _lib.check(tile(self.packed.data_ptr(), self.scales.data_ptr(), K, N, self.group, tiles.data_ptr(), _lib.stream_ptr()), "cgk_int4_tile_weights")
            _lib.count_launch()
            return tiles

        with self._counters.lock:
            self._counters.prepare(L.cgk_int4_gemm_counters(self.DENSE_ROWS, N), device)
            if self._tiles.get(wa) is None or self._tiles[wa].device != device:
                made = _lib.Made(make)
                self._tiled[wa], self._tiles[wa] = made, made.value
            return self._tiles[wa]

    def _takes_dense(self, rows: int, splits: int = 0) -> bool:
        return self.kernel == "auto" and splits == 0 and rows > self.DENSE_ROWS

    def _dense(self, x2, **kw):
        from ..ops.gemm import gemm
        return gemm(x2.to(torch.bfloat16).contiguous(), self.dequantized(torch.bfloat16), b_mn=True, bias=self.bias, **kw)

    def forward_f32(self, x: torch.Tensor) -> torch.Tensor:
        """fp32 result (logits); the result leaves the GEMM in fp32 without a bf16 copy in between."""
        rows = x.numel() // self.in_features
        if x.is_cuda and self._takes_dense(rows):
            try:
                return self._dense(x.reshape(rows, self.in_features), out_dtype=torch.float32).view(*x.shape[:-1], self.out_features)
            except torch.OutOfMemoryError:
                pass                                       # no room for the weights in bf16: by the streaming kernel
        if x.is_cuda and 0 < rows <= self.DENSE_ROWS and self._streams():
            return self._stream(x.reshape(rows, self.in_features), f32=True).view(*x.shape[:-1], self.out_features)
        return self.forward(x).float()

    def forward(self, x: torch.Tensor, splits: int = 0, out: torch.Tensor | None = None, f32: bool = False) -> torch.Tensor:
        """``out``: an optional contiguous [rows, out_features] buffer for the result (bf16 on CUDA),
        e.g. a slot of symmetric memory that a collective kernel reads next.  ``f32``: the result of ``forward_f32``."""
        if f32:
            if out is not None or splits:
                raise ValueError("an fp32 result takes neither out nor splits")
            return self.forward_f32(x)
        lead = x.shape[:-1]
        x2 = x.reshape(-1, self.in_features)
        M = x2.shape[0]

        def done(y):
            if out is None:
                return y.view(*lead, self.out_features)
            out.copy_(y.view(out.shape))
            return out.view(*lead, self.out_features)

        if not x2.is_cuda:
            y = x2.float() @ self.dequantized()
            if self.bias is not None:
                y = y + self.bias.float()
            return done(y.to(x.dtype))
        N, K = self.out_features, self.in_features
        if not self._streams():
            return done(self._dense(x2))
        if self._takes_dense(M, splits):
            if out is not None and (out.dtype != torch.bfloat16 or not out.is_contiguous() or out.numel() != M * N):
                raise ValueError("out must be a contiguous bf16 [rows, out_features] tensor")
            try:
                return self._dense(x2, out=None if out is None else out.view(M, N)).view(*lead, N)
            except torch.OutOfMemoryError:
                pass                                       # no room for the weights in bf16: by the streaming kernel
        return self._stream(x2, splits, out).view(*lead, N)

    def _streams(self) -> bool:
        """A shape that the streaming kernels cover; for others the weights are dequantised, then the bf16 GEMM."""
        return self.out_features % 128 == 0 and self.in_features % 64 == 0 and self.group % 64 == 0

    def _streams_few(self, rows: int) -> bool:
        """"wa" (needs one scale per k for a 128-feature tile)."""
        return (self.kernel == "wa" or (self.kernel == "auto" and rows <= self.FEW_ROWS)) and self.group % 128 == 0 \
            and self.in_features % 128 == 0 and self.out_features % 128 == 0

    def _stream(self, x2: torch.Tensor, splits: int = 0, out: torch.Tensor | None = None, f32: bool = False) -> torch.Tensor:
        """[rows, in] through "wa" or "wb"; ``f32``: an fp32 result."""
        x2 = x2.to(torch.bfloat16).contiguous()
        L = _lib.lib()
        M, N, K = x2.shape[0], self.out_features, self.in_features
        wa = self._streams_few(M)
        tiles = self._tiles.get(wa)
        if tiles is None or tiles.device != x2.device:
            tiles = self._tile(wa, x2.device)
        made = self._tiled.get(wa)
        if made is not None:
            made.here()
            if made.event is None:
                self._tiled.pop(wa, None)
        # for the output tiles that several CTAs share: a place for their parts (of this call alone), and counters
        parts = torch.empty((L.cgk_int4_wa_gemm_parts_floats if wa else L.cgk_int4_gemm_parts_floats)(M, N, K, splits), dtype=torch.float32, device=x2.device)
        counters = self._counters.get(L.cgk_int4_gemm_counters(M, N), L.cgk_int4_gemm_counters(self.DENSE_ROWS, N), x2.device)
        if out is None:
            out = torch.empty(M, N, dtype=torch.float32 if f32 else torch.bfloat16, device=x2.device)
        elif out.dtype != torch.bfloat16 or not out.is_contiguous() or out.numel() != M * N:
            raise ValueError("out must be a contiguous bf16 [rows, out_features] tensor")
        if wa:
            entry = L.cgk_int4_wa_gemm_parts_f32 if f32 else L.cgk_int4_wa_gemm_parts
        else:
            entry = L.cgk_int4_gemm_parts_f32 if f32 else L.cgk_int4_gemm_parts
        _lib.check(entry(x2.data_ptr(), K, tiles.data_ptr(), parts.data_ptr(), counters.data_ptr(),
                         out.data_ptr(), N, _lib.ptr(self.bias), M, N, K, splits, _lib.stream_ptr()), "cgk_int4_gemm")
        _lib.count_launch()
        return out
