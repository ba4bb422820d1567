// Rotary position embedding, rotate-half convention (element i pairs with
// i + D/2), applied in place to a strided bf16 or fp32 tensor [B, T, H, D].
// The backward pass is the same kernel with the sine negated.
//
// Reference counterparts: rope_kernel (src/cuda/flash_attn_kernels.c:216-249),
// the host backward (:656-682) and cg_rope_precompute_freqs
// (src/attention/flash_attn.c:318-362): cos/sin tables of shape [max_seq, D/2]
// with angle = pos * theta^(-2i/D).
#include "../../include/cogito_kernels.h"
#include "host_common.h"
#include "sm100.cuh"

namespace cgk {

__global__ void rope_table_kernel(float* __restrict__ cos_t, float* __restrict__ sin_t, int max_seq,
                                  int half, float theta) {
  const long long n = (long long)max_seq * half;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int pos = (int)(i / half), j = (int)(i % half);
    const float freq = powf(theta, -2.0f * (float)j / (float)(2 * half));
    float s, c;
    sincosf((float)pos * freq, &s, &c);
    cos_t[i] = c;
    sin_t[i] = s;
  }
}

template <typename T>
__device__ __forceinline__ float rd(const T* p);
template <> __device__ __forceinline__ float rd<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float rd<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T>
__device__ __forceinline__ void wr(T* p, float v);
template <> __device__ __forceinline__ void wr<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void wr<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }

// positions: int32 [B, T] or null (then position = pos_offset + t).
template <typename T>
__global__ void rope_apply_kernel(T* x, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                  const int* __restrict__ positions, int B, int Tn, int H, int D,
                                  long long bs, long long ts, long long hs, int pos_offset,
                                  int max_seq, float sign) {
  const int half = D / 2;
  const long long n = (long long)B * Tn * H * half;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int j = (int)(i % half);
    long long r = i / half;
    const int h = (int)(r % H); r /= H;
    const int t = (int)(r % Tn);
    const int b = (int)(r / Tn);
    int pos = positions ? positions[(long long)b * Tn + t] : pos_offset + t;
    if (pos < 0) pos = 0;
    if (pos >= max_seq) pos = max_seq - 1;
    const float c = cos_t[(long long)pos * half + j], s = sign * sin_t[(long long)pos * half + j];
    T* p = x + b * bs + t * ts + h * hs;
    const float a = rd<T>(p + j), bb = rd<T>(p + j + half);
    wr<T>(p + j, a * c - bb * s);
    wr<T>(p + j + half, bb * c + a * s);
  }
}

// bf16 rows whose halves are multiples of 8 elements on 16-byte boundaries: eight pairs per thread, two 16-byte loads and stores, and
// the row's index worked out once (three 64-bit divisions per pair of elements bound the kernel above).
__global__ void __launch_bounds__(256)
rope_apply_vec_kernel(__nv_bfloat16* x, const float* __restrict__ cos_t, const float* __restrict__ sin_t, const int* __restrict__ positions,
                      int units, int Tn, int H, int half, long long bs, long long ts, long long hs, int pos_offset, int max_seq, float sign) {
  const int u = blockIdx.x * 256 + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (u >= units) return;
  const int upr = half >> 3, row = u / upr, j = (u - row * upr) * 8, bt = row / H, h = row - bt * H, b = bt / Tn, t = bt - b * Tn;
  int pos = positions ? positions[bt] : pos_offset + t;
  if (pos < 0) pos = 0;
  if (pos >= max_seq) pos = max_seq - 1;
  const float4* cp = reinterpret_cast<const float4*>(cos_t + (long long)pos * half + j);
  const float4* sp = reinterpret_cast<const float4*>(sin_t + (long long)pos * half + j);
  const float4 c0 = __ldg(cp), c1 = __ldg(cp + 1), s0 = __ldg(sp), s1 = __ldg(sp + 1);
  __nv_bfloat16* p = x + b * bs + t * ts + h * hs + j;
  const uint4 lo = *reinterpret_cast<const uint4*>(p), hi = *reinterpret_cast<const uint4*>(p + half);
  const uint32_t lw[4] = {lo.x, lo.y, lo.z, lo.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w};
  const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
  uint32_t lr[4], hr[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 a = unpack_bf16x2(lw[e]), bb = unpack_bf16x2(hw[e]);
    const float ca = cs[2 * e], cb = cs[2 * e + 1], sa = sign * sn[2 * e], sb = sign * sn[2 * e + 1];
    // the contractions of rope_apply_kernel, written out: the same bits
    lr[e] = pack_bf16x2(fmaf(a.x, ca, -(bb.x * sa)), fmaf(a.y, cb, -(bb.y * sb)));
    hr[e] = pack_bf16x2(fmaf(a.x, sa, bb.x * ca), fmaf(a.y, sb, bb.y * cb));
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(lr[0], lr[1], lr[2], lr[3]);
  *reinterpret_cast<uint4*>(p + half) = make_uint4(hr[0], hr[1], hr[2], hr[3]);
}

}  // namespace cgk

using namespace cgk;

CGK_API int cgk_rope_table(float* cos_t, float* sin_t, int max_seq, int head_dim, float theta,
                           void* stream) {
  CGK_REQUIRE(cos_t && sin_t && head_dim % 2 == 0 && max_seq > 0, "cgk_rope_table: bad argument");
  const long long n = (long long)max_seq * (head_dim / 2);
  int grid = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  rope_table_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(cos_t, sin_t, max_seq, head_dim / 2, theta);
  CGK_LAUNCH_CHECK();
  return 0;
}

// dtype 0 = fp32, 1 = bf16.  backward != 0 applies the inverse rotation.
CGK_API int cgk_rope_apply(int dtype, void* x, const float* cos_t, const float* sin_t,
                           const int* positions, int B, int T, int H, int D, long long bs,
                           long long ts, long long hs, int pos_offset, int max_seq, int backward,
                           void* stream) {
  CGK_REQUIRE(x && cos_t && sin_t && D % 2 == 0, "cgk_rope_apply: bad argument");
  const long long n = (long long)B * T * H * (D / 2);
  if (n == 0) return 0;
  int dev = 0;
  cudaGetDevice(&dev);
  long long blocks = (n + 255) / 256, cap = (long long)sm_count(dev) * 16;
  if (blocks > cap) blocks = cap;
  const float sign = backward ? -1.0f : 1.0f;
  if (dtype != 0 && D % 16 == 0 && ((bs | ts | hs) & 7) == 0 && n / 8 <= 0x7fffff00LL &&
      (((uintptr_t)x | (uintptr_t)cos_t | (uintptr_t)sin_t) & 15) == 0) {
    CGK_CUDA_CHECK(launch_overlapped(rope_apply_vec_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, 0,
                                     (__nv_bfloat16*)x, cos_t, sin_t, positions, (int)(n / 8), T, H, D / 2, bs, ts, hs, pos_offset, max_seq, sign));
    return 0;
  }
  if (dtype == 0)
    rope_apply_kernel<float><<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(
        (float*)x, cos_t, sin_t, positions, B, T, H, D, bs, ts, hs, pos_offset, max_seq, sign);
  else
    rope_apply_kernel<__nv_bfloat16><<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(
        (__nv_bfloat16*)x, cos_t, sin_t, positions, B, T, H, D, bs, ts, hs, pos_offset, max_seq, sign);
  CGK_LAUNCH_CHECK();
  return 0;
}
