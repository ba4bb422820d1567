// INT4 weight-only GEMM for few rows (decoding): the weight stream goes through registers into warp-level MMAs.
// out[M,N] = X[M,K] (bf16) . dequant(W)[K,N] (+ bias), W in the reference's format
// (src/quantize/int4.c:10-59: row-major [K,N], flat groups along N, fp32 scale per group).
//
// With few rows in X the product is bound by the weight stream, and what stands between the stream and its bandwidth is the
// way from nibbles to the tensor core.  A tcgen05 operand has to be written to shared or tensor memory, fenced, handed over by
// an mbarrier and multiplied by one issuing thread: about 2200 cycles per 128 x 128 weights and SM for 16 rows, of which the
// conversion is 150.  mma.sync takes the converted words from the registers they were converted in, at a third of
// the rate, of which 16 rows would need three quarters if the bytes came at copy rate:
//   * the weights are the A operand: m16 = 16 output features, n8 = 8 rows of X.  A warp owns all 128 features of a tile for 32 k
//     at a time, so that X costs little beside the weights, and the warps of a CTA take the 32-k steps in turn: no warp waits for
//     another inside a tile;
//   * a lane fetches with cp.async exactly the 16-byte words that it converts itself (and its own pieces of X), into a ring of
//     its warp: nothing but the lane's own copies to wait for, no registers spent on what is under way;
//   * the scale of a weight depends on (k, n / group).  With group % 128 == 0 a tile's 128 features share one scale per k, which is
//     moved into X: x'[t,k] = bf16(x[t,k] * s[k]), worked out in registers by every warp for its k;
//   * nibbles become bf16 by bit tricks only: the stream holds u = q + 8, and bf16 bits 0x4300 | u are 128 + u exactly.  The
//     MMAs therefore sum x' . (q + 136); one more MMA with ones for weights sums x' over k in the same order, and 136 times that
//     is subtracted in fp32.
// The tile stream is prepared once per weight (cgk_int4_wa_tile_weights): per (128 features, 32 k) a step of 2176 bytes: four 16-byte
// words per lane, [word][lane], then the step's 32 scales.  In an MMA the order of k does not matter as long as both operands
// have the same: lane l (g = l / 4, q = l % 4) holds k = 8 q .. 8 q + 7 of features g and g + 8 of each 16, which are two MMAs of
// 16 k, and whose eight values of X are 16 consecutive bytes.  32-bit word (m, s) of a lane: features 16 m + g (+ 8), MMA s; its
// nibble r and r + 4 are register r of the A fragment.
//
// Work is dealt out by steps, not by tiles: the steps of all feature tiles are one line (which is also how the stream lies in
// memory) and every resident CTA takes an equal piece of it, so that no SM has two tiles while its neighbour has one, and a
// K of 11 008 fills the machine like any other.  A piece covers the end of one tile and the start of the next.  At a tile's end the
// warps' sums meet in shared memory, summed in the order of the warps; a tile covered by one CTA is written at once, the parts of the
// others go to fp32 slots of their own, and the CTA that arrives last at the tile's counter sums them in the order of the CTAs,
// adds the bias, writes bf16 and leaves the counter zeroed.  Both orders are fixed, so a call gives the same bits every time.  Few
// tiles are shared by clusters instead (see launch_wa).
//
// What bounds it (counters of one launch, 16 rows, 4096 x 32000): the two warps of a scheduler do their MMAs and their integer work nearly
// in turn.  Of 43 500 cycles the tensor pipe is busy for 36 % and the integer pipe (a shift and a logic operation per pair of weights) for
// 39 %; that is 286 and 308 cycles for each of a scheduler's 54 steps of 128 x 32 weights, which at copy rate would arrive every 390.
// Of the warps' time, barriers (a tile's end) take 13 %, data that has not arrived 9 %.  16 rows, layers one after the other, us:
// 4096 x 32000 42.9 through tcgen05, 25.6 like this (10.9 for the bytes); 4096 x 22016 34.0, 20.6; 1 row, 4096 x 32000 40.8, 19.8.
#include <cuda_bf16.h>

#include <atomic>

#include "host_common.h"
#include "int4_tile.cuh"
#include "mma_sync.cuh"
#include "cogito_kernels.h"

namespace {
using namespace cgk;

constexpr int WF = 128, WK = 32;                               // features per tile, k per step
constexpr int W_NIB = WF * WK / 2, W_STEP = W_NIB + WK * 4;    // 2048 + 128 bytes
constexpr int W_UNIT = 2 * W_STEP, W_LD = WF + 4;              // what a warp takes at a time; row of the output tile in shared memory: lanes of a store in different banks
constexpr int W_WARPS = 8, W_THREADS = W_WARPS * 32;
constexpr int W_MAXROWS = 32;                                  // rows of X per CTA: four n8 columns of MMAs

template <int NT>                                              // n8 columns of MMAs
struct WaCfg {
  static constexpr int STAGE = W_UNIT + NT * 1024;             // a warp's unit: weights, scales, its pieces of X
  static constexpr int STAGES = NT <= 2 ? 3 : 2;
  static constexpr int RING = W_WARPS * STAGES * STAGE;
  static constexpr int ROUNDS = NT <= 2 ? 2 : 4, M_ROUND = 8 / ROUNDS;    // sums of M_ROUND * 16 features meet at a time
  static constexpr int RED = W_WARPS * M_ROUND * NT * 512;
  static constexpr int OUT = 8 * NT * W_LD * 4;
  static constexpr int SMEM = RING + RED + OUT + 16;
};

struct WaDev {
  const uint8_t* tiles;            // [N/128][K/32][2176]
  const __nv_bfloat16* x; long long ldx;
  float4* parts;                   // slots of shared tiles' parts: [m_tiles][ctas][2][256 * NT]
  int* counters;                   // [m_tiles * n_tiles], zero between calls (shared tiles only)
  void* out; long long ldo;        // bf16, or fp32 with out_f32
  const __nv_bfloat16* bias;
  int M, N, K;
  int out_f32;
  int cluster;                     // CTAs that share every tile as a cluster; 0: pieces of the line
};

// The CTAs lo .. hi of a row tile that share feature tile nt.  A CTA's piece may end one shared tile and begin another: its
// slot 0 is for the part that its piece begins with, slot 1 for the other.
struct WaShare { uint32_t lo, hi, first; };
__device__ __forceinline__ WaShare wa_share(uint32_t k_units, const Pieces& pieces, uint32_t nt) {
  WaShare w;
  w.lo = pieces.of(nt * k_units);
  w.hi = pieces.of((nt + 1) * k_units - 1);
  w.first = pieces.begin(w.lo) < nt * k_units;               // slot of CTA lo; the others begin with this tile
  return w;
}

template <int NT>
__global__ void __launch_bounds__(W_THREADS, 1)
int4_wa_kernel(const WaDev g) {
  using C = WaCfg<NT>;
  constexpr int P = 256 * NT;                                              // float4s of a tile
  extern __shared__ __align__(16) uint8_t smem[];
  float4* const red = reinterpret_cast<float4*>(smem + C::RING);          // [warp][m of the round][n][lane]
  float* const out_s = reinterpret_cast<float*>(smem + C::RING + C::RED); // [row][W_LD]
  volatile int* const is_last = reinterpret_cast<volatile int*>(smem + C::RING + C::RED + C::OUT);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
  const uint8_t* const stages = smem + warp * (C::STAGES * C::STAGE);
  const uint32_t ring = smem_u32(stages) + lane * 16, k_units = g.K / (2 * WK);
  const int m0 = blockIdx.y * W_MAXROWS;
  const Pieces pieces((uint32_t)(g.N / WF) * k_units, gridDim.x);
  auto piece = [&](uint32_t c) -> uint32_t { return g.cluster ? c / g.cluster * k_units + c % g.cluster * k_units / g.cluster : pieces.begin(c); };
  const uint32_t u0 = piece(blockIdx.x), u1 = piece(blockIdx.x + 1);              // this CTA's units; warp w has u0 + w, + 8, ..

  // The weights depend on no earlier kernel: this CTA's share of the stream (its first 128 KB) starts on its way to L2 before
  // the predecessor, which is still running, has finished.  A prefetch has no result, so nothing can be read too early.
  if (warp == 0) {
    const unsigned long long hi = (unsigned long long)u1 * W_UNIT, from = (unsigned long long)u0 * W_UNIT + lane * 4096ull;
    if (from < hi && blockIdx.y == 0) prefetch_l2(g.tiles + from, (uint32_t)min(hi - from, 4096ull));
  }
  pdl_trigger();
  pdl_wait();

  uint32_t fu = u0 + warp, fs = ring;                                       // unit and ring slot of the next fetch
  const uint32_t ring_end = ring + C::STAGES * C::STAGE;
  const uint8_t* wsrc = g.tiles + (unsigned long long)fu * W_UNIT + lane * 16;
  uint32_t kx = fu % k_units * (2 * WK);                                    // its first k
  const uint32_t kx_step = W_WARPS % k_units * (2 * WK);
  const __nv_bfloat16* xrow[NT];                                           // this lane's rows of X, 8 q elements in
  uint32_t xbytes[NT];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int t = m0 + n * 8 + gq;
    xbytes[n] = t < g.M ? 16 : 0;
    xrow[n] = g.x + (long long)(t < g.M ? t : m0) * g.ldx + q * 8;
  }
  auto fetch = [&]() {
    if (fu < u1) {
#pragma unroll
      for (int h = 0; h < 8; ++h) cp_async_16(fs + (h & 3) * 512 + (h >> 2) * W_STEP, wsrc + (h & 3) * 512 + (h >> 2) * W_STEP);
      if (lane < 8) {
        cp_async_16(fs + W_NIB, wsrc + W_NIB);
        cp_async_16(fs + W_STEP + W_NIB, wsrc + W_STEP + W_NIB);
      }
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        cp_async_16_or_zero(fs + W_UNIT + n * 1024, xrow[n] + kx, xbytes[n]);
        cp_async_16_or_zero(fs + W_UNIT + n * 1024 + 512, xrow[n] + kx + WK, xbytes[n]);
      }
      wsrc += W_WARPS * W_UNIT;
      fu += W_WARPS;
      kx += kx_step;
      if (kx >= (uint32_t)g.K) kx -= g.K;
      fs += C::STAGE;
      if (fs == ring_end) fs = ring;
    }
    cp_async_commit();                    // an empty group past the end: the count below stays right
  };
#pragma unroll
  for (int i = 0; i < C::STAGES - 1; ++i) fetch();

  uint32_t u = u0 + warp, slot = 0, mask = 0x000F000Fu, magic = 0x43004300u;
  asm volatile("" : "+r"(mask), "+r"(magic));
  for (uint32_t from = u0; from < u1;) {                                    // the tiles that the piece covers
    const uint32_t nt = from / k_units, to = min(u1, (nt + 1) * k_units);
    float acc[8][NT][4], sum[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sum[n][e] = 0.0f;
#pragma unroll
        for (int m = 0; m < 8; ++m) acc[m][n][e] = 0.0f;
      }
    }
    for (; u < to; u += W_WARPS) {
      cp_async_wait<C::STAGES - 2>();
      __syncwarp();                                                         // the scales came through the first lanes; the slot fetched next was read by all
      const uint8_t* src = stages + slot * C::STAGE;
      slot = slot + 1 == C::STAGES ? 0 : slot + 1;
      fetch();
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint8_t* step = src + half * W_STEP;
        const float4 s0 = *reinterpret_cast<const float4*>(step + W_NIB + q * 32), s1 = *reinterpret_cast<const float4*>(step + W_NIB + q * 32 + 16);
        uint32_t b[NT][4];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 v = *reinterpret_cast<const uint4*>(src + W_UNIT + n * 1024 + half * 512 + lane * 16);
          const float2 x0 = unpack_bf16x2(v.x), x1 = unpack_bf16x2(v.y), x2 = unpack_bf16x2(v.z), x3 = unpack_bf16x2(v.w);
          b[n][0] = pack_bf16x2(x0.x * s0.x, x0.y * s0.y);
          b[n][1] = pack_bf16x2(x1.x * s0.z, x1.y * s0.w);
          b[n][2] = pack_bf16x2(x2.x * s1.x, x2.y * s1.y);
          b[n][3] = pack_bf16x2(x3.x * s1.z, x3.y * s1.w);
        }
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int n = 0; n < NT; ++n) mma_bf16(sum[n], 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u, b[n][2 * s], b[n][2 * s + 1]);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const uint4 w4 = *reinterpret_cast<const uint4*>(step + h * 512 + lane * 16);
          const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int ms = (i & 1) * 2 + (i >> 1);                          // the two features' first MMAs, then their second ones
            const uint32_t v = w[ms];
            const uint32_t a0 = pick(v, mask, magic), a1 = pick(v >> 4, mask, magic), a2 = pick(v >> 8, mask, magic), a3 = pick(v >> 12, mask, magic);
#pragma unroll
            for (int n = 0; n < NT; ++n) mma_bf16(acc[2 * h + (ms >> 1)][n], a0, a1, a2, a3, b[n][2 * (ms & 1)], b[n][2 * (ms & 1) + 1]);
          }
        }
      }
    }
    // The tile's end: a fragment's four sums are features (16 m + g, + 8) x rows (8 n + 2 q, + 1).
    const WaShare w = g.cluster ? WaShare{0, 0, 0} : wa_share(k_units, pieces, nt);
    float4* const part = g.cluster ? reinterpret_cast<float4*>(out_s) : w.lo == w.hi ? nullptr : g.parts + (unsigned long long)((blockIdx.y * gridDim.x + blockIdx.x) * 2 + (from > u0)) * P;
    float* const tile = g.cluster ? reinterpret_cast<float*>(red) : out_s;  // the output tile; a cluster's parts are in out_s
    auto to_out = [&](int e, float4 v) {                                    // e: (m * NT + n) * 32 + lane
      const int l = e & 31, mn = e >> 5, m = mn / NT, t = (mn - m * NT) * 8 + (l & 3) * 2, f = m * 16 + (l >> 2);
      tile[t * W_LD + f] = v.x;
      tile[(t + 1) * W_LD + f] = v.y;
      tile[t * W_LD + f + 8] = v.z;
      tile[(t + 1) * W_LD + f + 8] = v.w;
    };
#pragma unroll
    for (int r = 0; r < C::ROUNDS; ++r) {
#pragma unroll
      for (int m = 0; m < C::M_ROUND; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const float (&a)[4] = acc[r * C::M_ROUND + m][n];
          red[((warp * C::M_ROUND + m) * NT + n) * 32 + lane] =
              make_float4(a[0] - 136.0f * sum[n][0], a[1] - 136.0f * sum[n][1], a[2] - 136.0f * sum[n][2], a[3] - 136.0f * sum[n][3]);
        }
      __syncthreads();
#pragma unroll
      for (int e = tid; e < C::M_ROUND * NT * 32; e += W_THREADS) {
        float4 v = red[e];
#pragma unroll
        for (int k = 1; k < W_WARPS; ++k) {
          const float4 o = red[k * (C::M_ROUND * NT * 32) + e];
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        const int whole = r * (C::M_ROUND * NT * 32) + e;
        if (part) part[whole] = v;
        else to_out(whole, v);
      }
      __syncthreads();
    }
    bool write = !part;
    int c0 = 0, cols = WF;                                                  // columns of the tile that this CTA writes
    if (g.cluster) {
      // every CTA of the cluster sums and writes its share of the features, over the ranks in order
      const int S = g.cluster, rank = (int)cluster_rank();
      c0 = 8 * rank / S * 16;
      cols = 8 * (rank + 1) / S * 16 - c0;
      cluster_sync_all();
      for (int e = c0 / 16 * (NT * 32) + tid; e < (c0 + cols) / 16 * (NT * 32); e += W_THREADS) {
        const uint32_t at = smem_u32(part + e);
        float4 v = ld_cluster_f4(cluster_map(at, 0));
        for (int k = 1; k < S; ++k) {
          const float4 o = ld_cluster_f4(cluster_map(at, k));
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        to_out(e, v);
      }
      cluster_sync_all();                                                   // the share is whole, and nobody leaves while its part is read
      write = true;
    } else if (part) {
      if (tid == 0) *is_last = arrive_acq_rel(g.counters + blockIdx.y * (g.N / WF) + nt) == (int)(w.hi - w.lo);
      __syncthreads();
      write = *is_last;
      if (write) {
        const float4* first = g.parts + (unsigned long long)((blockIdx.y * gridDim.x + w.lo) * 2 + w.first) * P;
        const float4* next = g.parts + (unsigned long long)((blockIdx.y * gridDim.x + w.lo + 1) * 2) * P;
#pragma unroll
        for (int e = tid; e < P; e += W_THREADS) {
          float4 v = __ldcg(first + e);
#pragma unroll 4
          for (uint32_t c = 0; c < w.hi - w.lo; ++c) {
            const float4 o = __ldcg(next + (unsigned long long)c * (2 * P) + e);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
          to_out(e, v);
        }
        if (tid == 0) g.counters[blockIdx.y * (g.N / WF) + nt] = 0;
      }
      __syncthreads();                                                      // the output tile is whole; is_last has been read
    }
    if (write) {
      for (int i = tid; i < NT * 8 * (cols / 4); i += W_THREADS) {
        const int t = i / (cols / 4), c = c0 + (i - t * (cols / 4)) * 4, n = (int)nt * WF + c;
        if (m0 + t >= g.M) continue;
        float4 v = *reinterpret_cast<const float4*>(tile + t * W_LD + c);
        if (g.bias) {
          v.x += __bfloat162float(g.bias[n]); v.y += __bfloat162float(g.bias[n + 1]);
          v.z += __bfloat162float(g.bias[n + 2]); v.w += __bfloat162float(g.bias[n + 3]);
        }
        const long long o = (long long)(m0 + t) * g.ldo + n;
        if (g.out_f32) *reinterpret_cast<float4*>((float*)g.out + o) = v;
        else *reinterpret_cast<uint2*>((__nv_bfloat16*)g.out + o) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      }
      // the next tile's sums come to out_s behind at least one more barrier
    }
    from = to;
  }
}

// packed [K][N/2] bytes + scales (flat groups along N) -> tiles [N/128][K/32][2176].  A thread has eight k of 32 columns: 16-byte word h of
// the eight lanes 4 g + q.  4096 x 32000: 34 us (130 with single nibbles out of eight rows for every word).
__global__ void __launch_bounds__(256)
int4_wa_tile_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ scales, int K, int N, int group, uint8_t* __restrict__ tiles, bool words) {
  const int k_tiles = K / WK, groups = N / group;
  const long long blk = ((long long)blockIdx.x * 256 + threadIdx.x) >> 4;
  if (blk >= (long long)(N / WF) * k_tiles) return;
  const int nt = (int)(blk / k_tiles), kt = (int)(blk % k_tiles), t = threadIdx.x & 15, h = t & 3, q = t >> 2;
  uint8_t* const dst = tiles + blk * W_STEP;
  const uint8_t* const src = packed + ((long long)(kt * WK + q * 8) * N + nt * WF) / 2 + h * 16;
  uint32_t w[4][8];                                                       // [word of the lane: features' MMA, k's MMA][nibble]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 8; ++e) {                                         // nibble e: register e % 4 of the fragment, its low or high half
      const int r = e & 3, k = (i & 1) * 4 + (r >> 1) * 2 + (e >> 2);
      w[i][e] = load_nibbles(src + (long long)k * (N / 2) + (i >> 1) * 8 + (r & 1) * 4, words) ^ 0x88888888u;
    }
  const float s0 = scales[(long long)(kt * WK + t * 2) * groups + nt * WF / group], s1 = scales[(long long)(kt * WK + t * 2 + 1) * groups + nt * WF / group];
#pragma unroll
  for (int i = 0; i < 4; ++i) transpose_nibbles(w[i]);
#pragma unroll
  for (int g = 0; g < 8; ++g) *reinterpret_cast<uint4*>(dst + h * 512 + (g * 4 + q) * 16) = make_uint4(w[0][g], w[1][g], w[2][g], w[3][g]);
  *reinterpret_cast<float2*>(dst + W_NIB + t * 8) = make_float2(s0, s1);
}

// The clusters of S CTAs that a device runs at once (asked for once; concurrent callers would store the same value).
template <int NT>
int clusters_at_once(int dev, int S, int* fit) {
  static std::atomic<int> known[64][9];
  if (dev < 64 && known[dev][S].load(std::memory_order_relaxed)) {
    *fit = known[dev][S].load(std::memory_order_relaxed) - 1;
    return 0;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)S);
  cfg.blockDim = dim3(W_THREADS);
  cfg.dynamicSmemBytes = WaCfg<NT>::SMEM;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  CGK_CUDA_CHECK(cudaOccupancyMaxActiveClusters(fit, int4_wa_kernel<NT>, &cfg));
  if (dev < 64) known[dev][S].store(*fit + 1, std::memory_order_relaxed);
  return 0;
}

// Few tiles (at most one for every second SM) are shared by clusters: as many CTAs per tile as run at once, each with a unit per warp at least.
// The parts meet over distributed shared memory, without the fence, the counter and the round trips of parts in global memory:
// 16 rows, layers one after the other, us by clusters / by pieces / by whole tiles: 4096 x 4096 (four CTAs) 6.5 / 9.9 / 11.9, 11008 x 4096
// (four) 10.9 / 13.5 / 26.1, 4096 x 6144 (two) 8.5 / 11.1 / 11.8.  More tiles would leave SMs idle, whole ones too: 4096 x 22016 (172 tiles)
// by pieces 20.6, whole 23.4.
template <int NT>
int launch_wa(WaDev g, dim3 grid, int dev, bool choose, cudaStream_t st) {
  CGK_CUDA_CHECK(cudaFuncSetAttribute(int4_wa_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, WaCfg<NT>::SMEM));
  const int tiles = g.N / WF * (int)grid.y, sms = sm_count(dev), units = g.K / (2 * WK);
  for (int S = sms / tiles < 8 ? sms / tiles : 8; choose && S > 1; --S) {
    int fit = 0;
    if (S * W_WARPS > units) continue;
    const int rc = clusters_at_once<NT>(dev, S, &fit);
    if (rc) return rc;
    if (fit < tiles) continue;
    g.cluster = S;
    grid.x = (unsigned)(g.N / WF * S);
    break;
  }
  CGK_CUDA_CHECK(launch_overlapped(int4_wa_kernel<NT>, grid, dim3(W_THREADS), WaCfg<NT>::SMEM, st, g.cluster, g));
  return 0;
}
}  // namespace

CGK_API long long cgk_int4_wa_tiles_bytes(int K, int N) { return (long long)(N / WF) * (K / WK) * W_STEP; }
// Reorders reference-format weights (packed [K, N/2] bytes, fp32 scales per flat group) into the
// stream cgk_int4_wa_gemm reads.  group: a multiple of 128 that divides N.
CGK_API int cgk_int4_wa_tile_weights(const void* packed, const float* scales, int K, int N, int group, void* tiles, void* stream) {
  CGK_REQUIRE(packed && scales && tiles, "cgk_int4_wa_tile_weights: null pointer");
  CGK_REQUIRE(N % WF == 0 && K % 64 == 0, "cgk_int4_wa_tile_weights: need N %% 128 == 0 and K %% 64 == 0 (got K=%d N=%d)", K, N);
  CGK_REQUIRE(group >= 128 && group % 128 == 0 && N % group == 0, "cgk_int4_wa_tile_weights: group %d must be a multiple of 128 that divides N", group);
  CGK_REQUIRE(((uintptr_t)tiles & 15) == 0, "cgk_int4_wa_tile_weights: misaligned buffer");
  const long long blocks = (long long)(N / WF) * (K / WK);
  int4_wa_tile_kernel<<<(unsigned)((blocks * 16 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint8_t*)packed, scales, K, N, group, (uint8_t*)tiles,
                                                                                            ((uintptr_t)packed & 3) == 0);
  CGK_LAUNCH_CHECK();
  return 0;
}

static int wa_columns(int M) { return M <= 8 ? 1 : M <= 16 ? 2 : 4; }
// CTAs per row tile: one per SM, with at least eight steps each (one per warp), and of those the fewest with the same longest piece
// (fewer parts to store and to sum); given splits: that many equal parts of every tile; without a place for parts: whole tiles.
static long long wa_ctas(int sms, int M, int N, int K, int splits, bool parts) {
  const long long n_tiles = N / WF, m_tiles = (M + W_MAXROWS - 1) / W_MAXROWS, total = n_tiles * (K / (2 * WK));
  if (splits > 0 || !parts) return n_tiles * (splits > 0 ? splits : 1);
  long long ctas = sms / m_tiles;
  if (ctas > total / W_WARPS) ctas = total / W_WARPS;
  if (ctas < 1) ctas = 1;
  const long long longest = (total + ctas - 1) / ctas;
  return (total + longest - 1) / longest;
}

CGK_API long long cgk_int4_wa_gemm_parts_floats(int M, int N, int K, int splits) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || M <= 0 || N < WF || K < 128) return 0;
  return (long long)((M + W_MAXROWS - 1) / W_MAXROWS) * wa_ctas(cgk::sm_count(dev), M, N, K, splits, true) * 2 * WF * 8 * wa_columns(M);
}

static int wa_gemm(const void* x, long long ldx, const void* tiles, float* parts, int* counters, void* out, long long ldo,
                   const void* bias, int M, int N, int K, int splits, int out_f32, void* stream) {
  using namespace cgk;
  CGK_REQUIRE(x && tiles && out, "cgk_int4_wa_gemm: null pointer");
  CGK_REQUIRE(M > 0 && N > 0 && K > 0 && N % WF == 0 && K % 128 == 0, "cgk_int4_wa_gemm: need N %% 128 == 0 and K %% 128 == 0 (got M=%d N=%d K=%d)", M, N, K);
  CGK_REQUIRE(ldx % 8 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)tiles & 15) == 0 && ((uintptr_t)parts & 15) == 0 && ldo % 4 == 0 && ((uintptr_t)out & (out_f32 ? 15 : 7)) == 0,
              "cgk_int4_wa_gemm: misaligned operand");
  int dev = 0;
  CGK_CUDA_CHECK(cudaGetDevice(&dev));
  CGK_REQUIRE(splits <= 0 || (K / 128) % splits == 0, "cgk_int4_wa_gemm: K/128 = %d is not divisible by splits = %d", K / 128, splits);
  CGK_REQUIRE(splits <= 1 || (parts && counters), "cgk_int4_wa_gemm: split-K needs scratch and counters");
  const WaDev g{(const uint8_t*)tiles, (const __nv_bfloat16*)x, ldx, (float4*)parts, counters, out, ldo, (const __nv_bfloat16*)bias, M, N, K, out_f32, 0};
  const dim3 grid((unsigned)wa_ctas(sm_count(dev), M, N, K, splits, parts && counters), (unsigned)((M + W_MAXROWS - 1) / W_MAXROWS));
  cudaStream_t st = (cudaStream_t)stream;
  switch (wa_columns(M)) {
    case 1: return launch_wa<1>(g, grid, dev, splits <= 0, st);
    case 2: return launch_wa<2>(g, grid, dev, splits <= 0, st);
    default: return launch_wa<4>(g, grid, dev, splits <= 0, st);
  }
}

// x bf16 [M, ldx]; tiles from cgk_int4_wa_tile_weights; out bf16 [M, ldo]; bias bf16 [N] or null.  parts (fp32
// [cgk_int4_wa_gemm_parts_floats], any contents) and counters (int32 [cgk_int4_gemm_counters(M, N)], zero before the first call and
// left zero by every call) serve tiles shared by several CTAs; without them every tile is computed whole.  splits 0 = chosen here.
CGK_API int cgk_int4_wa_gemm_parts(const void* x, long long ldx, const void* tiles, float* parts, int* counters, void* out, long long ldo,
                                   const void* bias, int M, int N, int K, int splits, void* stream) {
  return wa_gemm(x, ldx, tiles, parts, counters, out, ldo, bias, M, N, K, splits, 0, stream);
}
// The same with an fp32 output (logits), whose rows start on 16-byte boundaries.
CGK_API int cgk_int4_wa_gemm_parts_f32(const void* x, long long ldx, const void* tiles, float* parts, int* counters, float* out, long long ldo,
                                       const void* bias, int M, int N, int K, int splits, void* stream) {
  return wa_gemm(x, ldx, tiles, parts, counters, out, ldo, bias, M, N, K, splits, 1, stream);
}

// The same for callers that hold an accumulator (see cgk_int4_gemm).
CGK_API int cgk_int4_wa_gemm(const void* x, long long ldx, const void* tiles, float* acc, int* counters, void* out, long long ldo,
                             const void* bias, int M, int N, int K, int splits, void* stream) {
  const bool shared = acc && counters;
  return cgk::with_stream_scratch(shared ? cgk_int4_wa_gemm_parts_floats(M, N, K, splits) : 0, (cudaStream_t)stream, [&](float* parts) {
    return wa_gemm(x, ldx, tiles, parts, parts ? counters : nullptr, out, ldo, bias, M, N, K, shared && !parts ? 0 : splits, 0, stream);
  });
}
