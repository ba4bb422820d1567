// INT4 weight-only GEMM for serving: out[M,N] = X[M,K] (bf16) . dequant(W)[K,N] (+ bias).
//
// W holds the reference's quantised values (src/quantize/int4.c:10-59, 90-114: row-major [K,N],
// 4-bit two's complement, even column in the low nibble, one fp32 scale per flat group of
// `group` elements), reordered tile-major without re-quantising (cgk_int4_tile_weights): per 128 columns ("features") and 64 k one
// block of 4352 bytes: for each half of the k 16 bytes of nibbles (q + 8) a feature, nibbles j and j + 4 of a word for k 2 j and
// 2 j + 1; then, for each half of the features, the 64 k's scales rounded to bf16, which is what the product takes them as.  A CTA's
// share is then one sequential stream, which is what keeps HBM efficient (64-byte pieces of the row-major layout are not).
//
// The weights are the A operand (128 features) and come from tensor memory, the rows of X are the B operand.  The shape is bound by
// the weights' bytes and by what turns them into an operand.  With the weights written to and read from shared memory that was the
// limit (1080 of 1110 cycles a step of 128 k, of which 512 for weights and 256 for 128 rows of X however many there are); a thread
// that has one feature stores its k straight into its lane of tensor memory, its scales are read by all lanes of a warp at once.
//   warp 0    bulk copies of W blocks into a ring as deep as shared memory allows (bytes in flight cover HBM latency)
//   warp 3    TMA: X tiles [rows, 64 k] into their own ring of up to 6 stages; round_up(M, 16) rows.  One lane issues: eight lanes,
//             each with its own ring slots, held one another up in their waits (80 rows of 4096 x 32000: 47 -> 37 us)
//   warps 4-19 two groups: nibbles -> bf16: exact integer (magic-number trick), one multiply by the scale, to tensor memory
//   warp 1    tcgen05.mma, two accumulators in TMEM (128 lanes x up to 128 columns)
//   warps 20-23 epilogue, a lane a feature.  Whole tile: TMEM -> bias -> bf16 (or fp32) -> global.  Part of a tile: into the part's
//             own fp32 slot; the CTA that arrives last at the tile's counter sums the slots in the
//             order of the CTAs, adds the bias, writes the output and leaves the counter zeroed for the
//             next call.  The order is fixed, so a call gives the same bits every time.
// 80 rows, layers one after the other, operand through shared / through tensor memory (the deal below included): 4096 x 6144
// 17.7 / 11.4 us, 4096 x 4096 14.5 / 10.2, 4096 x 22016 32.1 / 24.8, 11008 x 4096 20.8 / 17.2, 4096 x 32000 44.8 / 34.3,
// 2048 x 11264 15.0 / 11.3.  A step takes some 850 cycles: eight MMAs of 16 k with A in tensor memory (70 to 90 each, whatever the
// rows), issue slots that the converting warps share with the MMA warp, and from 128 rows on the 32 KB of X.
// One CTA per SM.  Each takes as many whole tiles as there are for all of them; the tiles that are left over are shared (deal, below).
// The sum of the CTA's last shared tile is work of all its threads; four of a thread's quads are on their way at a time (one: 22016
// columns took 45 us instead of 32).
#include <cuda_bf16.h>
#include <stdlib.h>

#include "host_common.h"
#include "int4_tile.cuh"
#include "mma_sync.cuh"
#include "cogito_kernels.h"

namespace {
using namespace cgk;

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int SUB = 2;                                        // 64-row sub-tiles per pipeline step (a step covers 128 k)
constexpr int B_STAGES = 4, MAX_RAW_STAGES = 16, MAX_A_STAGES = 8;
constexpr int ACC_COLS = 2 * BM, W_COLS = SUB * BK / 2, TMEM_COLS = 512;              // two accumulators, then B_STAGES operands of W_COLS columns
constexpr int GROUPS = 2, GROUP_WARPS = 8, CONVERT_WARPS = GROUPS * GROUP_WARPS;     // converting warps: groups that take the steps in turn
// A group waits for a ring slot by the parity of its phase, which also holds while the slot's last step but one has not arrived (with an
// odd depth that step is the other group's).  Before it comes to step i it has ended step i - GROUPS, for which step i - GROUPS - B_STAGES
// was multiplied and so all steps before it were converted: a ring of this many steps or more is safe.
constexpr int MIN_RAW_STAGES = GROUPS + B_STAGES;
constexpr int NIB_BYTES = BK * BN / 2, SCALE_BYTES = BK * 2 * 2, RAW_BYTES = NIB_BYTES + SCALE_BYTES;   // 4096 + 256
constexpr int EPI_WARP0 = 4 + CONVERT_WARPS, THREADS = 32 * (EPI_WARP0 + 4);
constexpr int SMEM_BYTES = 226 * 1024;                       // alignment slack | X ring | W ring | barriers
constexpr int RING_BUDGET = SMEM_BYTES - 1024 - 2048;        // shared by the X and W rings
static_assert((RING_BUDGET - 3 * SUB * BM * 128) / (SUB * RAW_BYTES) >= MIN_RAW_STAGES, "the W ring beside the least X ring");

struct Int4Dev {
  const uint8_t* w_tiles;          // [N/128][K/64][4352]
  float4* parts;                   // slots of shared tiles' parts: [m_tiles][sharers][2][a_rows][32 column quads]
  int* counters;                   // int32 [m_tiles * n_tiles], zero between calls (shared tiles only)
  void* out; long long ldo;        // bf16, or fp32 with out_f32
  const __nv_bfloat16* bias;
  int M, N, K, out_f32;
  int a_rows, a_stages;            // rows fetched per X tile (multiple of 16: columns of the MMA), depth of the X ring
  int raw_stages;                  // depth of the W ring
  int sharers, per_tile;           // CTAs that the left-over tiles are dealt to; with per_tile: that many to each of them
  int piece, longer;               // steps of a sharer's piece; how many have one more
  int* status;
};

// The steps of the left-over tiles, dealt to the sharers in order, in pieces that differ by one step at most: of the whole line, or
// (per_tile > 0) of each tile.
struct Shares {
  uint32_t per_tile, k_tiles, q, r;                          // a line is q steps for each piece and one more for the first r
  __device__ __forceinline__ explicit Shares(const Int4Dev& g, uint32_t k_tiles) : per_tile(g.per_tile), k_tiles(k_tiles), q(g.piece), r(g.longer) {}
  __device__ __forceinline__ uint32_t begin(uint32_t c) const {
    const uint32_t t = per_tile ? c / per_tile : 0, j = c - t * per_tile;
    return t * k_tiles + j * q + min(j, r);
  }
  // the sharers that left-over tile t begins and ends with
  __device__ __forceinline__ int first(uint32_t t) const { return per_tile ? t * per_tile : of(t * k_tiles); }
  __device__ __forceinline__ int last(uint32_t t) const { return per_tile ? t * per_tile + per_tile - 1 : of((t + 1) * k_tiles - 1); }
  __device__ __forceinline__ uint32_t of(uint32_t step) const { return step < r * (q + 1) ? step / (q + 1) : r + (step - r * (q + 1)) / q; }
};

// Slot `which` of a sharer: [a_rows][32 column quads] float4s.
__device__ __forceinline__ float4* part_slot(const Int4Dev& g, int mt, int sharer, int which) {
  return g.parts + (long long)((mt * g.sharers + sharer) * 2 + which) * ((BN / 4) * g.a_rows);
}

// Four neighbouring elements of the output.
__device__ __forceinline__ void store4(const Int4Dev& g, long long at, const float4& v) {
  if (g.out_f32) *reinterpret_cast<float4*>((float*)g.out + at) = v;
  else *reinterpret_cast<uint2*>((__nv_bfloat16*)g.out + at) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}

// The output of a tile out of its parts, summed in the order of the CTAs lo .. hi; `first`: the slot that CTA lo's is in.
__device__ __forceinline__ void sum_parts(const Int4Dev& g, int mt, int nt, int lo, int hi, int first_slot, int tid, int threads) {
  const int m0 = mt * BM, n0 = nt * BN, rows = min(BM, g.M - m0), stride = 2 * (BN / 4) * g.a_rows;
  const float4* first = part_slot(g, mt, lo, first_slot);
  const float4* others = part_slot(g, mt, lo, 0);
  constexpr int U = 4;                                     // quads of a thread on their way at a time, times two parts
  const int quads = rows * (BN / 4), c1 = hi - lo;
  for (int e0 = tid; e0 < quads; e0 += U * threads) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = __ldcg(first + min(e0 + u * threads, quads - 1));
#pragma unroll 2
    for (int c = 1; c <= c1; ++c) {
      float4 x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = __ldcg(others + (long long)c * stride + min(e0 + u * threads, quads - 1));
#pragma unroll
      for (int u = 0; u < U; ++u) { v[u].x += x[u].x; v[u].y += x[u].y; v[u].z += x[u].z; v[u].w += x[u].w; }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * threads, t = e / (BN / 4), n = n0 + e % (BN / 4) * 4;
      if (e >= quads) break;
      if (g.bias) {
        v[u].x += __bfloat162float(g.bias[n]); v[u].y += __bfloat162float(g.bias[n + 1]);
        v[u].z += __bfloat162float(g.bias[n + 2]); v[u].w += __bfloat162float(g.bias[n + 3]);
      }
      store4(g, (long long)(m0 + t) * g.ldo + n, v[u]);
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1)
int4_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const Int4Dev g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sA = base;                                         // a_stages x SUB x (a_rows * 128 B)
  const uint32_t sRaw = sA + (uint32_t)g.a_stages * SUB * (uint32_t)g.a_rows * 128u;   // raw_stages x SUB x 4352 B
  const uint32_t sBar = base + SMEM_BYTES - 2048;
  const uint8_t* raw_s = gen + (sRaw - base);
  volatile int* dead = reinterpret_cast<volatile int*>(gen + (sBar - base) + 960);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + (sBar - base) + 968);
  volatile int* is_last = reinterpret_cast<volatile int*>(gen + (sBar - base) + 976);
  auto a_full = [&](int s) { return sBar + 8u * s; };
  auto a_empty = [&](int s) { return sBar + 8u * (MAX_A_STAGES + s); };
  auto b_full = [&](int s) { return sBar + 8u * (2 * MAX_A_STAGES + s); };
  auto b_empty = [&](int s) { return sBar + 8u * (2 * MAX_A_STAGES + B_STAGES + s); };
  auto raw_full = [&](int s) { return sBar + 8u * (2 * MAX_A_STAGES + 2 * B_STAGES + s); };
  auto raw_empty = [&](int s) { return sBar + 8u * (2 * MAX_A_STAGES + 2 * B_STAGES + MAX_RAW_STAGES + s); };
  auto acc_full = [&](int a) { return sBar + 8u * (2 * MAX_A_STAGES + 2 * B_STAGES + 2 * MAX_RAW_STAGES + a); };
  auto acc_empty = [&](int a) { return sBar + 8u * (2 * MAX_A_STAGES + 2 * B_STAGES + 2 * MAX_RAW_STAGES + 2 + a); };

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_tiles = g.N / BN, k_tiles = g.K / (SUB * BK), mt = blockIdx.y, m0 = mt * BM;
  // This CTA's steps of 128 k: its `own` steps of whole tiles, then its piece of the line of the tiles that are left over.
  const int ctas = gridDim.x, whole = n_tiles / ctas * ctas, own = n_tiles / ctas * k_tiles, sharers = g.sharers;
  const Shares pieces(g, (uint32_t)k_tiles);
  const int cta = blockIdx.x, r0 = (int)pieces.begin(min(cta, sharers));
  const int ksteps = own + (int)pieces.begin(min(cta + 1, sharers)) - r0, a_stages = g.a_stages, RAW_STAGES = g.raw_stages;
  auto line = [&](int i) -> int { return i < own ? cta * own + i : whole * k_tiles + r0 + (i - own); };
  auto part_steps = [&](int i) -> int { return min(ksteps - i, k_tiles - line(i) % k_tiles); };
  const uint32_t a_bytes = (uint32_t)g.a_rows * 128u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_A_STAGES; ++s) { mbar_init(a_full(s), 1); mbar_init(a_empty(s), 1); }
    for (int s = 0; s < B_STAGES; ++s) { mbar_init(b_full(s), GROUP_WARPS); mbar_init(b_empty(s), 1); }
    for (int s = 0; s < MAX_RAW_STAGES; ++s) { mbar_init(raw_full(s), 1); mbar_init(raw_empty(s), GROUP_WARPS); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), 4); }
    *dead = 0;
    *is_last = 0;
    mbar_fence_init();
  }
  if (warp == 2) { tmem_alloc(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish(); }
  // the first weights (no earlier kernel's business) start on their way to L2 while the predecessor still runs
  if (warp == 0 && blockIdx.y == 0 && lane < min(ksteps, 14)) prefetch_l2(g.w_tiles + (long long)line(lane) * (SUB * RAW_BYTES), SUB * RAW_BYTES);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  pdl_wait();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int r = 0;
      uint32_t par = 1;
      for (int i = 0; i < ksteps; ++i) {
        if (!mbar_wait(raw_empty(r), par, dead, g.status, 300)) break;
        mbar_expect_tx(raw_full(r), SUB * RAW_BYTES);
        bulk_load_1d(sRaw + r * (SUB * RAW_BYTES), g.w_tiles + (long long)line(i) * (SUB * RAW_BYTES), SUB * RAW_BYTES, raw_full(r));
        if (++r == RAW_STAGES) { r = 0; par ^= 1; }
      }
    }
  } else if (warp == 3) {
    if (lane == 0) {
      tma_prefetch_desc(&tmX);
      int s = 0;
      uint32_t par = 1;
      for (int i = 0; i < ksteps; ++i) {
        const int ks = line(i) % k_tiles;                             // step within its tile
        if (!mbar_wait(a_empty(s), par, dead, g.status, 301)) break;
        mbar_expect_tx(a_full(s), SUB * a_bytes);
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
          tma_load_2d(sA + (s * SUB + sub) * a_bytes, &tmX, a_full(s), (ks * SUB + sub) * BK, m0);
        if (++s == a_stages) { s = 0; par ^= 1; }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BN, g.a_rows, 0, 0);
      bool ok = true;
      int left = 0, part = -1;
      bool first = true;
      int sa = 0, sb = 0;
      uint32_t pa = 0, pb = 0;
      for (int i = 0; i < ksteps && ok; ++i) {
        if (left == 0) {
          left = part_steps(i);
          first = true;
          ++part;
          if (!mbar_wait(acc_empty(part & 1), ((part >> 1) & 1) ^ 1, dead, g.status, 307)) { ok = false; break; }
        }
        // both polls are under way together: an answer takes some 200 cycles, also where it is yes
        const uint32_t a_there = mbar_try_wait(a_full(sa), pa), b_there = mbar_try_wait(b_full(sb), pb);
        if (!(a_there & b_there) && (!mbar_wait(a_full(sa), pa, dead, g.status, 302) || !mbar_wait(b_full(sb), pb, dead, g.status, 303))) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(part & 1) * BM, w = tmem + ACC_COLS + (uint32_t)sb * W_COLS;
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub) {
          const uint32_t a_addr = sA + (sa * SUB + sub) * a_bytes;
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)             // 16 k: 8 columns of W, 32 bytes along a row of X
            umma_f16_ts(d, w + (sub * (BK / 16) + kk) * 8, make_smem_desc_sw128(a_addr + kk * 32, 16u, 1024u), idesc, (!first || (sub | kk) != 0) ? 1u : 0u);
        }
        first = false;
        umma_commit(a_empty(sa));
        umma_commit(b_empty(sb));
        if (++sa == a_stages) { sa = 0; pa ^= 1; }
        if (++sb == B_STAGES) { sb = 0; pb ^= 1; }
        if (--left == 0) umma_commit(acc_full(part & 1));
      }
    }
  } else if (warp >= 4 && warp < EPI_WARP0) {
    // Group gi has steps gi, gi + 2, ..: while one waits for its buffers or for the answers to its polls, the other converts.
    // A thread has one feature (a lane of tensor memory) and one 64-k block of a step.
    const int gi = (warp - 4) / GROUP_WARPS, quad = warp & 3, sub = ((warp - 4) >> 2) & 1, f = quad * 32 + lane;
    const uint8_t* const raw0 = raw_s + sub * RAW_BYTES + f * 16;
    const uint8_t* const scale0 = raw_s + sub * RAW_BYTES + NIB_BYTES + (quad >> 1) * (BK * 2);
    const uint32_t dst0 = tmem + ((uint32_t)(quad * 32) << 16) + ACC_COLS + sub * (BK / 2);
    uint32_t mask = 0x000F000Fu, magic = 0x43004300u;
    asm volatile("" : "+r"(mask), "+r"(magic));
    const __nv_bfloat162 off = __float2bfloat162_rn(136.0f);
    int r = gi, s = gi;
    uint32_t pr = 0, ps = 1;
    if (r >= RAW_STAGES) { r -= RAW_STAGES; pr ^= 1; }
    for (int i = gi; i < ksteps; i += GROUPS) {
      // one lane polls for the warp (256+ threads hammering one barrier word cost ~150 cycles a wait), both barriers at once
      uint32_t got = 1;
      if (lane == 0) {
        const uint32_t raw_there = mbar_try_wait(raw_full(r), pr), b_there = mbar_try_wait(b_empty(s), ps);
        got = raw_there & b_there;
        if (!got) got = mbar_wait(raw_full(r), pr, dead, g.status, 304) && mbar_wait(b_empty(s), ps, dead, g.status, 305);
      }
      if (!__shfl_sync(0xffffffffu, got, 0)) break;
      tc_fence_after();
      const uint8_t* raw = raw0 + r * (SUB * RAW_BYTES);
      const uint8_t* scales = scale0 + r * (SUB * RAW_BYTES);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint4 w4 = *reinterpret_cast<const uint4*>(raw + half * (NIB_BYTES / 2));
        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        uint32_t t[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 s4 = *reinterpret_cast<const uint4*>(scales + (half * 4 + c) * 16);      // of eight k, for all lanes
          const uint32_t sc[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t u = pick(w[c] >> (4 * j), mask, magic);        // bf16 (128 + q + 8) of k 2 j and 2 j + 1
            const __nv_bfloat162 h = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&u), off), *reinterpret_cast<const __nv_bfloat162*>(&sc[j]));
            t[4 * c + j] = *reinterpret_cast<const uint32_t*>(&h);
          }
        }
        __syncwarp();
        tmem_st16(dst0 + s * W_COLS + half * 16, t);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(b_full(s)); mbar_arrive(raw_empty(r)); }
      r += GROUPS;
      if (r >= RAW_STAGES) { r -= RAW_STAGES; pr ^= 1; }
      s += GROUPS;
      if (s >= B_STAGES) { s -= B_STAGES; ps ^= 1; }
    }
  } else if (warp >= EPI_WARP0) {
    // ---- epilogue: lane = output feature of the tile, accumulator column = row of X.
    // Every thread goes through every part and its barriers, also after a wait that gave up (later waits return at once).
    const int q = warp & 3, et = threadIdx.x - 32 * EPI_WARP0, f = q * 32 + lane;
    bool ok = true;
    int part = 0;
    for (int i = 0; i < ksteps; ++part) {
      const int nt = line(i) / k_tiles, n0 = nt * BN, a = part & 1;
      // the CTAs that share a left-over tile
      const uint32_t t0 = (uint32_t)((nt - whole) * k_tiles);
      const int lo = nt < whole ? 0 : pieces.first(nt - whole), hi = nt < whole ? 0 : pieces.last(nt - whole);
      // a CTA's piece may end one shared tile and begin another: slot 0 for the part it begins with, 1 for the other
      float* const mine = lo == hi ? nullptr : reinterpret_cast<float*>(part_slot(g, mt, cta, i != own)) + f;
      const float bias = g.bias && !mine ? __bfloat162float(g.bias[n0 + f]) : 0.0f;
      i += part_steps(i);
      ok = __all_sync(0xffffffffu, mbar_wait(acc_full(a), (part >> 1) & 1, dead, g.status, 306)) && ok;
      tc_fence_after();
      if (ok) {
        const int rows = min(g.a_rows, g.M - m0);
        float* const out_f = (float*)g.out + (long long)m0 * g.ldo + n0 + f;
        __nv_bfloat16* const out_b = (__nv_bfloat16*)g.out + (long long)m0 * g.ldo + n0 + f;
#pragma unroll 1
        for (int c = 0; c < g.a_rows; c += 16) {
          uint32_t rr[16];
          __syncwarp();
          tmem_ld16(tmem + a * BM + ((uint32_t)(q * 32) << 16) + c, rr);
          tmem_ld_wait();
          if (mine) {
#pragma unroll
            for (int j = 0; j < 16; ++j) mine[(c + j) * BN] = __uint_as_float(rr[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float v = __uint_as_float(rr[j]) + bias;
              if (c + j >= rows) break;
              if (g.out_f32) out_f[(c + j) * g.ldo] = v;
              else out_b[(c + j) * g.ldo] = __float2bfloat16(v);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(a));
      if (lo == hi) continue;
      // the CTA that arrives last at the tile's counter turns the parts into the output
      asm volatile("bar.sync 1, 128;" ::: "memory");
      int* counter = g.counters + mt * n_tiles + nt;
      if (et == 0) *is_last = arrive_acq_rel(counter) == hi - lo && !*dead;      // the barriers hand the others' parts to this thread and its view to them
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (i == ksteps) break;                               // the CTA's last part: all its threads take part in the sum, below
      if (*is_last) {
        sum_parts(g, mt, nt, lo, hi, pieces.begin(lo) < t0, et, 128);
        if (et == 0) *counter = 0;
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");        // is_last has been read
    }
  }
  if (*dead) __nanosleep(100000);
  tc_fence_before();
  __syncthreads();
  if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
  if (ksteps > own && *is_last) {
    const int nt = line(ksteps - 1) / k_tiles;
    const uint32_t t0 = (uint32_t)((nt - whole) * k_tiles);
    const int lo = pieces.first(nt - whole), hi = pieces.last(nt - whole);
    if (lo != hi) {
      sum_parts(g, mt, nt, lo, hi, pieces.begin(lo) < t0, threadIdx.x, THREADS);
      if (threadIdx.x == 0) g.counters[mt * n_tiles + nt] = 0;
    }
  }
}

// packed [K][N/2] bytes + scales (flat groups) -> tiles [N/128][K/64][4352].  A thread has eight columns of half a block's k.
// 4096 x 32000: 39 us (92 with single nibbles out of eight rows for every word).
__global__ void __launch_bounds__(256)
int4_tile_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ scales, int K, int N, int group, uint8_t* __restrict__ tiles) {
  const int k_tiles = K / BK, groups = N / group;
  const long long blk = ((long long)blockIdx.x * 256 + threadIdx.x) >> 5;
  if (blk >= (long long)(N / BN) * k_tiles) return;
  const int nt = (int)(blk / k_tiles), ks = (int)(blk % k_tiles), t = threadIdx.x & 31, c8 = t & 15, half = t >> 4;
  uint8_t* const dst = tiles + blk * RAW_BYTES;
  const uint8_t* const src = packed + ((long long)(ks * BK + half * 32) * N + nt * BN) / 2 + c8 * 4;
  uint32_t w[4][8];                                                       // [eight k][nibble of the result: k 2 j at j, 2 j + 1 at j + 4]
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int e = 0; e < 8; ++e) w[c][e] = load_nibbles(src + (long long)(c * 8 + (e & 3) * 2 + (e >> 2)) * (N / 2), true) ^ 0x88888888u;
  float s[4];                                                             // scales of four k of a half of the columns
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = scales[(long long)(ks * BK + c8 * 4 + j) * groups + (nt * BN + half * 64) / group];
#pragma unroll
  for (int c = 0; c < 4; ++c) transpose_nibbles(w[c]);
#pragma unroll
  for (int g = 0; g < 8; ++g) *reinterpret_cast<uint4*>(dst + half * (NIB_BYTES / 2) + (c8 * 8 + g) * 16) = make_uint4(w[0][g], w[1][g], w[2][g], w[3][g]);
  *reinterpret_cast<uint2*>(dst + NIB_BYTES + half * (BK * 2) + c8 * 8) = make_uint2(pack_bf16x2(s[0], s[1]), pack_bf16x2(s[2], s[3]));
}
}  // namespace

CGK_API long long cgk_int4_tiles_bytes(int K, int N) { return (long long)(N / BN) * (K / BK) * RAW_BYTES; }
// Reorders reference-format weights (packed [K, N/2] bytes, fp32 scales per flat group) into the
// tile-major stream the GEMM reads.  group: a multiple of 64 with N % group == 0.
CGK_API int cgk_int4_tile_weights(const void* packed, const float* scales, int K, int N, int group, void* tiles, void* stream) {
  CGK_REQUIRE(packed && scales && tiles, "cgk_int4_tile_weights: null pointer");
  CGK_REQUIRE(N % BN == 0 && K % BK == 0, "cgk_int4_tile_weights: need N %% 128 == 0 and K %% 64 == 0 (got K=%d N=%d)", K, N);
  CGK_REQUIRE(group >= 64 && group % 64 == 0 && N % group == 0, "cgk_int4_tile_weights: group %d must be a multiple of 64 that divides N", group);
  CGK_REQUIRE(((uintptr_t)packed & 3) == 0 && ((uintptr_t)tiles & 15) == 0, "cgk_int4_tile_weights: misaligned buffer");
  const long long blocks = (long long)(N / BN) * (K / BK);
  int4_tile_kernel<<<(unsigned)((blocks * 32 + 255) / 256), 256, 0, (cudaStream_t)stream>>>((const uint8_t*)packed, scales, K, N, group, (uint8_t*)tiles);
  CGK_LAUNCH_CHECK();
  return 0;
}
// one per output tile; the smallest tiles of cgk_int4_wa_gemm are 32 x 32
CGK_API long long cgk_int4_gemm_counters(int M, int N) { return (long long)((M + 31) / 32) * (N / 32); }

// How the tiles are dealt out: one CTA per SM (of a row tile's share of them), each with at least two steps of the left-over
// tiles; given splits: that many equal parts of every tile; without a place for parts: whole tiles.
// The left-over tiles, by the fewest steps of: each tile's steps in p pieces of its own (1: the tile stays whole), 2 p steps' worth of
// time for storing and summing the parts; or the line of all their steps in equal pieces, 10 for parts of two tiles in most CTAs and
// tiles that wait for CTAs which have another one to end first.  80 rows, line / own pieces: 4096 x 4096 (4 pieces) 12.1 / 10.2 us,
// 4096 x 22016 (4) 31.4 / 24.8, 4096 x 6144 (3) 13.1 / 11.4, 2048 x 11264 (whole, 88 CTAs) 12.0 / 11.3; 11008 x 4096 stays a line
// (17.0 / 17.0), 4096 x 32000 has 102 whole tiles (35.2 / 34.3).
struct Deal { long long ctas, sharers; int per_tile; };
static Deal deal(int sms, int M, int N, int K, int splits, bool parts) {
  const long long n_tiles = N / BN, m_tiles = (M + BM - 1) / BM, ksteps = K / (SUB * BK);
  if (splits > 0 || !parts) return {n_tiles * (splits > 0 ? splits : 1), splits > 1 ? n_tiles * splits : 1, splits > 1 ? splits : 0};
  long long ctas = sms / m_tiles;
  if (ctas > n_tiles * ksteps / 2) ctas = n_tiles * ksteps / 2;
  if (ctas < 1) ctas = 1;
  const long long left = n_tiles % ctas, rest = left * ksteps;
  if (left == 0) return {ctas, 1, 0};
  const long long most = rest / 2 < 1 ? 1 : rest / 2 < ctas ? rest / 2 : ctas, longest = (rest + most - 1) / most;
  long long best = longest + 10;
  Deal d = {ctas, (rest + longest - 1) / longest, 0};                        // the fewest sharers with the same longest piece
  for (long long p = ctas / left < ksteps / 2 ? ctas / left : ksteps / 2; p >= 1; --p) {
    const long long cost = (ksteps + p - 1) / p + (p > 1 ? 2 * p : 0);
    if (cost <= best) { best = cost; d = {ctas, left * p, (int)p}; }
  }
  return d;
}
static int part_rows(int M) { return M > BM ? BM : (M + 15) / 16 * 16; }

CGK_API long long cgk_int4_gemm_parts_floats(int M, int N, int K, int splits) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || M <= 0 || N < BN || K < SUB * BK) return 0;
  const Deal d = deal(cgk::sm_count(dev), M, N, K, splits, true);
  return (long long)((M + BM - 1) / BM) * d.sharers * 2 * BN * part_rows(M);
}

static int wb_gemm(const void* x, long long ldx, const void* w_tiles, float* parts, int* counters, void* out, long long ldo,
                   const void* bias, int M, int N, int K, int splits, int out_f32, void* stream) {
  using namespace cgk;
  CGK_REQUIRE(x && w_tiles && out, "cgk_int4_gemm: null pointer");
  CGK_REQUIRE(M > 0 && N > 0 && K > 0 && N % BN == 0 && K % (SUB * BK) == 0, "cgk_int4_gemm: need N %% 128 == 0 and K %% 128 == 0 (got M=%d N=%d K=%d)", M, N, K);
  CGK_REQUIRE(ldx % 8 == 0 && ldo % 8 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w_tiles & 15) == 0 && ((uintptr_t)out & 15) == 0 && ((uintptr_t)parts & 15) == 0,
              "cgk_int4_gemm: operands must be 16-byte aligned with leading dimensions that are multiples of 8");
  int dev = 0;
  CGK_CUDA_CHECK(cudaGetDevice(&dev));
  const int m_tiles = (M + BM - 1) / BM, ksteps = K / (SUB * BK);
  CGK_REQUIRE(splits <= 0 || ksteps % splits == 0, "cgk_int4_gemm: K/128 = %d is not divisible by splits = %d", ksteps, splits);
  CGK_REQUIRE(splits <= 1 || (parts && counters), "cgk_int4_gemm: split-K needs scratch and counters");
  const Deal d = deal(sm_count(dev), M, N, K, splits, parts && counters);
  const int a_rows = part_rows(M);
  // X comes from L2 a microsecond after it is asked for: six stages of it, at least three, as long as eight of W fit beside them
  int a_stages = 6;
  while (a_stages > 3 && RING_BUDGET - a_stages * SUB * a_rows * 128 < 8 * SUB * RAW_BYTES) --a_stages;
  if (a_stages > MAX_A_STAGES) a_stages = MAX_A_STAGES;
  int raw_stages = (RING_BUDGET - a_stages * SUB * a_rows * 128) / (SUB * RAW_BYTES);
  if (raw_stages > MAX_RAW_STAGES) raw_stages = MAX_RAW_STAGES;
  static const int raw_cap = getenv("CGK_INT4_RAW_STAGES") ? atoi(getenv("CGK_INT4_RAW_STAGES")) : 0;
  if (raw_cap > 0 && raw_cap < raw_stages) raw_stages = raw_cap;
  if (raw_stages < MIN_RAW_STAGES) raw_stages = MIN_RAW_STAGES;
  CUtensorMap tmX;
  int rc = encode_tmap_bf16_2d(&tmX, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)a_rows, BK);
  if (rc) return rc;
  static bool attr_set[64] = {};
  if (dev < 64 && !attr_set[dev]) {
    CGK_CUDA_CHECK(cudaFuncSetAttribute(int4_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    attr_set[dev] = true;
  }
  // a line to deal (each left-over tile's, or all of theirs) and its pieces
  const long long steps = (long long)(d.per_tile ? 1 : N / BN % d.ctas) * ksteps, pieces = d.per_tile ? d.per_tile : d.sharers;
  Int4Dev g{(const uint8_t*)w_tiles, (float4*)parts, counters, out, ldo, (const __nv_bfloat16*)bias, M, N, K, out_f32,
            a_rows, a_stages, raw_stages, (int)d.sharers, d.per_tile, (int)(steps / pieces), (int)(steps % pieces), device_status(dev)};
  CGK_CUDA_CHECK(launch_overlapped(int4_gemm_kernel, dim3((unsigned)d.ctas, m_tiles), dim3(THREADS), SMEM_BYTES, (cudaStream_t)stream, 0, tmX, g));
  return 0;
}

// x bf16 [M, ldx]; w_tiles from cgk_int4_tile_weights; out bf16 [M, ldo]; bias bf16 [N] or null.  parts (fp32
// [cgk_int4_gemm_parts_floats], any contents) and counters (int32 [cgk_int4_gemm_counters], zero before the first call and left
// zero by every call) serve tiles shared by several CTAs; without them every tile is computed whole.  splits 0 = chosen here.
CGK_API int cgk_int4_gemm_parts(const void* x, long long ldx, const void* w_tiles, float* parts, int* counters, void* out, long long ldo,
                                const void* bias, int M, int N, int K, int splits, void* stream) {
  return wb_gemm(x, ldx, w_tiles, parts, counters, out, ldo, bias, M, N, K, splits, 0, stream);
}
// The same with an fp32 output (logits).
CGK_API int cgk_int4_gemm_parts_f32(const void* x, long long ldx, const void* w_tiles, float* parts, int* counters, float* out, long long ldo,
                                    const void* bias, int M, int N, int K, int splits, void* stream) {
  return wb_gemm(x, ldx, w_tiles, parts, counters, out, ldo, bias, M, N, K, splits, 1, stream);
}

// The same for callers that hold an accumulator (fp32 [M, N], zero, left zero) instead of parts, which then come from the stream's
// memory pool (whole tiles where that has none left).
CGK_API int cgk_int4_gemm(const void* x, long long ldx, const void* w_tiles, float* acc, int* counters, void* out, long long ldo,
                          const void* bias, int M, int N, int K, int splits, void* stream) {
  const bool shared = acc && counters;
  return cgk::with_stream_scratch(shared ? cgk_int4_gemm_parts_floats(M, N, K, splits) : 0, (cudaStream_t)stream, [&](float* parts) {
    return wb_gemm(x, ldx, w_tiles, parts, parts ? counters : nullptr, out, ldo, bias, M, N, K, shared && !parts ? 0 : splits, 0, stream);
  });
}
