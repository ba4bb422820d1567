// INT4 weight-only GEMM for serving: out[M,N] = X[M,K] (bf16) . dequant(W)[K,N] (+ bias).
//
// W holds the reference's quantised values (src/quantize/int4.c:10-59, 90-114: row-major [K,N],
// 4-bit two's complement, even column in the low nibble, one fp32 scale per flat group of
// `group` elements), reordered tile-major without re-quantising: for n-tile nt (128 columns)
// and k-step ks (64 rows) one contiguous 4608-byte block holds the tile's 64 rows of 64 bytes
// followed by the tile's scales as fp32 [64 rows][2 column halves].  A CTA's slab is then one
// sequential stream, which is what keeps HBM efficient (64-byte pieces of the row-major
// layout are not); cgk_int4_tile_weights does the reordering.
//
// The shape is weight-bandwidth bound (M <= 128 rows against megabytes of weights):
//   warp 0    bulk copies of W blocks into a 12-deep ring (bytes in flight cover HBM latency)
//   warp 3    TMA: X tiles [rows, 64 k] into their own ring of up to 12 stages; only
//             round_up(M, 8) rows are fetched — the tensor core still multiplies 128 rows, the
//             others hold whatever shared memory held and only feed output rows nobody stores
//   warps 4-19 nibbles -> bf16: exact integer (magic-number trick), one multiply by the scale,
//             stored in the 128-byte-swizzled MN-major operand layout tcgen05 reads.  Columns
//             stay in the pair order the extraction yields (0,4,1,5,2,6,3,7 within each group
//             of 8); the epilogue undoes the permutation when it addresses the output.
//   warp 1    tcgen05.mma, two accumulators in TMEM (128 lanes x 128 columns)
//   warps 20-23 epilogue.  Whole tile: TMEM -> bias -> bf16 -> global.  Part of a tile: into the part's
//             own fp32 slot; the CTA that arrives last at the tile's counter sums the slots in the
//             order of the CTAs, adds the bias, writes bf16 and leaves the counter zeroed for the
//             next call.  The order is fixed, so a call gives the same bits every time.
// One CTA per SM.  Each takes as many whole tiles as there are for all of them, then an equal piece of the line of the left-over
// tiles' steps of 128 k (see int4_gemm_wa.cu).  Whole tiles only left 172 of them (22 016 columns) in two waves on 148 SMs, and a
// K of 11 008 on 64 CTAs.  80 rows, layers one after the other, whole tiles or equal parts of them by atomics / like this: 4096 x 22016
// 68.8 / 46.5 us, 11008 x 4096 52.1 / 28.7, 4096 x 32000 70.1 / 61.6, 2048 x 11264 (a tile per CTA on 88 SMs) 19.9 / 19.5.
// The sum of the CTA's last shared tile is work of all its threads: by the epilogue's 128 these took 50.9, 33.3, 64.7 and 24.0.
#include <cuda_bf16.h>
#include <stdlib.h>

#include "host_common.h"
#include "mma_sync.cuh"
#include "cogito_kernels.h"

namespace {
using namespace cgk;

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int ISSUE_LANES = 8;                                // threads of a producer warp that issue copies
constexpr int SUB = 2;                                        // 64-row sub-tiles per pipeline step (a step covers 128 k)
constexpr int B_STAGES = 3, MAX_RAW_STAGES = 16, MAX_A_STAGES = 8;
constexpr int GROUPS = 2, GROUP_WARPS = 8, CONVERT_WARPS = GROUPS * GROUP_WARPS;     // converting warps: groups that take the steps in turn
constexpr int B_BYTES = BK * BN * 2;
constexpr int NIB_BYTES = BK * BN / 2, SCALE_BYTES = BK * 2 * 4, RAW_BYTES = NIB_BYTES + SCALE_BYTES;   // 4096 + 512
constexpr int EPI_WARP0 = 4 + CONVERT_WARPS, THREADS = 32 * (EPI_WARP0 + 4);
constexpr int SMEM_BYTES = 226 * 1024;                       // alignment slack | X ring | B ring | W ring | barriers
constexpr int RING_BUDGET = SMEM_BYTES - 1024 - B_STAGES * SUB * B_BYTES - 2048;   // shared by the X and W rings

struct Int4Dev {
  const uint8_t* w_tiles;          // [N/128][K/64][4608]
  float4* parts;                   // slots of shared tiles' parts: [m_tiles][sharers][2][32 column quads][a_rows]
  int* counters;                   // int32 [m_tiles * n_tiles], zero between calls (shared tiles only)
  void* out; long long ldo;        // bf16, or fp32 with out_f32
  const __nv_bfloat16* bias;
  int M, N, K, out_f32;
  int a_rows, a_stages;            // rows fetched per X tile (multiple of 8), depth of the X ring
  int raw_stages;                  // depth of the W ring
  int sharers;                     // CTAs that the left-over tiles are dealt to
  int* status;
};

// Slot `which` of a sharer: [32 column quads][a_rows] float4s.
__device__ __forceinline__ float4* part_slot(const Int4Dev& g, int mt, int sharer, int which) {
  return g.parts + (long long)((mt * g.sharers + sharer) * 2 + which) * ((BN / 4) * g.a_rows);
}

// Eight neighbouring elements of the output.
__device__ __forceinline__ void store8(const Int4Dev& g, long long at, const float4& u, const float4& v) {
  if (g.out_f32) {
    float4* p = reinterpret_cast<float4*>((float*)g.out + at);
    p[0] = u;
    p[1] = v;
  } else {
    *reinterpret_cast<uint4*>((__nv_bfloat16*)g.out + at) = make_uint4(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
  }
}

// The output of a tile out of its parts, summed in the order of the CTAs lo .. hi; `first`: the slot that CTA lo's is in.
__device__ __forceinline__ void sum_parts(const Int4Dev& g, int mt, int nt, int lo, int hi, int first_slot, int tid, int threads) {
  __threadfence();
  const int m0 = mt * BM, n0 = nt * BN, rows = min(BM, g.M - m0), stride = 2 * (BN / 4) * g.a_rows;
  const float4* first = part_slot(g, mt, lo, first_slot);
  const float4* others = part_slot(g, mt, lo, 0);
  for (int e = tid; e < rows * (BN / 8); e += threads) {
    const int c8 = e / rows, r = e - c8 * rows, at = 2 * c8 * g.a_rows + r, n = n0 + c8 * 8;
    float4 u = __ldcg(first + at), v = __ldcg(first + at + g.a_rows);
#pragma unroll 4
    for (int c = 1; c <= hi - lo; ++c) {
      const float4* src = others + (long long)c * stride + at;
      const float4 x = __ldcg(src), y = __ldcg(src + g.a_rows);
      u.x += x.x; u.y += x.y; u.z += x.z; u.w += x.w;
      v.x += y.x; v.y += y.y; v.z += y.z; v.w += y.w;
    }
    if (g.bias) {
      u.x += __bfloat162float(g.bias[n]); u.y += __bfloat162float(g.bias[n + 1]);
      u.z += __bfloat162float(g.bias[n + 2]); u.w += __bfloat162float(g.bias[n + 3]);
      v.x += __bfloat162float(g.bias[n + 4]); v.y += __bfloat162float(g.bias[n + 5]);
      v.z += __bfloat162float(g.bias[n + 6]); v.w += __bfloat162float(g.bias[n + 7]);
    }
    store8(g, (long long)(m0 + r) * g.ldo + n, u, v);
  }
}

__global__ void __launch_bounds__(THREADS, 1)
int4_gemm_kernel(const __grid_constant__ CUtensorMap tmX, const Int4Dev g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t sA = base;                                         // a_stages x (a_rows * 128 B); reads of 128 rows may run into sB
  const uint32_t sB = sA + (uint32_t)g.a_stages * SUB * (uint32_t)g.a_rows * 128u;   // B_STAGES x SUB x 16 KiB
  const uint32_t sRaw = sB + B_STAGES * SUB * B_BYTES;              // raw_stages x SUB x 4608 B
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
  const Pieces pieces((uint32_t)((n_tiles - whole) * k_tiles), (uint32_t)sharers);
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
  if (warp == 2) { tmem_alloc(smem_u32(tmem_slot), 2 * BN); tmem_relinquish(); }
  // the first weights (no earlier kernel's business) start on their way to L2 while the predecessor still runs
  if (warp == 0 && blockIdx.y == 0 && lane < min(ksteps, 14)) prefetch_l2(g.w_tiles + (long long)line(lane) * (SUB * RAW_BYTES), SUB * RAW_BYTES);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  pdl_wait();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // A thread's bulk copies run one after the other (measured: ~0.43 us each, whatever the ring
    // depth), so several lanes issue, each with its own copies in flight.  A ring slot always
    // belongs to the same lane: its uses are then waited for in order, which the one-bit phase
    // parity of an mbarrier requires.
    if (lane < ISSUE_LANES) {
      int r = 0;
      uint32_t par = 1;
      for (int i = 0; i < ksteps; ++i) {
        const int here = r;
        const uint32_t phase = par;
        if (++r == RAW_STAGES) { r = 0; par ^= 1; }
        if (here % ISSUE_LANES != lane) continue;
        if (!mbar_wait(raw_empty(here), phase, dead, g.status, 300)) break;
        mbar_expect_tx(raw_full(here), SUB * RAW_BYTES);
        bulk_load_1d(sRaw + here * (SUB * RAW_BYTES), g.w_tiles + (long long)line(i) * (SUB * RAW_BYTES), SUB * RAW_BYTES, raw_full(here));
      }
    }
  } else if (warp == 3) {
    if (lane < ISSUE_LANES) {
      if (lane == 0) tma_prefetch_desc(&tmX);
      int next = 0;
      uint32_t par = 1;
      for (int i = 0; i < ksteps; ++i) {
        const int s = next;
        const uint32_t phase = par;
        if (++next == a_stages) { next = 0; par ^= 1; }
        if (s % ISSUE_LANES != lane) continue;
        const int ks = line(i) % k_tiles;                             // step within its tile
        if (!mbar_wait(a_empty(s), phase, dead, g.status, 301)) break;
        mbar_expect_tx(a_full(s), SUB * a_bytes);
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub)
          tma_load_2d(sA + (s * SUB + sub) * a_bytes, &tmX, a_full(s), (ks * SUB + sub) * BK, m0);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, BN, 0, 1);
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
        const uint32_t d = tmem + (uint32_t)(part & 1) * BN;
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub) {
          const uint32_t a_addr = sA + (sa * SUB + sub) * a_bytes, b_addr = sB + (sb * SUB + sub) * B_BYTES;
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            umma_f16(d, make_smem_desc_sw128(a_addr + kk * 32, 16u, 1024u), make_smem_desc_sw128(b_addr + kk * 2048, 8192u, 1024u), idesc,
                     (!first || (sub | kk) != 0) ? 1u : 0u);
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
    const int gi = (warp - 4) / GROUP_WARPS, tid = threadIdx.x - 128 - gi * (32 * GROUP_WARPS);
    constexpr int WORDS = BK * BN / 8 / (32 * GROUP_WARPS);            // per thread and 64-row sub-tile: rows 16 apart, the same 8 columns
    const int k0 = tid >> 4, jw = tid & 15;
    const uint8_t* const raw0 = raw_s + tid * 4;
    const uint8_t* const scale0 = raw_s + NIB_BYTES + k0 * 8 + (jw >> 3) * 4;
    const uint32_t dst0 = sB + (jw >> 3) * 8192u + sw128_offset((uint32_t)k0, (uint32_t)(jw & 7));    // 16 rows on: 2048 bytes
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
      const uint8_t* raw = raw0 + r * (SUB * RAW_BYTES);
      const uint8_t* scales = scale0 + r * (SUB * RAW_BYTES);
      const uint32_t dst = dst0 + s * (SUB * B_BYTES);
#pragma unroll
      for (int sub = 0; sub < SUB; ++sub) {
        uint32_t v[WORDS];
        float sc[WORDS];
#pragma unroll
        for (int it = 0; it < WORDS; ++it) {
          v[it] = *reinterpret_cast<const uint32_t*>(raw + sub * RAW_BYTES + it * (32 * GROUP_WARPS * 4));
          sc[it] = *reinterpret_cast<const float*>(scales + sub * RAW_BYTES + it * (16 * 8));
        }
#pragma unroll
        for (int it = 0; it < WORDS; ++it) {
          const uint32_t w = v[it] ^ 0x88888888u;          // two's complement -> q + 8
          const __nv_bfloat162 sc2 = __float2bfloat162_rn(sc[it]);
          uint32_t t[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t u = pick(w >> (4 * j), mask, magic);           // bf16 (128 + q + 8) for columns j and j + 4
            const __nv_bfloat162 h = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&u), off), sc2);
            t[j] = *reinterpret_cast<const uint32_t*>(&h);
          }
          // positions 0..7 of the chunk hold columns 0,4,1,5,2,6,3,7
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + sub * B_BYTES + it * 2048), "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]) : "memory");
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { mbar_arrive(b_full(s)); mbar_arrive(raw_empty(r)); }
      r += GROUPS;
      if (r >= RAW_STAGES) { r -= RAW_STAGES; pr ^= 1; }
      s += GROUPS;
      if (s >= B_STAGES) { s -= B_STAGES; ps ^= 1; }
    }
  } else if (warp >= EPI_WARP0) {
    // ---- epilogue: lane = output row inside the 128-row tile.
    // Accumulator positions j..j+7 of a group of 8 are columns j + {0,4,1,5,2,6,3,7}.
    // Every thread goes through every part and its barriers, also after a wait that gave up (later waits return at once).
    const int q = warp & 3, et = threadIdx.x - 32 * EPI_WARP0, row = m0 + q * 32 + lane;
    bool ok = true;
    int part = 0;
    for (int i = 0; i < ksteps; ++part) {
      const int nt = line(i) / k_tiles, n0 = nt * BN, a = part & 1;
      // the CTAs that share a left-over tile
      const uint32_t t0 = (uint32_t)((nt - whole) * k_tiles);
      const int lo = nt < whole ? 0 : (int)pieces.of(t0), hi = nt < whole ? 0 : (int)pieces.of(t0 + k_tiles - 1);
      // a CTA's piece may end one shared tile and begin another: slot 0 for the part it begins with, 1 for the other
      float4* const mine = part_slot(g, mt, cta, i != own) + q * 32 + lane;
      i += part_steps(i);
      ok = __all_sync(0xffffffffu, mbar_wait(acc_full(a), (part >> 1) & 1, dead, g.status, 306)) && ok;
      tc_fence_after();
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t rr[32];
          __syncwarp();
          tmem_ld32(tmem + a * BN + ((uint32_t)(q * 32) << 16) + c, rr);
          tmem_ld_wait();
          // a slot takes all its rows, so that no memory sector is written in part (17 rows, 4096 x 22016, cold caches: 55 -> 51 us)
          if (lo == hi ? row >= g.M : q * 32 + lane >= g.a_rows) continue;
          if (lo == hi) {
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float v[8] = {__uint_as_float(rr[j]), __uint_as_float(rr[j + 2]), __uint_as_float(rr[j + 4]), __uint_as_float(rr[j + 6]),
                            __uint_as_float(rr[j + 1]), __uint_as_float(rr[j + 3]), __uint_as_float(rr[j + 5]), __uint_as_float(rr[j + 7])};
              if (g.bias) {
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] += __bfloat162float(g.bias[n0 + c + j + e]);
              }
              store8(g, (long long)row * g.ldo + n0 + c + j, make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]));
            }
          } else {
            // neighbouring lanes hold neighbouring rows: 16 bytes each, side by side
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              float4* dstp = mine + (c + j) / 4 * g.a_rows;
              dstp[0] = make_float4(__uint_as_float(rr[j]), __uint_as_float(rr[j + 2]), __uint_as_float(rr[j + 4]), __uint_as_float(rr[j + 6]));
              dstp[g.a_rows] = make_float4(__uint_as_float(rr[j + 1]), __uint_as_float(rr[j + 3]), __uint_as_float(rr[j + 5]), __uint_as_float(rr[j + 7]));
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(a));
      if (lo == hi) continue;
      // the CTA that arrives last at the tile's counter turns the parts into the output
      __threadfence();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      int* counter = g.counters + mt * n_tiles + nt;
      if (et == 0) *is_last = (atomicAdd(counter, 1) == hi - lo) && !*dead;
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
  if (warp == 2) { tc_fence_after(); tmem_dealloc(tmem, 2 * BN); }
  if (ksteps > own && *is_last) {
    const int nt = line(ksteps - 1) / k_tiles;
    const uint32_t t0 = (uint32_t)((nt - whole) * k_tiles);
    const int lo = (int)pieces.of(t0), hi = (int)pieces.of(t0 + k_tiles - 1);
    if (lo != hi) {
      sum_parts(g, mt, nt, lo, hi, pieces.begin(lo) < t0, threadIdx.x, THREADS);
      if (threadIdx.x == 0) g.counters[mt * n_tiles + nt] = 0;
    }
  }
}

// packed [K][N/2] bytes + scales (flat groups) -> tiles [N/128][K/64][4608]
__global__ void int4_tile_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ scales, int K, int N, int group,
                                 uint8_t* __restrict__ tiles) {
  const int k_tiles = K / BK;
  const long long blocks = (long long)(N / BN) * k_tiles;
  for (long long blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
    const int nt = (int)(blk / k_tiles), ks = (int)(blk % k_tiles);
    uint8_t* dst = tiles + blk * RAW_BYTES;
    for (int i = threadIdx.x; i < NIB_BYTES / 4; i += blockDim.x) {
      const int k = i >> 4, wj = i & 15;
      reinterpret_cast<uint32_t*>(dst)[i] = *reinterpret_cast<const uint32_t*>(packed + ((long long)(ks * BK + k) * N + nt * BN) / 2 + wj * 4);
    }
    for (int i = threadIdx.x; i < BK * 2; i += blockDim.x) {
      const int k = i >> 1, half = i & 1;
      reinterpret_cast<float*>(dst + NIB_BYTES)[i] = scales[((long long)(ks * BK + k) * N + nt * BN + half * 64) / group];
    }
  }
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
  int4_tile_kernel<<<(unsigned)(blocks < 4736 ? blocks : 4736), 256, 0, (cudaStream_t)stream>>>((const uint8_t*)packed, scales, K, N, group, (uint8_t*)tiles);
  CGK_LAUNCH_CHECK();
  return 0;
}
// one per output tile; the smallest tiles of cgk_int4_wa_gemm are 32 x 32
CGK_API long long cgk_int4_gemm_counters(int M, int N) { return (long long)((M + 31) / 32) * (N / 32); }

// How the tiles are dealt out: one CTA per SM (of a row tile's share of them), each with at least two steps of the left-over
// tiles; given splits: that many equal parts of every tile; without a place for parts: whole tiles.
struct Deal { long long ctas, sharers; };
static Deal deal(int sms, int M, int N, int K, int splits, bool parts) {
  const long long n_tiles = N / BN, m_tiles = (M + BM - 1) / BM, ksteps = K / (SUB * BK);
  if (splits > 0 || !parts) return {n_tiles * (splits > 0 ? splits : 1), splits > 1 ? n_tiles * splits : 1};
  long long ctas = sms / m_tiles;
  if (ctas > n_tiles * ksteps / 2) ctas = n_tiles * ksteps / 2;
  if (ctas < 1) ctas = 1;
  // the fewest sharers with the same longest piece: fewer parts to store and to sum
  const long long rest = n_tiles % ctas * ksteps, most = rest / 2 < 1 ? 1 : rest / 2 < ctas ? rest / 2 : ctas, longest = (rest + most - 1) / most;
  return {ctas, rest > 0 ? (rest + longest - 1) / longest : 1};
}
static int part_rows(int M) { return M > BM ? BM : (M + 7) / 8 * 8; }

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
  // X comes from L2 a microsecond after it is asked for: four stages of it, as long as five of W fit beside them (at least 2),
  // and up to a quarter of the ring budget where rows are few
  int a_stages = (RING_BUDGET / 4) / (SUB * a_rows * 128);
  if (a_stages < 4) a_stages = 4;
  while (a_stages > 2 && RING_BUDGET - a_stages * SUB * a_rows * 128 < 5 * SUB * RAW_BYTES) --a_stages;
  if (a_stages > MAX_A_STAGES) a_stages = MAX_A_STAGES;
  int raw_stages = (RING_BUDGET - a_stages * SUB * a_rows * 128) / (SUB * RAW_BYTES);
  if (raw_stages > MAX_RAW_STAGES) raw_stages = MAX_RAW_STAGES;
  static const int raw_cap = getenv("CGK_INT4_RAW_STAGES") ? atoi(getenv("CGK_INT4_RAW_STAGES")) : 0;
  if (raw_cap > 0 && raw_cap < raw_stages) raw_stages = raw_cap;
  CUtensorMap tmX;
  int rc = encode_tmap_bf16_2d(&tmX, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, (uint32_t)a_rows, BK);
  if (rc) return rc;
  static bool attr_set[64] = {};
  if (dev < 64 && !attr_set[dev]) {
    CGK_CUDA_CHECK(cudaFuncSetAttribute(int4_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    attr_set[dev] = true;
  }
  Int4Dev g{(const uint8_t*)w_tiles, (float4*)parts, counters, out, ldo, (const __nv_bfloat16*)bias, M, N, K, out_f32,
            a_rows, a_stages, raw_stages, (int)d.sharers, device_status(dev)};
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
