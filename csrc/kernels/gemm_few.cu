// bf16 GEMM for products with few output tiles: decoding (up to 128 rows against a whole weight matrix), small training
// batches, routers.  The persistent kernel of gemm_tcgen05.cu gives such a product as many CTAs as it has tiles, and a CTA
// streams its operands at a fraction of an SM's share of HBM; 2048 x 2048 weights with 32 rows are 32 tiles of 64 columns.
//
// Here a cluster of S CTAs computes one 128 x BN tile, each over its part of the K range (TMA ring -> tcgen05.mma -> TMEM),
// and the S partial tiles meet in shared memory: every CTA writes its accumulator there, and after one cluster barrier sums
// its share of the tile's rows over the cluster (distributed shared memory, ranks in order, so the result does not vary)
// and applies the epilogue.  No workspace, no atomics, no second kernel.  Rows beyond M are neither fetched (K-major A: the
// box has round_up(M, 8) rows; the tensor core multiplies what lies behind them into rows nobody reads) nor summed.  About
// 100 KB of shared memory per CTA, so two CTAs stream per SM and one's prologue runs under the other's loop.
#include "gemm_host.h"

namespace cgk {
namespace {

constexpr int FEW_THREADS = 256;                 // warp 0 loads, warp 1 issues, warp 2 allocates, warps 4-7 drain; all sum
constexpr int FEW_RING = 96 * 1024;              // A ring, then B ring; the partial tile overlays them afterwards
constexpr int FEW_MAX_STAGES = 8;
constexpr int FEW_SMEM = 1024 + FEW_RING + 256;

struct FewDev {
  int a_rows, stages;                            // rows of A per stage (multiple of 8), depth of the rings
  int vec4;                                      // the output takes four elements per store
  const __nv_bfloat16* b; long long ldb, strideB;
};

// epilogue_scalar for four neighbouring columns, all inside the output
__device__ __forceinline__ void epilogue4(const GemmDev& g, int b, int m, int n, float (&v)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] *= g.alpha;
    if (g.bias) v[j] += g.bias_fp32 ? reinterpret_cast<const float*>(g.bias)[n + j] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g.bias)[n + j]);
    if (g.aux_out) g.aux_out[(long long)m * g.ldaux + n + j] = __float2bfloat16(v[j]);
    if (g.act) v[j] = apply_act(g.act, v[j]);
    if (g.aux_in) v[j] *= apply_dact(g.dact, __bfloat162float(g.aux_in[(long long)m * g.ldauxin + n + j]));
    if (g.residual) v[j] += __bfloat162float(g.residual[(long long)m * g.ldr + n + j]);
  }
  bool fp32;
  void* dst = out_address(g, b, m, n, fp32);
  if (fp32) {
    float4* p = reinterpret_cast<float4*>(dst);
    float4 w = make_float4(v[0], v[1], v[2], v[3]);
    if (g.accumulate) {
      const float4 old = *p;
      w.x += old.x; w.y += old.y; w.z += old.z; w.w += old.w;
    }
    *p = w;
  } else {
    uint2* p = reinterpret_cast<uint2*>(dst);
    if (g.accumulate) {
      const uint2 old = *p;
      const float2 a = unpack_bf16x2(old.x), c = unpack_bf16x2(old.y);
      v[0] += a.x; v[1] += a.y; v[2] += c.x; v[3] += c.y;
    }
    *p = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
  }
}

template <int BN>
__global__ void __launch_bounds__(FEW_THREADS, 2)
gemm_few_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmDev g, const FewDev f) {
  constexpr int LDP = BN + 4;                    // floats per row of the partial tile: 16-byte rows that start in different banks
  static_assert(BM * LDP * 4 <= FEW_RING, "the partial tile overlays the rings");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t base = smem_u32(smem), bars = base + FEW_RING;
  const uint32_t a_bytes = (uint32_t)f.a_rows * 128u, sB = base + (uint32_t)f.stages * a_bytes;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (FEW_MAX_STAGES + s); };
  const uint32_t acc_full = bars + 8u * 2 * FEW_MAX_STAGES;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(smem + FEW_RING + 8 * (2 * FEW_MAX_STAGES + 1));
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_holder + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int S = g.split_k, rank = (int)blockIdx.x % S;
  int t = (int)blockIdx.x / S;
  const int b = t / (g.tiles_m * g.tiles_n);
  t -= b * (g.tiles_m * g.tiles_n);
  const int tn = t / g.tiles_m, m0 = (t - tn * g.tiles_m) * BM, n0 = tn * BN;
  const int kblocks = (g.K + BK - 1) / BK, kb0 = kblocks * rank / S, kb1 = kblocks * (rank + 1) / S;

  if (threadIdx.x == 0) {
    for (int s = 0; s < FEW_MAX_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(acc_full, 1);
    *dead = 0;
    mbar_fence_init();
  }
  if (warp == 2) {
    tmem_alloc(smem_u32(tmem_holder), BN);
    tmem_relinquish();
  }
  // B is a weight matrix where few rows meet it: this CTA's part of it (as much as its rings hold) starts on its way to L2 while the
  // predecessor still runs.  A prefetch has no result, so it does not matter who wrote the operand.
  if (warp >= 4 && !g.b_mn) {
    const int row = n0 + (int)threadIdx.x - 128, k = kb0 * BK, len = min(g.K, min(kb1, kb0 + FEW_MAX_STAGES) * BK) - k;
    if (row < min(g.N, n0 + BN) && len >= 8) prefetch_l2(f.b + b * f.strideB + (long long)row * f.ldb + k, (uint32_t)(len / 8 * 16));
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  pdl_trigger();
  pdl_wait();

  if (warp == 0) {
    if (elect_one()) {
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, s = i % f.stages;
        if (!mbar_wait(empty_bar(s), ((i / f.stages) & 1) ^ 1, dead, g.status, 400)) break;
        mbar_expect_tx(full_bar(s), a_bytes + BN * 128u);
        const uint32_t a = base + s * a_bytes, w = sB + s * (BN * 128u);
        if (!g.a_mn) {
          tma_load_3d(a, &tmA, full_bar(s), kb * BK, m0, b);
        } else {
#pragma unroll
          for (int blk = 0; blk < BM / 64; ++blk) tma_load_3d(a + blk * 8192, &tmA, full_bar(s), m0 + blk * 64, kb * BK, b);
        }
        if (!g.b_mn) {
          tma_load_3d(w, &tmB, full_bar(s), kb * BK, n0, b);
        } else {
#pragma unroll
          for (int blk = 0; blk < BN / 64; ++blk) tma_load_3d(w + blk * 8192, &tmB, full_bar(s), n0 + blk * 64, kb * BK, b);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, BN, g.a_mn, g.b_mn);
      const uint32_t a_lbo = g.a_mn ? 8192u : 16u, b_lbo = g.b_mn ? 8192u : 16u, a_k16 = g.a_mn ? 2048u : 32u, b_k16 = g.b_mn ? 2048u : 32u;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, s = i % f.stages;
        if (!mbar_wait(full_bar(s), (i / f.stages) & 1, dead, g.status, 401)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a = base + s * a_bytes, w = sB + s * (BN * 128u);
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
          umma_f16(tmem, make_smem_desc_sw128(a + kk * a_k16, a_lbo, 1024u), make_smem_desc_sw128(w + kk * b_k16, b_lbo, 1024u), idesc, (i | kk) != 0 ? 1u : 0u);
        umma_commit(empty_bar(s));
      }
      if (ok) umma_commit(acc_full);
    }
  } else if (warp >= 4) {
    const int q = warp & 3;
    // all MMAs are done with the rings once the accumulator is complete; the partial tile [rows][LDP] takes their place
    if (__all_sync(0xffffffffu, mbar_wait(acc_full, 0, dead, g.status, 402)) && q * 32 < f.a_rows) {
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        __syncwarp();
        tmem_ld32(tmem + c + ((uint32_t)(q * 32) << 16), r);
        tmem_ld_wait();
        float4* dst = reinterpret_cast<float4*>(smem) + ((q * 32 + lane) * LDP + c) / 4;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          dst[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
      }
    }
  }
  if (*dead) __nanosleep(100000);                // a role that gave up leaves copies in flight
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_sync_all();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem, BN);
  }
  const int units = min(BM, g.M - m0) * (BN / 4), per = (units + S - 1) / S;
  for (int u = rank * per + (int)threadIdx.x; u < min(units, (rank + 1) * per); u += FEW_THREADS) {
    const int row = u / (BN / 4), c = (u % (BN / 4)) * 4, m = m0 + row, n = n0 + c;
    if (n >= g.N) continue;
    const uint32_t at = base + (uint32_t)(row * LDP + c) * 4u;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int s = 0; s < S; ++s) {
      const float4 p = S > 1 ? ld_cluster_f4(cluster_map(at, s)) : *reinterpret_cast<const float4*>(smem + (at - base));
      v[0] += p.x; v[1] += p.y; v[2] += p.z; v[3] += p.w;
    }
    if (f.vec4 && n + 4 <= g.N) {
      epilogue4(g, b, m, n, v);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < g.N) epilogue_scalar(g, b, m, n + j, v[j]);
    }
  }
  if (S > 1) cluster_sync_all();                 // nobody leaves while its part is still read
}

template <int BN>
int launch(const cgk_gemm_args& a, GemmDev g, int S, cudaStream_t stream) {
  g.tiles_m = (a.M + BM - 1) / BM;
  g.tiles_n = (a.N + BN - 1) / BN;
  g.split_k = S;
  FewDev f;
  f.a_rows = (a.a_mn || a.M > BM) ? BM : (a.M + 7) / 8 * 8;
  // the MMA reads 128 rows from the start of A's last stage: the rows behind it are B's ring, inside the allocation
  const int stage = f.a_rows * 128 + BN * 128;
  f.stages = FEW_RING / stage < FEW_MAX_STAGES ? FEW_RING / stage : FEW_MAX_STAGES;
  const uintptr_t out = (uintptr_t)a.out;
  f.b = (const __nv_bfloat16*)a.B; f.ldb = a.ldb; f.strideB = a.strideB;
  f.vec4 = a.ldc % 4 == 0 && (a.batch == 1 || a.strideC % 4 == 0) && (out & (a.out_fp32 ? 15 : 7)) == 0;
  CUtensorMap tmA, tmB;
  int rc = make_gemm_tmaps(a, BN, &tmA, &tmB, f.a_rows);
  if (rc) return rc;
  CGK_CUDA_CHECK(cudaFuncSetAttribute(gemm_few_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, FEW_SMEM));
  CGK_CUDA_CHECK(launch_overlapped(gemm_few_kernel<BN>, dim3((unsigned)(g.batch * g.tiles_m * g.tiles_n * S)), dim3(FEW_THREADS), FEW_SMEM, stream, S, tmA, tmB, g, f));
  return 0;
}

}  // namespace

// Where the line lies (times with cold caches and about 7 us of event and launch in each, 128 x 64 tiles here / persistent kernel):
//   one row tile, while 128-column tiles fit two to an SM: 32 x 768 x 2048 13.1 / 18.4 us, x 2048 x 2048 14.3 / 19.2,
//   x 2048 x 5632 18.4 / 36.9, x 32000 x 2048 (128 columns, no split) 39.6 / 47.1;
//   several row tiles, if the K range is long enough (32 blocks) for at least four CTAs per tile: 256 x 2048 x 2048 16.4 / 19.5,
//   512 x 768 x 3072 18.4 / 24.6, 2048 x 64 x 2048 15.2 / 18.4; with two CTAs per tile (512 x 2048 x 2048) both take 20.4, and
//   256 x 3072 x 768 (12 blocks) 16.4 / 14.3, warm 2089 x 128 x 1584 (25 blocks in eight parts) 13.8 / 11.9;
//   a column count that is no multiple of 32, whose last tiles the persistent kernel stores element by element: weight
//   gradient 512 x 784 x 256 14.5 / 47.1.  With one CTA per tile its longer loop over 64 columns has to be short (warm: 2811 x 808 x 784
//   15.6 / 25.7, but 6635 x 200 x 1064 19.5 / 18.8, 7321 x 136 x 1976 28.0 / 23.6), or the sum is added to the output, which costs the other
//   kernel a read per element too (1248 x 1272 over 2936 rows 32.8 / 46.7, 1672 x 968 over 4840 rows 55.6 / 46.0).
bool gemm_few_plan(const cgk_gemm_args& a, int ctas, FewPlan* p) {
  if (a.rope_cos || a.split_k > 1) return false;
  const long long tm = (long long)a.batch * ((a.M + BM - 1) / BM), slots = a.max_ctas > 0 ? ctas : 2LL * ctas;
  const int kb = (a.K + BK - 1) / BK;
  auto tiles = [&](int bn) { return tm * ((a.N + bn - 1) / bn); };
  auto split = [&](long long t) { int s = 1; while (s < 8 && t * s * 2 <= slots && kb >= 4 * s) s *= 2; return s; };
  if (a.M <= BM) {
    p->bn = tiles(64) * 2 <= slots ? 64 : 128;
    p->split = split(tiles(p->bn));
    return tiles(p->bn) <= slots;
  }
  p->bn = 64;
  p->split = split(tiles(64));
  if (a.N % 32 != 0 && a.N % 4 == 0 && a.N > 32)
    return tiles(64) * p->split <= slots && (p->split > 1 || kb <= 16 || (a.accumulate && kb <= 64));
  return kb >= 32 && p->split >= 4 && tiles(64) * p->split <= slots;
}

int launch_gemm_few(const cgk_gemm_args& a, const GemmDev& g, const FewPlan& p, cudaStream_t stream) {
  return p.bn == 128 ? launch<128>(a, g, p.split, stream) : launch<64>(a, g, p.split, stream);
}

}  // namespace cgk

CGK_BOUNDS_READER(gemm_few)
