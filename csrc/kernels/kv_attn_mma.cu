// Attention of few query rows over the paged INT4 KV cache (head_dim 128): decoding and the verify pass of speculative decoding.
//
// A kv head has R = Tq * (Hq / Hk) query rows, 4 for one new token and 20 for five with four query heads per kv head.  tcgen05 tiles
// of 128 keys (kv_attn_tc.cu) spent some 4 us per tile on writing the converted values to shared memory and on two hand-overs to the
// MMA-issuing thread; here every warp works through its own blocks of 32 keys with mma.sync, from the nibbles to its part of the
// result, and meets the others only at the end:
//   * S[rows, 8 keys] = Q . K^T: lane (g, q) holds the 32 elements 32 q .. 32 q + 31 of key g, 16 bytes of nibbles,
//     which are its fragments of eight MMAs; the elements' order in a word (0,4,1,5,2,6,3,7) is given to Q's fragments instead;
//   * O[rows, 128] += P . V: the sums of S are the A fragments of P; lane (g, q) holds elements 16 g .. 16 g + 15 of keys 2 q, 2 q + 1,
//     2 q + 8, 2 q + 9, and column g of the MMAs' eight columns j is element 16 g + j;
//   * raw rows come by cp.async into a ring of the warp, two blocks ahead; where the next 32 groups of 16 keys start is held one by
//     lane.  Scales come as one copy per key: with a copy per lane and scale the copies of a block (a tag per key and instruction)
//     took as long as its arithmetic (16 sequences, one token: 15.7 us).
// The parts (row maximum, sum, O) of the warps of a cluster of CTAs that share a (sequence, kv head) meet over distributed shared
// memory, in the order of the ranks and warps.
// Values are those of kv_attn_tc.cu: K and V as bf16(q * bf16(scale)), P rounded to bf16 before it is summed.
//
// 16 sequences of 640 tokens, 32 query and 8 kv heads, one new token: 10.4 us (29.2 by tcgen05 with combined splits); five: 15.8 (42.3).
// 13 MB of cache are 2 us at copy rate.  A round of a CTA's eight blocks takes 2.1 us for one row tile and 3.1 for two (conversion and
// MMAs of two warps per scheduler); the chain lengths -> page -> keys at the start and the merge are the rest.
// Long histories of few heads are shared by up to 16 CTAs, if that many clusters run at once.  One sequence of 32 000 tokens, 8 kv heads:
// 40.8 us (by four CTAs 70.8, tcgen05 with combined splits 66.4), five tokens 64.4 (110; 87.9); one kv head 25.4 (68.5; 35.8), five
// tokens 38.9 (106; 44.7).
#include <cuda_bf16.h>

#include <atomic>

#include "host_common.h"
#include "kv_dev.cuh"
#include "mma_sync.cuh"

namespace cgk {
namespace {

constexpr int KM_WARPS = 8, KM_THREADS = KM_WARPS * 32, KM_D = 128, KM_NK = 2, KM_KB = 16 * KM_NK, KM_STAGES = 3;
// a warp's 16 keys: K by lane, V rows of 64 bytes (80 apart: the lanes of a load in different banks), four scales per key of K and of V
constexpr int KM_V = 1024, KM_VLD = 80, KM_S = KM_V + 16 * KM_VLD, KM_GROUP = KM_S + 2 * 16 * 16, KM_STAGE = KM_NK * KM_GROUP;
constexpr int KM_LD = 8 * 20 + 4;                                     // row of a part: eight pieces of 16 elements, 20 apart: no two lanes of a store share banks

// MT: 16-row tiles of Q.  LP: parts that a lane weighs, so up to 4 * LP CTAs (with four parts a lane in every launch, the compiler kept
// values of the loop over two row tiles in local memory: 16 sequences, five tokens, 15.7 -> 16.6 us)
template <int MT, int LP>
struct KmSmem {
  static constexpr int MAX_CLUSTER = LP * 32 / KM_WARPS;
  static constexpr int ROWS = 16 * MT;
  static constexpr int RING = KM_WARPS * KM_STAGES * KM_STAGE;
  static constexpr int PART = ROWS * KM_LD * 4;                        // a warp's O
  static constexpr int O_BYTES = KM_WARPS * PART;                      // overlays the rings once the loop is over
  static constexpr int BODY = RING > O_BYTES ? RING : O_BYTES;
  static constexpr int OFF_ML = BODY;                                  // float [warp][2][ROWS]: maximum, sum
  static constexpr int OFF_W = OFF_ML + KM_WARPS * 2 * ROWS * 4;       // float [MAX_CLUSTER * KM_WARPS][ROWS]: weights of all parts
  static constexpr int OFF_Q = OFF_W + MAX_CLUSTER * KM_WARPS * ROWS * 4;
  static constexpr int TOTAL = OFF_Q + (MT > 1 ? MT * 8 * 512 : 0);    // Q fragments of more than one tile: [tile][MMA][lane] 16 bytes
};

// eight nibbles -> four pairs of bf16 (elements 0,4 1,5 2,6 3,7), times the group scale
__device__ __forceinline__ void km_convert(uint32_t w, __nv_bfloat162 s2, uint32_t mask, uint32_t magic, uint32_t (&o)[4]) {
  const uint32_t v = w ^ 0x88888888u, c136 = 0x43084308u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t x = pick(v >> (4 * j), mask, magic);                // 128 + (nibble ^ 8) in both halves
    const __nv_bfloat162 h = __hmul2(__hsub2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&c136)), s2);
    o[j] = *reinterpret_cast<const uint32_t*>(&h);
  }
}

template <int MT, int LP>
__global__ void __launch_bounds__(KM_THREADS, 1)
kv_attention_mma_kernel(KvDev c, const __nv_bfloat16* __restrict__ q, long long q_bs, long long q_ts, long long q_hs, int Tq, int Hq, float scale_log2,
                        __nv_bfloat16* __restrict__ out) {
  using S = KmSmem<MT, LP>;
  constexpr int ROWS = S::ROWS;
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, qq = lane & 3;
  const int splits = gridDim.x, rank = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  const int rep = Hq / c.heads, R = Tq * rep, G = KM_D / c.group;
  pdl_trigger();
  pdl_wait();
  const int len = c.lengths[b] + Tq;                                   // the Tq new tokens were appended before the call
  // Q rows of this warp's tile (all warps: the only tile; else one warp per tile): asked for before the chain of page and keys
  const bool loads_q = MT == 1 || warp < MT;
  uint4 qr[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = (MT == 1 ? 0 : warp * 16) + gq + 8 * h, t = r / rep;
    const __nv_bfloat16* p = q + b * q_bs + t * q_ts + (hk * rep + r - t * rep) * q_hs + qq * 32;
#pragma unroll
    for (int w = 0; w < 4; ++w) qr[h][w] = loads_q && r < R ? *reinterpret_cast<const uint4*>(p + w * 8) : make_uint4(0, 0, 0, 0);
  }
  const int blocks = (len + KM_KB - 1) / KM_KB, stride = splits * KM_WARPS;
  const int first = rank * KM_WARPS + warp;                            // this warp's blocks of keys: first, first + stride, ..
  const int mine = first < blocks ? (blocks - first + stride - 1) / stride : 0;
  const bool one_page = c.page_size % 16 == 0;                         // 16 keys never cross pages

  const uint32_t ring = smem_u32(smem) + warp * (KM_STAGES * KM_STAGE);
  auto token = [&](int key) {                                          // a key's place in the pool, in tokens
    const int lp = key / c.page_size;
    return c.page_table[CGK_IDX(b * c.max_pages + lp, c.batch * c.max_pages)] * c.page_size + key - lp * c.page_size;
  };
  const uint8_t* const k_src = c.k_pages + hk * (KM_D / 2) + qq * 16;
  const uint8_t* const v_src = c.v_pages + hk * (KM_D / 2) + qq * 16;
  const float* const s_src = (lane < 16 ? c.k_scales : c.v_scales) + hk * G;
  const int row_bytes = c.heads * (KM_D / 2), row_scales = c.heads * G;
  int held = 0;                                                        // lane l: where group (last multiple of 32) + l of 16 keys starts
  auto fetch = [&](int i) {
    if (i < mine) {
#pragma unroll
      for (int n = 0; n < KM_NK; ++n) {
        const int group = i * KM_NK + n, kb = (first + i * stride) * KM_KB + n * 16, left = len - kb;      // keys from here on
        if (one_page && (group & 31) == 0) {
          const int j = group + lane, key = (first + j / KM_NK * stride) * KM_KB + j % KM_NK * 16;
          held = key < len ? token(key) : 0;
        }
        const int base = __shfl_sync(0xffffffffu, held, group & 31);
        auto place = [&](int k) -> long long { return k >= left ? base : one_page ? base + k : token(kb + k); };   // beyond the end nothing is read
        const uint32_t dst = ring + (i % KM_STAGES) * KM_STAGE + n * KM_GROUP;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = gq + 8 * h;
          const long long t = place(k);
          cp_async_16_or_zero(dst + h * 512 + lane * 16, k_src + t * row_bytes, k < left ? 16 : 0);
          cp_async_16_or_zero(dst + KM_V + k * KM_VLD + qq * 16, v_src + t * row_bytes, k < left ? 16 : 0);
        }
        const int k = lane & 15;                                       // lanes 0-15: the scales of K, 16-31: of V
        const float* src = s_src + place(k) * row_scales;
        if (G == 4) cp_async_16_or_zero(dst + KM_S + lane * 16, src, k < left ? 16 : 0);
        else if (G == 2) cp_async_or_zero<8>(dst + KM_S + lane * 16, src, k < left ? 8 : 0);
        else cp_async_or_zero<4>(dst + KM_S + lane * 16, src, k < left ? 4 : 0);
      }
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int i = 0; i < KM_STAGES - 1; ++i) fetch(i);

  // Fragment registers 0 / 2 (row g) and 1 / 3 (row g + 8) of MMAs 2 w and 2 w + 1 are elements 32 q + 8 w ..
  uint32_t qf[MT == 1 ? 8 : 1][4];
  uint4* const q_s = reinterpret_cast<uint4*>(smem + S::OFF_Q);
  if (loads_q) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      uint32_t p[2][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 v = qr[h][w];
        p[h][0] = __byte_perm(v.x, v.z, 0x5410); p[h][1] = __byte_perm(v.x, v.z, 0x7632);
        p[h][2] = __byte_perm(v.y, v.w, 0x5410); p[h][3] = __byte_perm(v.y, v.w, 0x7632);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if constexpr (MT == 1) {
          qf[2 * w + s][0] = p[0][2 * s]; qf[2 * w + s][1] = p[1][2 * s]; qf[2 * w + s][2] = p[0][2 * s + 1]; qf[2 * w + s][3] = p[1][2 * s + 1];
        } else {
          q_s[(warp * 8 + 2 * w + s) * 32 + lane] = make_uint4(p[0][2 * s], p[1][2 * s], p[0][2 * s + 1], p[1][2 * s + 1]);
        }
      }
    }
  }
  if (MT > 1) __syncthreads();

  float o[MT][16][4], m[MT][2], l[MT][2];
  int last[MT][2];                                                     // the last key that a row sees
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      m[mt][h] = -INFINITY;
      l[mt][h] = 0.0f;
      last[mt][h] = len - Tq + min((mt * 16 + gq + 8 * h) / rep, Tq - 1);      // causal among the new tokens
    }
#pragma unroll
    for (int j = 0; j < 16; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[mt][j][e] = 0.0f;
  }
  const int k_group = qq * 32 / c.group, v_group = gq * 16 / c.group;
  uint32_t mask = 0x000F000Fu, magic = 0x43004300u;
  asm volatile("" : "+r"(mask), "+r"(magic));

  for (int i = 0; i < mine; ++i) {
    cp_async_wait<KM_STAGES - 2>();
    __syncwarp();
    fetch(i + KM_STAGES - 1);
    const uint8_t* src = smem + warp * (KM_STAGES * KM_STAGE) + (i % KM_STAGES) * KM_STAGE;
    const int kb = (first + i * stride) * KM_KB;
    float s[MT][2 * KM_NK][4];
#pragma unroll
    for (int h = 0; h < 2 * KM_NK; ++h) {                              // keys 8 h + g: the columns of an MMA
      float odd[MT][4];                                                // two chains of four MMAs instead of one of eight
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[mt][h][e] = odd[mt][e] = 0.0f;
      const uint8_t* group = src + h / 2 * KM_GROUP;
      const uint4 raw = *reinterpret_cast<const uint4*>(group + h % 2 * 512 + lane * 16);
      const __nv_bfloat162 s2 = __float2bfloat162_rn(*reinterpret_cast<const float*>(group + KM_S + (h % 2 * 8 + gq) * 16 + k_group * 4));
      const uint32_t w4[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        uint32_t k[4];
        km_convert(w4[w], s2, mask, magic, k);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if constexpr (MT == 1) {
              mma_bf16(t ? odd[0] : s[0][h], qf[2 * w + t][0], qf[2 * w + t][1], qf[2 * w + t][2], qf[2 * w + t][3], k[2 * t], k[2 * t + 1]);
            } else {
              const uint4 a = q_s[(mt * 8 + 2 * w + t) * 32 + lane];
              mma_bf16(t ? odd[mt] : s[mt][h], a.x, a.y, a.z, a.w, k[2 * t], k[2 * t + 1]);
            }
          }
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[mt][h][e] += odd[mt][e];
    }
    uint32_t p[MT][KM_NK][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {                                    // rows g and g + 8; values 2 h, 2 h + 1 of all tiles
        float x[4 * KM_NK], mx = -INFINITY;
#pragma unroll
        for (int e = 0; e < 4 * KM_NK; ++e) {
          const int key = kb + (e >> 1) * 8 + 2 * qq + (e & 1);
          x[e] = key <= last[mt][h] ? s[mt][e >> 1][2 * h + (e & 1)] * scale_log2 : -INFINITY;
          mx = fmaxf(mx, x[e]);
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mo = m[mt][h], mn = fmaxf(mo, mx);
        if (__any_sync(0xffffffffu, mn > mo)) {
          const float corr = mo > -INFINITY ? fast_exp2(mo - mn) : 1.0f;       // nothing summed yet: nothing to rescale
          l[mt][h] *= corr;
          m[mt][h] = mn;
#pragma unroll
          for (int j = 0; j < 16; ++j) { o[mt][j][2 * h] *= corr; o[mt][j][2 * h + 1] *= corr; }
        }
#pragma unroll
        for (int n = 0; n < KM_NK; ++n) {
          float e4[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) e4[e] = x[4 * n + e] > -INFINITY ? fast_exp2(x[4 * n + e] - mn) : 0.0f;
          const uint32_t lo = pack_bf16x2(e4[0], e4[1]), hi = pack_bf16x2(e4[2], e4[3]);
          const float2 a = unpack_bf16x2(lo), d = unpack_bf16x2(hi);
          l[mt][h] += (a.x + a.y) + (d.x + d.y);
          p[mt][n][h] = lo;                                            // A registers 0 / 1: keys 2 q, 2 q + 1
          p[mt][n][2 + h] = hi;                                        // 2 / 3: eight more
        }
      }
    }
    // V: two words (elements 16 g .. 16 g + 7, 8 more) of each of four keys
#pragma unroll
    for (int n = 0; n < KM_NK; ++n) {
      const uint8_t* group = src + n * KM_GROUP;
      uint2 raw[4];
      __nv_bfloat162 s2[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int k = 2 * qq + (h & 1) + 8 * (h >> 1);
        raw[h] = *reinterpret_cast<const uint2*>(group + KM_V + k * KM_VLD + gq * 8);
        s2[h] = __float2bfloat162_rn(*reinterpret_cast<const float*>(group + KM_S + 256 + k * 16 + v_group * 4));
      }
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        uint32_t v[4][4];
#pragma unroll
        for (int h = 0; h < 4; ++h) km_convert(w ? raw[h].y : raw[h].x, s2[h], mask, magic, v[h]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {                                  // elements 8 w + j (low halves) and 8 w + 4 + j (high halves)
          const uint32_t b0 = __byte_perm(v[0][j], v[1][j], 0x5410), b1 = __byte_perm(v[2][j], v[3][j], 0x5410);
          const uint32_t c0 = __byte_perm(v[0][j], v[1][j], 0x7632), c1 = __byte_perm(v[2][j], v[3][j], 0x7632);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            mma_bf16(o[mt][8 * w + j], p[mt][n][0], p[mt][n][1], p[mt][n][2], p[mt][n][3], b0, b1);
            mma_bf16(o[mt][8 * w + 4 + j], p[mt][n][0], p[mt][n][1], p[mt][n][2], p[mt][n][3], c0, c1);
          }
        }
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();                                                     // the rings make room for the parts
  // sum j's columns 2 q and 2 q + 1 are elements 16 (2 q) + j and 16 (2 q + 1) + j
  float* const part = reinterpret_cast<float*>(smem) + warp * (S::PART / 4);
  float* const ml = reinterpret_cast<float*>(smem + S::OFF_ML);
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = mt * 16 + gq + 8 * h;
      float sum = l[mt][h];
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      if (qq == 0) { ml[warp * 2 * ROWS + r] = m[mt][h]; ml[warp * 2 * ROWS + ROWS + r] = sum; }
#pragma unroll
      for (int col = 0; col < 2; ++col)
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4*>(part + r * KM_LD + 20 * (2 * qq + col) + j) =
              make_float4(o[mt][j][2 * h + col], o[mt][j + 1][2 * h + col], o[mt][j + 2][2 * h + col], o[mt][j + 3][2 * h + col]);
    }
  if (splits > 1) cluster_sync_all();
  else __syncthreads();
  // every CTA writes its share of the rows: weights 2^(m_part - m) / sum of all parts, then the weighted sum; part p is that of warp
  // p % KM_WARPS of CTA p / KM_WARPS, which began with block p: those beyond the last block are empty
  const int parts = LP == 1 ? splits * KM_WARPS : min(splits * KM_WARPS, (len + KM_KB - 1) / KM_KB), r0 = min(R, ROWS) * rank / splits, r1 = min(R, ROWS) * (rank + 1) / splits;
  float* const wts = reinterpret_cast<float*>(smem + S::OFF_W);
  auto at = [&](uint32_t addr, int p) { return splits > 1 ? cluster_map(addr, p / KM_WARPS) : addr; };
  for (int r = r0 + warp; r < r1; r += KM_WARPS) {
    float pm[LP], pl[LP], top = -INFINITY, total = 0.0f;
#pragma unroll
    for (int i = 0; i < LP; ++i) {
      const int p = lane + 32 * i;
      pm[i] = -INFINITY;
      pl[i] = 0.0f;
      if (p < parts) {
        const float* src = ml + p % KM_WARPS * 2 * ROWS + r;
        const uint32_t a = at(smem_u32(src), p);
        pm[i] = splits > 1 ? ld_cluster_f1(a) : src[0];
        pl[i] = splits > 1 ? ld_cluster_f1(a + ROWS * 4) : src[ROWS];
      }
      top = fmaxf(top, pm[i]);
    }
    top = warp_max(top);
#pragma unroll
    for (int i = 0; i < LP; ++i) {
      pm[i] = pm[i] > -INFINITY ? fast_exp2(pm[i] - top) : 0.0f;
      total += pm[i] * pl[i];
    }
    total = warp_sum(total);
#pragma unroll
    for (int i = 0; i < LP; ++i)
      if (lane + 32 * i < parts) wts[(lane + 32 * i) * ROWS + r] = total > 0.0f ? pm[i] / total : 0.0f;
    __syncwarp();
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int p = 0; p < parts; ++p) {
      const float* src = reinterpret_cast<const float*>(smem) + p % KM_WARPS * (S::PART / 4) + r * KM_LD + (lane >> 2) * 20 + (lane & 3) * 4;
      const float4 v = splits > 1 ? ld_cluster_f4(at(smem_u32(src), p)) : *reinterpret_cast<const float4*>(src);
      const float wp = wts[p * ROWS + r];
      acc.x += wp * v.x; acc.y += wp * v.y; acc.z += wp * v.z; acc.w += wp * v.w;
    }
    const int t = r / rep, h = hk * rep + r % rep;
    *reinterpret_cast<uint2*>(out + (((long long)b * Tq + t) * Hq + h) * KM_D + lane * 4) = make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
  }
  if (splits > 1) cluster_sync_all();                                  // nobody leaves while its parts are read
}

// The clusters of S CTAs that a device runs at once, 0 if none (asked for once; concurrent callers would store the same value).
template <int MT, int LP>
cudaError_t clusters_at_once(int S, int* fit) {
  static std::atomic<int> known[64][KmSmem<MT, LP>::MAX_CLUSTER + 1];
  int dev = 0;
  if (cudaError_t e = cudaGetDevice(&dev)) return e;
  if (dev < 64 && known[dev][S].load(std::memory_order_relaxed)) {
    *fit = known[dev][S].load(std::memory_order_relaxed) - 1;
    return cudaSuccess;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)S);
  cfg.blockDim = dim3(KM_THREADS);
  cfg.dynamicSmemBytes = KmSmem<MT, LP>::TOTAL;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(fit, kv_attention_mma_kernel<MT, LP>, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    *fit = 0;
  }
  if (dev < 64) known[dev][S].store(*fit + 1, std::memory_order_relaxed);
  return cudaSuccess;
}

template <int MT, int LP>
cudaError_t launch_cluster(const KvDev& c, const __nv_bfloat16* q, long long bs, long long ts, long long hs, int Tq, int Hq, float scale, int s, __nv_bfloat16* out,
                           cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(kv_attention_mma_kernel<MT, LP>, cudaFuncAttributeMaxDynamicSharedMemorySize, KmSmem<MT, LP>::TOTAL);
  if (e != cudaSuccess) return e;
  return launch_overlapped(kv_attention_mma_kernel<MT, LP>, dim3(s, c.heads, c.batch), dim3(KM_THREADS), KmSmem<MT, LP>::TOTAL, stream, s > 1 ? s : 0,
                           c, q, bs, ts, hs, Tq, Hq, scale * 1.44269504089f, out);
}

template <int MT>
cudaError_t launch_mt(const KvDev& c, const __nv_bfloat16* q, long long bs, long long ts, long long hs, int Tq, int Hq, float scale, int splits, __nv_bfloat16* out,
                      cudaStream_t stream) {
  constexpr int FEW = KmSmem<MT, 1>::MAX_CLUSTER, MANY = KmSmem<MT, 4>::MAX_CLUSTER;
  if (splits > FEW) {
    cudaError_t e = cudaFuncSetAttribute(kv_attention_mma_kernel<MT, 4>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kv_attention_mma_kernel<MT, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, KmSmem<MT, 4>::TOTAL);
    if (e != cudaSuccess) return e;
    // as many as run at once in clusters: a cluster lies in one GPC, whose SMs it may not fill
    for (int s = splits < MANY ? splits : MANY; s > FEW; s = s > 8 ? 8 : FEW) {
      int fit = 0;
      if ((e = clusters_at_once<MT, 4>(s, &fit)) != cudaSuccess) return e;
      if (fit >= (long long)c.heads * c.batch) return launch_cluster<MT, 4>(c, q, bs, ts, hs, Tq, Hq, scale, s, out, stream);
    }
  }
  return launch_cluster<MT, 1>(c, q, bs, ts, hs, Tq, Hq, scale, splits < FEW ? splits : FEW, out, stream);
}
}  // namespace

// R = Tq * (Hq / heads) <= 32.  splits: CTAs per (sequence, kv head), at most 16 are used.
cudaError_t launch_kv_attention_mma(const KvDev& c, const __nv_bfloat16* q, long long bs, long long ts, long long hs, int Tq, int Hq, float scale, int splits,
                                    __nv_bfloat16* out, cudaStream_t stream) {
  if (Tq * (Hq / c.heads) <= 16) return launch_mt<1>(c, q, bs, ts, hs, Tq, Hq, scale, splits, out, stream);
  return launch_mt<2>(c, q, bs, ts, hs, Tq, Hq, scale, splits, out, stream);
}
}  // namespace cgk

CGK_BOUNDS_READER(kv_attn_mma)
