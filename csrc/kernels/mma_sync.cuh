// Warp-level tensor-core and copy primitives for kernels whose rows are too few for tcgen05 (decoding): operands come from
// registers, so nothing is handed from one thread to another.  An mma.sync of 16 x 8 x 16 takes 8 to 9 cycles of a scheduler's tensor
// pipe on sm_100a: 540 TFLOP/s, about a third of what tcgen05 reaches.
// Fragments of m16n8k16, lane l, g = l / 4, q = l % 4: A rows g and g + 8 (registers 0 / 2 and 1 / 3), k 2 q, 2 q + 1 (0, 1) and
// 8 more (2, 3); B the same k of column g; sums of rows g (0, 1) and g + 8 (2, 3), columns 2 q and 2 q + 1.
#pragma once
#include "sm100.cuh"

namespace cgk {

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// (v & mask) | magic in one instruction: only one of two constants fits into it, so both come from registers
__device__ __forceinline__ uint32_t pick(uint32_t v, uint32_t mask, uint32_t magic) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(v), "r"(mask), "r"(magic));
  return r;
}

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void* src, uint32_t bytes) {     // bytes: 16, or 0 for zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
template <int BYTES>                                                                                      // 4 or 8
__device__ __forceinline__ void cp_async_or_zero(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

}  // namespace cgk
