// What the kernels that reorder reference-format INT4 weights (once per weight) share.  A thread takes 32 words of eight nibbles
// from rows N / 2 bytes apart, all on their way at once, transposes them eight by eight in registers and writes 16 bytes at a time.
#pragma once
#include <cstdint>

namespace cgk {

// word g of the result holds nibble g of every word, word e's at nibble e
__device__ __forceinline__ void transpose_nibbles(uint32_t (&w)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {                                        // 16 bits between words i and i + 4
    const uint32_t a = w[i], b = w[i + 4];
    w[i] = __byte_perm(a, b, 0x5410);
    w[i + 4] = __byte_perm(a, b, 0x7632);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {                                        // bytes between words i and i + 2
    const int i = (j >> 1) * 4 + (j & 1);
    const uint32_t a = w[i], b = w[i + 2];
    w[i] = __byte_perm(a, b, 0x6240);
    w[i + 2] = __byte_perm(a, b, 0x7351);
  }
#pragma unroll
  for (int i = 0; i < 8; i += 2) {                                     // nibbles between neighbours
    const uint32_t a = w[i], b = w[i + 1];
    w[i] = (a & 0x0F0F0F0Fu) | ((b & 0x0F0F0F0Fu) << 4);
    w[i + 1] = ((a >> 4) & 0x0F0F0F0Fu) | (b & 0xF0F0F0F0u);
  }
}

// eight nibbles from any byte boundary
__device__ __forceinline__ uint32_t load_nibbles(const uint8_t* p, bool word) {
  return word ? *reinterpret_cast<const uint32_t*>(p) : p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24;
}

}  // namespace cgk
