// Eight 4-bit codes of a word -> four bf16 pairs in memory order (shared by the two 4-bit products).  A 32-bit word holds its
// codes in the order (c0 c2 c4 c6 | c1 c3 c5 c7) per 16-bit half.
#pragma once

#include "common.cuh"

namespace mfq {

// A group's (scale, -offset) as bf16 pairs (scale, scale), (-offset, -offset).
__device__ __forceinline__ void w4_params(uint32_t g, uint32_t& s2, uint32_t& b2) {
  asm("prmt.b32 %0, %1, %1, 0x1010;" : "=r"(s2) : "r"(g));
  asm("prmt.b32 %0, %1, %1, 0x3232;" : "=r"(b2) : "r"(g));
}

// KIND 0: affine codes (NINT):  w = s * c - b.   KIND 1: MXFP4:  w = e2m1(c) * 2^(e - 127).
template <int KIND>
__device__ __forceinline__ void w4_decode(uint32_t word, uint32_t s2, uint32_t b2, uint32_t (&o)[4]) {
  if constexpr (KIND == 0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t pair = ((word >> (4 * j)) & 0x000F000Fu) | 0x43004300u;  // bf16 (128 + c, 128 + c')
      uint32_t qf;  // (c, c') exactly: integers below 256 are exact in bf16, so is the subtraction
      asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(qf) : "r"(pair), "r"(0x43004300u));
      asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(o[j]) : "r"(qf), "r"(s2), "r"(b2));  // s * c - b, one rounding
    }
  } else {
    // E2M1 magnitudes {0, .5, 1, 1.5, 2, 3, 4, 6} as bf16 = high bytes {00,3F,3F,3F,40,40,40,40}, low bytes
    // {00,00,80,C0,00,40,80,C0}: byte-permute instructions look four codes up at once (selector = code & 7)
    const uint32_t idx = word & 0x77777777u;
    uint32_t hiA, hiB, loA, loB;  // A: nibbles 0..3 (even columns), B: nibbles 4..7 (odd columns)
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(hiA) : "r"(0x3F3F3F00u), "r"(0x40404040u), "r"(idx & 0xFFFFu));
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(hiB) : "r"(0x3F3F3F00u), "r"(0x40404040u), "r"(idx >> 16));
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(loA) : "r"(0xC0800000u), "r"(0xC0804000u), "r"(idx & 0xFFFFu));
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(loB) : "r"(0xC0800000u), "r"(0xC0804000u), "r"(idx >> 16));
    uint32_t a01, a23, b01, b23;  // (bf16 n0, bf16 n1), (n2, n3), (n4, n5), (n6, n7)
    asm("prmt.b32 %0, %1, %2, 0x5140;" : "=r"(a01) : "r"(loA), "r"(hiA));
    asm("prmt.b32 %0, %1, %2, 0x7362;" : "=r"(a23) : "r"(loA), "r"(hiA));
    asm("prmt.b32 %0, %1, %2, 0x5140;" : "=r"(b01) : "r"(loB), "r"(hiB));
    asm("prmt.b32 %0, %1, %2, 0x7362;" : "=r"(b23) : "r"(loB), "r"(hiB));
    uint32_t mag[4];  // word j = (column 2j, column 2j+1) = (nibble j, nibble j + 4)
    asm("prmt.b32 %0, %1, %2, 0x5410;" : "=r"(mag[0]) : "r"(a01), "r"(b01));
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(mag[1]) : "r"(a01), "r"(b01));
    asm("prmt.b32 %0, %1, %2, 0x5410;" : "=r"(mag[2]) : "r"(a23), "r"(b23));
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(mag[3]) : "r"(a23), "r"(b23));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t sign = ((word >> (4 * j)) & 0x00080008u) << 12;  // code bit 3 -> bf16 sign bit
      asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(o[j]) : "r"(mag[j] | sign), "r"(s2));  // exact: s2 is a power of two
    }
  }
}

}  // namespace mfq
