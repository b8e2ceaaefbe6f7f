// iq1m.cuh - IQ1_M weights (include/basalt/ggml/ggml_common.h:350-362) in packed fp16, exactly, for the kernels that multiply on fp16
// tensor cores.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

namespace bsx {

__device__ __forceinline__ uint32_t iq1m_add2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t iq1m_mul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// A weight is d m (g + delta), g = c - 1 with c the codebook's 2-bit code, m = 2 s + 1 <= 15, delta = +-1/8.  8 m (g + delta) is an
// integer of at most 135 and exact in fp16 at every step.
// A code becomes its value by masking it where it lies in the codebook word and or-ing in an exponent that makes its place worth
// one: bits 4-5 under 2^6, 6-7 under 2^4, 8-9 under 2^2 (the constants -(2^E + 1) +- 1/8 stay within fp16's 11 bits only there), so
// two shifts bring all eight pairs into place and a pair costs one logic and two fp16x2 operations.
// q16: the two index bytes of 16 values; h8: their high bits and delta signs; s3: the scale field.
// out[i] = 8 w / d of values i (low half) and i + 8 (high half).
__device__ __forceinline__ void iq1m_units_16(uint32_t q16, uint32_t h8, uint32_t s3, const uint16_t* grid, uint32_t (&out)[8]) {
    const uint32_t ia = (q16 & 0xFFu) | ((h8 & 7u) << 8), ib = (q16 >> 8) | ((h8 & 0x70u) << 4);
    const uint32_t x = (uint32_t) grid[ia] | ((uint32_t) grid[ib] << 16);
    const uint32_t delta = 0x30003000u | ((h8 & 8u) << 12) | ((h8 & 0x80u) << 24);       // +-0.125 each
    const uint32_t k2 = iq1m_add2(delta, 0xC500C500u), k4 = iq1m_add2(delta, 0xCC40CC40u), k6 = iq1m_add2(delta, 0xD410D410u);   // -5, -17, -65
    const uint32_t m8 = iq1m_add2((0x6408u | (s3 << 4)) * 0x10001u, 0xE400E400u);       // 1024 + 16 s + 8 - 1024
    const uint32_t y = x << 4, z = x >> 6;
    const uint32_t v[8] = {iq1m_add2((y & 0x00300030u) | 0x54005400u, k6), iq1m_add2((y & 0x00C000C0u) | 0x4C004C00u, k4),
                           iq1m_add2((x & 0x00300030u) | 0x54005400u, k6), iq1m_add2((x & 0x00C000C0u) | 0x4C004C00u, k4),
                           iq1m_add2((x & 0x03000300u) | 0x44004400u, k2), iq1m_add2((z & 0x00300030u) | 0x54005400u, k6),
                           iq1m_add2((z & 0x00C000C0u) | 0x4C004C00u, k4), iq1m_add2((z & 0x03000300u) | 0x44004400u, k2)};
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = iq1m_mul2(v[i], m8);
}
// the block's fp16 super-scale d, from the top nibbles of its four scale words
__device__ __forceinline__ uint32_t iq1m_d_bits(uint2 sc) {
    return ((sc.x >> 12) & 0x000Fu) | ((sc.x >> 24) & 0x00F0u) | ((sc.y >> 4) & 0x0F00u) | ((sc.y >> 16) & 0xF000u);
}

}  // namespace bsx
