// Dequantisation of Q4_0 / Q8_0 payload words to exact fp16 in registers, for the prefill GEMMs.
#pragma once
#include "greta_common.cuh"

namespace {

// ---- dequant to exact fp16 -----------------------------------------------------------------
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
  __half2 r = __hsub2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
  return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
  __half2 r = __hfma2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b), *reinterpret_cast<__half2 *>(&c));
  return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
  __half2 r = __hmul2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
  return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t lop_and_or(uint32_t a, uint32_t m, uint32_t o) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(m), "r"(o));
  return r;
}
// One Q4_0 payload word -> 4 low-nibble elements (lo[0..1]) and 4 high-nibble elements (hi[0..1]) as half2,
// each half = round_to_half((q - 8) * d): the product of two halves rounded once, the same value as
// __float2half((float)(q - 8) * (float)d).
__device__ __forceinline__ void dq4_word(uint32_t w, uint32_t d2, uint32_t (&lo)[2], uint32_t (&hi)[2]) {
  const uint32_t MAGIC = 0x64006400u, C1032 = 0x64086408u, SIXTEENTH = 0x2C002C00u, CM72 = 0xD480D480u;
  uint32_t w8 = w >> 8;
  uint32_t a = h2mul(h2sub(lop_and_or(w, 0x000F000Fu, MAGIC), C1032), d2);            // e0, e2
  uint32_t b = h2mul(h2sub(lop_and_or(w8, 0x000F000Fu, MAGIC), C1032), d2);           // e1, e3
  uint32_t c = h2mul(h2fma(lop_and_or(w, 0x00F000F0u, MAGIC), SIXTEENTH, CM72), d2);  // E0, E2
  uint32_t e = h2mul(h2fma(lop_and_or(w8, 0x00F000F0u, MAGIC), SIXTEENTH, CM72), d2); // E1, E3
  lo[0] = __byte_perm(a, b, 0x5410);
  lo[1] = __byte_perm(a, b, 0x7632);
  hi[0] = __byte_perm(c, e, 0x5410);
  hi[1] = __byte_perm(c, e, 0x7632);
}
// One Q8_0 payload word (4 int8) -> 4 elements as two half2.
__device__ __forceinline__ void dq8_word(uint32_t w, uint32_t d2, uint32_t (&o)[2]) {
  const uint32_t C1152 = 0x64806480u;
  uint32_t t = w ^ 0x80808080u;
  o[0] = h2mul(h2sub(__byte_perm(t, 0x64646464u, 0x5140), C1152), d2);
  o[1] = h2mul(h2sub(__byte_perm(t, 0x64646464u, 0x7362), C1152), d2);
}

}  // namespace
