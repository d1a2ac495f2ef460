// sm_100's packed F32 arithmetic: two operations in one instruction, element by element the same IEEE operation as the
// scalar one, so the same bits; and small integers made F32 without a conversion instruction.
#pragma once
#include "common.cuh"

namespace osmos {

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack2u(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// An integer n < 1024 in the low bits of a half IS the subnormal F16 n 2^-24, and F16 to F32 is exact: codes masked in place, two
// to a word, reach F32 (times 2^-24, which a scale taken 2^24 times larger gives back) without a byte permute each, and the
// conversion runs beside the integer pipe.
__device__ __forceinline__ float low_half(uint32_t h) { return __half2float(__ushort_as_half((unsigned short) (h & 0xFFFFu))); }
__device__ __forceinline__ float high_half(uint32_t h) { return __half2float(__ushort_as_half((unsigned short) (h >> 16))); }

// byte J of `bytes` (n < 256) as the F32 32768 + n: bits 8 .. 15 of 0x47000000, one byte permute
template <int J> __device__ __forceinline__ uint32_t biased_byte(uint32_t bytes) { return __byte_perm(bytes, 0x47000000u, 0x7404 | (J << 4)); }
// a byte of a word as F32, exactly
template <int J> __device__ __forceinline__ float byte_value(uint32_t w) { return __fadd_rn(__uint_as_float(biased_byte<J>(w)), -32768.0f); }
// the codes of two chunks (a, b: eight bytes each, 0 .. 255) as eight pairs of the F32 n + minus, exact
__device__ __forceinline__ void code_pairs(uint2 a, uint2 b, float minus, uint64_t* v) {
  const uint64_t m = pack2(minus, minus);
  v[0] = add2(pack2u(biased_byte<0>(a.x), biased_byte<0>(b.x)), m), v[1] = add2(pack2u(biased_byte<1>(a.x), biased_byte<1>(b.x)), m);
  v[2] = add2(pack2u(biased_byte<2>(a.x), biased_byte<2>(b.x)), m), v[3] = add2(pack2u(biased_byte<3>(a.x), biased_byte<3>(b.x)), m);
  v[4] = add2(pack2u(biased_byte<0>(a.y), biased_byte<0>(b.y)), m), v[5] = add2(pack2u(biased_byte<1>(a.y), biased_byte<1>(b.y)), m);
  v[6] = add2(pack2u(biased_byte<2>(a.y), biased_byte<2>(b.y)), m), v[7] = add2(pack2u(biased_byte<3>(a.y), biased_byte<3>(b.y)), m);
}

// the 6-bit (scale, minimum) pairs of two neighbouring groups out of Q4_K's and Q5_K's twelve bytes (words b, c, d of the
// block): s, the bit at which the first one's byte lies in each word - 0 or 16; upper: groups 4 .. 7. Two bytes each.
__device__ __forceinline__ void k_scales(uint32_t b, uint32_t c, uint32_t d, uint32_t s, bool upper, uint32_t& sc, uint32_t& mn) {
  const uint32_t w0 = b >> s, w1 = c >> s, w2 = d >> s;
  sc = upper ? (w2 & 0x0F0Fu) | ((w0 >> 2) & 0x3030u) : w0 & 0x3F3Fu;
  mn = upper ? ((w2 >> 4) & 0x0F0Fu) | ((w1 >> 2) & 0x3030u) : w1 & 0x3F3Fu;
}

}  // namespace osmos
