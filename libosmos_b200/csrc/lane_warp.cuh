// What a lane kernel whose warps read a row with L lanes needs (lane_ring.cu): a lane's view of its
// sub-block of a superblock in shared memory, IQ3_XXS's sums without negated codes, and the IQ1 types' over a codebook of
// nibbles.
#pragma once
#include "lane_staged.cuh"

namespace osmos {
namespace lanes {

using namespace tma;
using staged::RepLuts2;

// a superblock's bytes through shared-memory loads at run-time offsets (2-byte aligned at best)
struct SmemReader {
  uint32_t b;
  __device__ __forceinline__ uint32_t u8(int o) const { return lds8(b + o); }
  __device__ __forceinline__ uint32_t u16(int o) const { return lds16(b + o); }
  __device__ __forceinline__ uint32_t u32(int o) const { return lds16(b + o) | lds16(b + o + 2) << 16; }
  __device__ __forceinline__ uint64_t u64(int o) const { return (uint64_t) u32(o) | (uint64_t) u32(o + 4) << 32; }
};

// What of a superblock a lane reads, worked out once: the lane's sub-block index j is the same for all its blocks,
// and so is its superblocks' alignment (a row is a multiple of 4 bytes, the lane's superblocks an even count apart)
struct LaneAt {
  uint32_t j;     // the sub-block
  uint32_t qoff;  // IQ3_XXS: the aligned word holding the sub-block's first grid index, from the superblock's start
  uint32_t sh;    // IQ3_XXS: 16 when that index lies mid-word (an aligned superblock), else 0
};

// sub-block at.j of the superblock at shared address sb
template <uint32_t T>
__device__ __forceinline__ void sub_codes(uint32_t sb, const LaneAt& at, LaneCodes& c, const RepLuts2<T>& lut) {
  if constexpr (T == QTYPE_IQ3_XXS) {
    // the 8 grid indices and the sign / scale word, each out of the aligned words around it: both lie 2 mod 4 bytes
    // into the superblock, so they start mid-word when the superblock is aligned and on a word when it is not
    const uint32_t sh = at.sh, al = sb + at.qoff;
    const uint32_t q0 = lds32(al), q1 = lds32(al + 4), q2 = lds32(al + 8);
    const uint32_t ala = al + 64u - 4u * at.j;
    const uint32_t aux = __funnelshift_r(lds32(ala), lds32(ala + 4), sh);
    const uint32_t w[2] = {__funnelshift_r(q0, q1, sh), __funnelshift_r(q1, q2, sh)};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t i0 = __byte_perm(w[k >> 1], 0, 0x4440 + 2 * (k & 1)), i1 = __byte_perm(w[k >> 1], 0, 0x4441 + 2 * (k & 1));
      const uint2 mm = lut.sign_masks2((aux >> (7 * k)) & 0x7F);
      c.w[2 * k] = negated4(lut.grid32(i0), mm.x, mm.x & kOnes), c.w[2 * k + 1] = negated4(lut.grid32(i1), mm.y, mm.y & kOnes);
    }
    c.s21[0] = c.s21[1] = 2 * (2 * (int) (aux >> 28) + 1);
    c.d = half_value(lds16(sb));
  } else {
    lane_codes_rd<T>(SmemReader{sb}, (int) at.j, c, lut);
  }
}

// IQ3_XXS's block sums without negating a code: the signed dot sum s_i g_i x_i is dp4a(g, x) - 2 dp4a(g & m, x) (m the
// byte mask of the negative values), so the mask costs one AND a word and a second dp4a a token instead of an XOR,
// an addition and a carry word - the integer pipe is the busier one here. Exact integers, the contract's products:
// the same bits as lane_block_sum.
template <int NTL, int NT, int NB>
__device__ __forceinline__ void iq3_block_sums(uint32_t sb, const LaneAt& at, const RepLuts2<QTYPE_IQ3_XXS>& lut,
                                               const int (&xq)[NT][NB][8], int k, float* out) {
  const uint32_t sh = at.sh, al = sb + at.qoff;
  const uint32_t q0 = lds32(al), q1 = lds32(al + 4), q2 = lds32(al + 8);
  const uint32_t ala = al + 64u - 4u * at.j;
  const uint32_t aux = __funnelshift_r(lds32(ala), lds32(ala + 4), sh);
  const uint32_t w[2] = {__funnelshift_r(q0, q1, sh), __funnelshift_r(q1, q2, sh)};
  int pos[NTL][2], neg[NTL][2];  // a half's dots: all values, and the negative ones
#pragma unroll
  for (int t = 0; t < NTL; t++) pos[t][0] = pos[t][1] = neg[t][0] = neg[t][1] = 0;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uint32_t i0 = __byte_perm(w[c >> 1], 0, 0x4440 + 2 * (c & 1)), i1 = __byte_perm(w[c >> 1], 0, 0x4441 + 2 * (c & 1));
    const uint2 mm = lut.sign_masks2((aux >> (7 * c)) & 0x7F);
    const int g0 = (int) lut.grid32(i0), g1 = (int) lut.grid32(i1);
    const int n0 = g0 & (int) mm.x, n1 = g1 & (int) mm.y;
#pragma unroll
    for (int t = 0; t < NTL; t++) {
      pos[t][c >> 1] = __dp4a(g1, xq[t][k][2 * c + 1], __dp4a(g0, xq[t][k][2 * c], pos[t][c >> 1]));
      neg[t][c >> 1] = __dp4a(n1, xq[t][k][2 * c + 1], __dp4a(n0, xq[t][k][2 * c], neg[t][c >> 1]));
    }
  }
  const int s21 = 2 * (2 * (int) (aux >> 28) + 1);
  const float d = half_value(lds16(sb));
#pragma unroll
  for (int t = 0; t < NTL; t++)
    out[t] = __fadd_rn(lane_part(d, s21, pos[t][0] - 2 * neg[t][0]), lane_part(d, s21, pos[t][1] - 2 * neg[t][1]));
}

// ---- IQ1_S, IQ1_M: the ternary codebook in shared memory as nibbles -------------------------------------------------
// An entry's eight values t (-1, 0, 1) as t + 1 in eight nibbles: byte b has value b low and value 4 + b high. One 4-byte
// word where the byte grid has eight: in eight copies (64 KB) a warp's 32 random lookups, four lanes a copy, meet about three
// deep in a bank, where two copies of 8-byte entries (32 KB) met six. Four copies take those 32 KB, for the row widths whose
// ring needs the room.
template <int COPIES> constexpr uint32_t kTernaryBytes = 2048u * COPIES * 4u;
template <uint32_t T> constexpr bool kTernary = (T == QTYPE_IQ1_S || T == QTYPE_IQ1_M);

// every thread of the block calls it; the table is complete at the block's next barrier
template <int COPIES> __device__ inline void build_ternary(uint8_t* smem, int threads) {
  constexpr int U = 4;
  for (int i0 = threadIdx.x; i0 < 2048; i0 += threads * U) {
    uint64_t g[U];
#pragma unroll
    for (int u = 0; u < U; u++) g[u] = i0 + u * threads < 2048 ? osmos_grid_iq1s[i0 + u * threads] : 0;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + u * threads < 2048) {
        const uint32_t w = __vadd4((uint32_t) g[u], kOnes) | __vadd4((uint32_t) (g[u] >> 32), kOnes) << 4;
        uint4* to = (uint4*) (smem + (uint32_t) (i0 + u * threads) * (COPIES * 4u));
#pragma unroll
        for (int c = 0; c < COPIES / 4; c++) to[c] = make_uint4(w, w, w, w);
      }
  }
}

// minus the sums of the four 8-value chunks of a block's int8 activations, two a word (each at most 8 x 127: 16 bits)
__device__ __forceinline__ void chunk_sums(const int (&x)[8], int (&out)[2]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int s0 = -__dp4a(0x01010101, x[4 * h + 1], __dp4a(0x01010101, x[4 * h], 0));
    const int s1 = -__dp4a(0x01010101, x[4 * h + 3], __dp4a(0x01010101, x[4 * h + 2], 0));
    out[h] = (int) __byte_perm((uint32_t) s0, (uint32_t) s1, 0x5410);
  }
}

// The block sums, bit for bit lane_block_sum's. A half's integer is S = sum over its two chunks of 8 (t . x) + delta (sum of
// x), delta +-1; with u = t + 1 that is 8 (u . x) - (8 - delta) (sum of x), formed doubled so that the high nibbles are
// multiplied where they lie: 2 S = 16 (u_low . x) + (16 u_high . x) - (14 or 18) (sum of x), the chunk sums worked out once
// a task (xc). The sum starts at 0x4B400000, so that it ends as the F32 12582912 + 2 S (|2 S| < 2^22): one subtraction
// instead of an integer conversion. Half of 2 S goes into the scale, (2 s + 1) / 16: d (2 s + 1) has 15 significant bits,
// so every product before the last is exact in any order and the last rounds the same number. (256 experts of 2048 x 7168
// IQ1_M, top-8 of 32 tokens, gate and up: 1.20 -> 0.88 ms; 102 thread-instructions a block and token at 72 % issue.)
template <uint32_t T, int COPIES, int NTL, int NT, int NB>
__device__ __forceinline__ void iq1_block_sums(uint32_t sb, const LaneAt& at, const uint8_t* table, uint32_t copy,
                                               const int (&xq)[NT][NB][8], const int (&xc)[NT][NB][2], int k, float* out) {
  const uint32_t j = at.j;
  uint32_t qs, qh, mult;
  float d, s[2];  // the superblock's scale; the halves' (2 s + 1) / 16 = (1 + s / 8) - 15 / 16
  if constexpr (T == QTYPE_IQ1_M) {
    // a 56-byte superblock starts on 8 bytes: four index bytes are one word, the four (index top, delta sign) nibbles one
    // half-word, the four scale words - their top nibbles the F16 scale, 3-bit scales below - one 8-byte read
    qs = lds32(sb + 4u * j), qh = lds16(sb + 32u + 2u * j);
    const uint2 sc = lds64(sb + 48u);
    const uint32_t tops = __byte_perm(sc.x, sc.y, 0x7531);
    const uint32_t d2 = ((tops >> 4) & 0x000F000Fu) | ((tops >> 8) & 0x00F000F0u);
    d = half_value(__byte_perm(d2, 0, 0x4420));
    const uint32_t fields = (j & 4u ? sc.y : sc.x) >> (16u * ((j >> 1) & 1u) + 6u * (j & 1u));
    s[0] = __uint_as_float(0x3F800000u | ((fields << 20) & 0x00700000u)), s[1] = __uint_as_float(0x3F800000u | ((fields << 17) & 0x00700000u));
    // a chunk's delta sign, bit 3 of its nibble, moved to bit 2 of byte c: 14, or 18 where it is set
    mult = (__byte_perm(qh >> 1, qh >> 5, 0x5140) & 0x04040404u) + 0x0E0E0E0Eu;
  } else {
    // a 50-byte superblock starts on a word or in its middle: the index bytes out of the two words around them
    const uint32_t al = sb + at.qoff - 4u * j;
    qs = __funnelshift_r(lds32(al), lds32(al + 4u), at.sh), qh = lds16(sb + 34u + 2u * j);
    d = half_value(lds16(sb));
    s[0] = s[1] = __uint_as_float(0x3F800000u | ((qh << 8) & 0x00700000u));
    mult = qh & 0x8000u ? 0x12121212u : 0x0E0E0E0Eu;
  }
  uint32_t w[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    constexpr int kTop = T == QTYPE_IQ1_M ? 4 : 3;  // bits a chunk has in qh
    constexpr int kSh = COPIES == 8 ? 5 : 4;  // (an entry's copies are 32 or 16 bytes)
    const uint32_t q = c == 0 ? qs << kSh : qs >> (8 * c - kSh), h = qh << (8 + kSh - kTop * c);
    w[c] = *(const uint32_t*) (table + ((h & (7u << (8 + kSh))) | ((q & (0xFFu << kSh)) | copy)));
  }
  int acc[NTL][2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int lo0 = (int) (w[2 * h] & kLow4), lo1 = (int) (w[2 * h + 1] & kLow4);
    const int hi0 = (int) (w[2 * h] & 0xF0F0F0F0u), hi1 = (int) (w[2 * h + 1] & 0xF0F0F0F0u);
#pragma unroll
    for (int t = 0; t < NTL; t++) {
      const int* x = xq[t][k] + 4 * h;
      int v = __dp4a(lo1, x[2], __dp4a(lo0, x[0], 0x04B40000)) << 4;
      v = __dp4a(hi1, x[3], __dp4a(hi0, x[1], v));
      acc[t][h] = h == 0 ? __dp2a_lo(xc[t][k][0], (int) mult, v) : __dp2a_hi(xc[t][k][1], (int) mult, v);
    }
  }
  const float p0 = mul_rn(d, __fadd_rn(s[0], -0.9375f)), p1 = mul_rn(d, __fadd_rn(s[1], -0.9375f));
#pragma unroll
  for (int t = 0; t < NTL; t++)
    out[t] = __fadd_rn(mul_rn(p0, __fadd_rn(__int_as_float(acc[t][0]), -12582912.0f)),
                       mul_rn(p1, __fadd_rn(__int_as_float(acc[t][1]), -12582912.0f)));
}

}  // namespace lanes
}  // namespace osmos
