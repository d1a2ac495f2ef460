// The prefill matrix products over f16 activations (include/osmos_b200/mm.h: mm_run, mm_run2, mm_group, mm_tokens)
// on the 5th-generation tensor cores: tcgen05.mma kind::f16, F32 accumulators in tensor memory.
//
// The weights' exact values are rounded to f16 (nearest) as they are decoded, the activations are the caller's x16
// (mm_x16's tiled f16), and every product is accumulated in F32 along K in one pass - the reference's arithmetic
// (kernels/mm.h: f16 operands, F32 accumulation) with the tensor core's own order of additions instead of its waves'
// partitions; a token's column is computed from that column alone, so its bits do not depend on the tokens beside
// it or on where in the batch it stands.
//
// The decoded weights are the products' operand in TENSOR MEMORY: a producer thread is a weight row, decodes 64 values
// of it and writes them to its own lane (tcgen05.st), so a decoded tile costs no shared-memory stores, no proxy fence and no
// operand reads from shared memory - which only the activations pass through.
//
// Blocks are persistent, one an SM; a tile is 128 weight rows x up to 256 tokens of one matrix. Tensor memory: two
// accumulators of 128 columns - a tile of up to 128 tokens takes one, so that its sums are stored while the next tile's
// products run; a larger tile takes both - and eight stages of 32 columns, 64 values of K each.
// Twenty-four warps, five roles that never meet in a tile:
//   epilogue (4 warps)   thread = one weight row (its TMEM lane): tcgen05.ld the sums, scale, store y[t][row] - or, for
//                        mm_run_silu, silu(scale sum) to y and as f16 into the next product's tiled activations; for
//                        mm_run_gated_mean the block's rows are hc streams' rows of the same dim values (row map
//                        below), each thread gates its sum, and the streams are added in order through shared memory
//   producers (16 warps, four teams of four on every fourth K step) decode the rows' bytes out of shared memory
//   issuer (1 warp)      a unit of one or two K steps: tcgen05.mma M128 N<=128 K16, eight a step (the even and the odd tokens; the
//                        first of a tile overwrite, the rest accumulate), then tcgen05.commit onto the unit's "empty" mbarrier; after
//                        a tile's last step a commit onto its accumulators' "full" ones. The whole warp runs this, one elected
//                        lane issues.
//   raw loaders (2 warps) the rows' bytes, 256 values of K at a time (128 of Q8_0, MXFP8 and Q5_1), a ring of three or four: one
//                        tensor-map copy where rows start on 16 bytes, else 16-byte cp.async pieces
//   token loader (1 warp) the tokens' x16, a K step a tensor-map copy; grouped tokens that start inside a tile of x16 by 16-byte
//                        cp.async pieces
// Bound by the decoders' integer and F32 pipes up to about 128 tokens a tile (a 64-value step of 128 Q4_K rows is 1,460 warp
// instructions, all roles together, of IQ3_XXS 2,260, at two thirds of the issue slots; its products are 128 cycles at 64 tokens), past
// that by the tokens' copies, 32 KB a step at 256 tokens where the products take 512 cycles (the tensor pipe is active 64 %). Measured,
// against decoded tiles in shared memory, a tile a block (with the tokens' rounding, passes of mm_tokens): Q4_K 4096 x 4096 at 777 /
// 2048 tokens 62.8 / 106 us -> 40.7 / 71; 128 MXFP4 experts of 1536 x 4096 over 2048 tokens, the layer, 1827 -> 769.
// Every mbarrier wait is bounded (%globaltimer) with one outcome a warp; a wait that runs out raises the status word, every
// role falls through to the common exit and tensor memory is released.
#include <cuda.h>

#include <cstring>

#include "act.cuh"
#include "decode.cuh"
#include "dispatch.cuh"
#include "fp4_tc_api.h"
#include "mm_tc_api.h"
#include "osmos_b200/mm.h"
#include "packed.cuh"
#include "tma.cuh"

namespace osmos {
namespace mm_tc {
namespace {

using namespace tma;

constexpr int kM = 128, kN = 128;  // rows a tile; tokens an accumulator
constexpr int kMaxAcc = 4;         // mm_col_tiles' largest class
constexpr int kEpiWarps = 4, kProdWarps = 16, kRawWarps = 2;
constexpr int kTeams = 4;          // producer teams: team t on the K steps t, t + 4, ...; its warp w has the rows 32 w .. 32 w + 31
constexpr int kFirstProd = kEpiWarps, kIssuerWarp = kFirstProd + kProdWarps, kFirstRaw = kIssuerWarp + 1, kTokenWarp = kFirstRaw + kRawWarps;
constexpr int kThreads = (kTokenWarp + 1) * kWarp;
static_assert(kFirstProd % 4 == 0 && kProdWarps == 4 * kTeams, "a producer warp's rows are its quarter of tensor memory (its index mod 4)");
constexpr int kStep = 64;                  // values of K a stage
constexpr int kSubs = kStep / 16;          // K = 16 products a stage
constexpr uint32_t kSteps = 8;             // stages of decoded weights
constexpr uint32_t kAccCols = 2 * kN;      // tensor memory: the accumulators' columns, then the stages', 32 each
constexpr uint32_t kStageCols = kStep / 2;
static_assert(kAccCols + kSteps * kStageCols == 512, "all of tensor memory");
constexpr uint32_t kMaxSpan = 2 * kN;      // tokens a tile
constexpr uint32_t kMaxMats = 768;        // matrices a launch: their first tiles are kept in shared memory

__device__ uint32_t g_status;
enum : uint32_t { kWaitRanOut = 1, kNotOfTensor = 2 };  // (mm_status's bits)

// shared-memory matrix descriptor of one K = 16 sub-tile of tokens: x16's fragments as they lie - a token's 16 values 32 bytes - as
// rows of 64 bytes, two tokens each, with the 64-byte swizzle; 8 rows are 512 bytes. A product takes the first 32 bytes of
// each row, the even tokens, or (the address 32 bytes on) the second, the odd ones: a copy of rows of 32 bytes under the
// 32-byte swizzle would be one product's operand, but moves 30 bytes a cycle, half of these.
__device__ __forceinline__ uint64_t tile_desc_sw64(uint32_t addr) {
  return (uint64_t) ((addr >> 4) & 0x3FFFu) | (uint64_t) 1 << 16 | (uint64_t) (512u >> 4) << 32 | (uint64_t) 1 << 46 | (uint64_t) 4 << 61;
}
// instruction descriptor: D F32, A and B f16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t idesc(uint32_t n) { return (1u << 4) | (n >> 3) << 17 | (uint32_t) (kM >> 4) << 24; }

__device__ __forceinline__ void bar_arrive_n(uint64_t* bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(n) : "memory");
}
__device__ __forceinline__ void arrive_when_copied(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// ---- the rows' raw bytes in shared memory ---------------------------------------------------------------------------
// This many values of K at a time (a whole number of blocks), in slots of an odd number of 16-byte pieces a row: the 16-byte
// reads of a warp - 32 rows - then take no more passes than their bytes need.
template <uint32_t T> constexpr uint32_t kRawK = (T == QTYPE_Q8_0 || T == QTYPE_MXFP8 || T == QTYPE_Q5_1) ? 128u : 256u;
template <uint32_t T> constexpr uint32_t kRawBytes = kRawK<T> / Fmt<T>::values * Fmt<T>::bytes;
template <uint32_t T> constexpr uint32_t kRawSlot = ((kRawBytes<T> + 30u + 15u) & ~15u) | 16u;
// a matrix whose rows all start on 16 bytes comes by tensor-map copies: a window of each row that starts on 16 bytes and holds the
// block's, again of an odd number of pieces
template <uint32_t T> constexpr uint32_t kLead = kRawBytes<T> % 16u == 0 ? 0u : kRawBytes<T> % 8u == 0 ? 8u : kRawBytes<T> % 4u == 0 ? 12u : 14u;
template <uint32_t T> constexpr uint32_t kWindow = ((kRawBytes<T> + kLead<T> + 15u) & ~15u) | 16u;
template <uint32_t T> constexpr uint32_t kRawPieces = (kRawBytes<T> + 30u) / 16u;  // of a row that starts anywhere in its first piece
template <uint32_t T> constexpr uint32_t kRawStages = (92u * 1024u) / (kM * kRawSlot<T>) < 4u ? (92u * 1024u) / (kM * kRawSlot<T>) : 4u;
// shared memory: the tokens' ring (1024-byte aligned), the raw ring, the gated mean's exchange, the matrices' first tiles
template <uint32_t EPI> constexpr uint32_t kTokenRing = (EPI == 2u ? 96u : 128u) * 1024u;
constexpr uint32_t kChunkTok = 16;  // tokens the epilogue reads at a time
constexpr uint32_t kExchange = kChunkTok * kM * 4u;
template <uint32_t T, uint32_t EPI> constexpr uint32_t kRawAt = kTokenRing<EPI>;
template <uint32_t T, uint32_t EPI> constexpr uint32_t kExAt = kRawAt<T, EPI> + kRawStages<T> * kM * kRawSlot<T>;
template <uint32_t T, uint32_t EPI> constexpr uint32_t kFirstAt = kExAt<T, EPI> + (EPI == 2u ? kExchange : 0u);
template <uint32_t T, uint32_t EPI> constexpr uint32_t kSmem = kFirstAt<T, EPI> + (kMaxMats + 1u) * 4u;

__device__ __forceinline__ uint32_t half2_bits(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *(const uint32_t*) &h;
}
__device__ __forceinline__ uint32_t half2_bits(uint64_t v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return half2_bits(lo, hi);
}
__device__ __forceinline__ uint32_t lds_half(uint32_t at) { return lds8(at) | lds8(at + 1) << 8; }  // (any address)

// the words of PIECES aligned 16-byte pieces of shared memory; bytes and words out of them at offsets known when compiled
template <int PIECES> struct Pieces {
  uint32_t w[4 * PIECES];
  __device__ __forceinline__ void load(uint32_t at) {
#pragma unroll
    for (int i = 0; i < PIECES; i++) {
      const int4 v = lds128(at + 16u * i);
      w[4 * i] = (uint32_t) v.x, w[4 * i + 1] = (uint32_t) v.y, w[4 * i + 2] = (uint32_t) v.z, w[4 * i + 3] = (uint32_t) v.w;
    }
  }
  __device__ __forceinline__ uint32_t word(int o) const { return o % 4 ? __funnelshift_r(w[o / 4], w[o / 4 + 1], 8 * (o % 4)) : w[o / 4]; }
  __device__ __forceinline__ uint32_t byte(int o) const { return __byte_perm(w[o / 4], 0, 0x4440 + o % 4); }
  __device__ __forceinline__ uint32_t half(int o) const { return word(o) & 0xFFFFu; }
};
// the step's bytes, N of them from any address, moved to the front of Pieces: the pieces around them, then the words and bytes
// shifted into place (a warp's aligned 4-byte reads of its 32 rows would meet four to a bank)
template <int N> struct Moved : Pieces<(N + 3) / 16 + 2> {
  __device__ __forceinline__ void load(uint32_t at) {
    constexpr int kWords = (N + 3) / 4, kAll = 4 * ((N + 3) / 16 + 2);
    static_assert(kWords + 4 <= kAll, "the words moved");
    Pieces<(N + 3) / 16 + 2>::load(at & ~15u);
    uint32_t(&w)[kAll] = this->w;
    const bool two = (at & 8u) != 0, one = (at & 4u) != 0;
    const uint32_t sh = (at & 3u) * 8u;
#pragma unroll
    for (int i = 0; i < kWords + 2; i++) w[i] = two ? w[i + 2] : w[i];
#pragma unroll
    for (int i = 0; i < kWords + 1; i++) w[i] = one ? w[i + 1] : w[i];
#pragma unroll
    for (int i = 0; i < kWords; i++) w[i] = __funnelshift_r(w[i], w[i + 1], sh);
  }
};
__device__ __forceinline__ uint4 lds_16(uint32_t at, bool whole) {  // 16 bytes on a word; whole: on 16 bytes
  if (whole) {
    const int4 v = lds128(at);
    return make_uint4((uint32_t) v.x, (uint32_t) v.y, (uint32_t) v.z, (uint32_t) v.w);
  }
  return make_uint4(lds32(at), lds32(at + 4u), lds32(at + 8u), lds32(at + 12u));
}

// ---- 64 values of a row to f16 --------------------------------------------------------------------------------------
// Every value is the F32 decode8 gives, then rounded to f16. A code n < 1024 in the low bits of a half IS the subnormal f16
// n 2^-24, which reaches F32 exactly (the bits of a word's codes are masked in place, two at a time; the conversion runs beside the
// integer pipe, which a byte permute a code kept busy); the scale is taken 2^24 times larger. Where d n (the scale's product
// with the integer fields included) has at most 24 significant bits, as in all of these types, fma(d, n, c) is the product
// rounded, exactly, and then the sum, rounded: decode8's two operations. An infinite or NaN scale is not exact times 2^24 or an
// integer, so such a step goes through decode8 (`odd`: the warp's, as tcgen05.st is the whole warp's).
struct Affine {  // n 2^-24 -> d n + c
  uint64_t d, c;
  __device__ __forceinline__ Affine(float scale, float plus) : d(pack2(mul_rn(scale, 16777216.0f), mul_rn(scale, 16777216.0f))), c(pack2(plus, plus)) {}
  // codes 0 and 2 (a0), 1 and 3 (a1) in the halves -> (r0, r1): the four values in order, as f16
  __device__ __forceinline__ void halves(uint32_t a0, uint32_t a1, uint32_t& r0, uint32_t& r1) const {
    r0 = half2_bits(fma2(d, pack2(low_half(a0), low_half(a1)), c));
    r1 = half2_bits(fma2(d, pack2(high_half(a0), high_half(a1)), c));
  }
  __device__ __forceinline__ void bytes(uint32_t u, uint32_t& r0, uint32_t& r1) const { halves(u & 0x00FF00FFu, __byte_perm(u, 0, 0x4341), r0, r1); }
};
// an E2M1 code's bits as an F16's sign, exponent's low two bits and mantissa's top one are its value times 2^-14 (a
// subnormal code is a subnormal F16): `top` holds such upper bytes of four values, times f
__device__ __forceinline__ void e2m1_halves(uint32_t top, __half2 f, uint32_t& r0, uint32_t& r1) {
  const uint32_t p0 = __byte_perm(top, 0, 0x1404), p1 = __byte_perm(top, 0, 0x3424);
  const __half2 h0 = __hmul2_rn(*(const __half2*) &p0, f), h1 = __hmul2_rn(*(const __half2*) &p1, f);
  r0 = *(const uint32_t*) &h0, r1 = *(const uint32_t*) &h1;
}
__device__ __forceinline__ bool inf_or_nan(uint32_t half_bits) { return (half_bits & 0x7C00u) == 0x7C00u; }

// K step `sub` of the raw K block whose row starts at shared address `at` (p: the same as a pointer): put(q, r) takes the
// values 16 q .. 16 q + 15 as eight f16 pairs; the whole warp calls it, in step
template <uint32_t T, class Put>
__device__ __forceinline__ void decode_step_any(const uint8_t* p, uint32_t sub, const Grids& g, const Put& put) {
#pragma unroll 1
  for (uint32_t q = 0; q < (uint32_t) kSubs; q++) {
    uint32_t r[8];
#pragma unroll
    for (uint32_t i = 0; i < 2; i++) {
      const uint32_t cl = sub * (kStep / kChunk) + 2u * q + i;  // the chunk's index in its K block
      float v[kChunk];
      decode8<T>(p + (cl / Fmt<T>::chunks) * Fmt<T>::bytes, (int) (cl % Fmt<T>::chunks), v, g);
#pragma unroll
      for (uint32_t j = 0; j < 4; j++) r[4 * i + j] = half2_bits(v[2 * j], v[2 * j + 1]);
    }
    put(q, r);
  }
}

// the 32-value types: a step's two blocks at byte O of b (a Pieces); false: an odd scale, nothing put
template <uint32_t T, int O, class B, class Put>
__device__ __forceinline__ bool two_blocks(const B& b, const Put& put) {
  constexpr int kNext = Fmt<T>::bytes;
  if constexpr (T == QTYPE_MXFP4) {
    // times 2^(e - 127): the f16 product by 2^(e - 113) is exact or rounds once, as the F32 value's conversion does - past
    // F16 infinite, below it zero. 2^(e - 113) is an F16 for e <= 128; below e = 99 every value is under half of F16's
    // least (6 2^-29), so the factor may be zero; a larger exponent is odd.
    const uint32_t e0 = b.byte(O), e1 = b.byte(O + kNext);
    if (__any_sync(0xFFFFFFFFu, max(e0, e1) > 128u)) return false;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t e = i ? e1 : e0, f = e >= 99u ? (e - 98u) << 10 : 0u, f2 = f | f << 16;
      const __half2 fh = *(const __half2*) &f2;
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t q = b.word(O + kNext * i + 1 + 4 * k);
        e2m1_halves(((q << 1) & 0x0E0E0E0Eu) | ((q << 4) & kTops), fh, lo[2 * k], lo[2 * k + 1]);
        e2m1_halves(((q >> 3) & 0x0E0E0E0Eu) | (q & kTops), fh, hi[2 * k], hi[2 * k + 1]);
      }
      put(2u * i, lo), put(2u * i + 1u, hi);
    }
  } else {
    const uint32_t h0 = b.half(O), h1 = b.half(O + kNext);
    if (__any_sync(0xFFFFFFFFu, inf_or_nan(h0) || inf_or_nan(h1))) return false;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const float d = half_value(i ? h1 : h0);
      uint32_t lo[8], hi[8];
      if constexpr (T == QTYPE_Q4_0) {  // (the high nibbles where they lie: 16 n under a sixteenth of the scale)
        const Affine a(d, mul_rn(d, -8.0f)), b16(mul_rn(d, 0.0625f), mul_rn(d, -8.0f));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t q = b.word(O + kNext * i + 2 + 4 * k), q8 = q >> 8;
          a.halves(q & 0x000F000Fu, q8 & 0x000F000Fu, lo[2 * k], lo[2 * k + 1]);
          b16.halves(q & 0x00F000F0u, q8 & 0x00F000F0u, hi[2 * k], hi[2 * k + 1]);
        }
      } else {  // Q8_0: the signed byte as q + 128
        const Affine a(d, mul_rn(d, -128.0f));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          a.bytes(b.word(O + kNext * i + 2 + 4 * k) ^ kTops, lo[2 * k], lo[2 * k + 1]);
          a.bytes(b.word(O + kNext * i + 18 + 4 * k) ^ kTops, hi[2 * k], hi[2 * k + 1]);
        }
      }
      put(2u * i, lo), put(2u * i + 1u, hi);
    }
  }
  return true;
}
// ... of step SUB, whose K block starts A bytes (0 or 8) into a 16-byte piece
template <uint32_t T, int SUB, int A, class Put>
__device__ __forceinline__ bool two_blocks_at(uint32_t piece, const Put& put) {
  constexpr int kFrom = A + SUB * 2 * Fmt<T>::bytes, kTo = kFrom + 2 * Fmt<T>::bytes, kPiece = kFrom / 16;
  Pieces<(kTo + 15) / 16 - kPiece> b;
  b.load(piece + 16u * kPiece);
  return two_blocks<T, kFrom - 16 * kPiece>(b, put);
}
template <uint32_t T, int A, class Put>
__device__ __forceinline__ bool two_blocks_in(uint32_t piece, uint32_t sub, const Put& put) {
  if (sub == 0) return two_blocks_at<T, 0, A>(piece, put);
  if constexpr (kRawK<T> == 256) {
    if (sub == 2) return two_blocks_at<T, 2, A>(piece, put);
    if (sub == 3) return two_blocks_at<T, 3, A>(piece, put);
  }
  return two_blocks_at<T, 1, A>(piece, put);
}

template <bool HI, class Put>  // Q6_K: HI, the step whose nibbles are the high ones
__device__ __forceinline__ void q6_step(uint32_t at, uint32_t sub, float d, const Put& put) {
  const uint32_t ql = at + 64u * (sub >> 1), qh = at + 128u + 32u * (sub >> 1);
#pragma unroll
  for (uint32_t i = 0; i < 2; i++) {
    Moved<16> top;
    top.load(qh + 16u * i);
#pragma unroll
    for (uint32_t b = 0; b < 2; b++) {  // sub-blocks 2 sub, 2 sub + 1: their top bit pairs at bits 4 HI + 2 b of the same bytes
      Moved<16> low;
      uint32_t r[8];
      low.load(ql + 32u * b + 16u * i);
      const float ds = mul_rn(d, (float) (int) (int8_t) lds8(at + 192u + 4u * sub + 2u * b + i));
      const Affine a(ds, mul_rn(ds, -32.0f));
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const uint32_t n = HI ? low.w[k] >> 4 : low.w[k];
        const uint32_t t = HI ? (b ? top.w[k] >> 2 : top.w[k]) : (b ? top.w[k] << 2 : top.w[k] << 4);
        a.bytes((n & kLow4) | (t & 0x30303030u), r[2 * k], r[2 * k + 1]);
      }
      put(2u * b + i, r);
    }
  }
}

// The other types (all but NVFP4 and MXFP8, whose codes are no integers): a step's bytes as words in registers, taken apart by
// decode.cuh's field readers - a sub-block's fields once, not once a chunk - and the codes to F16 as above, eight of them (c) to four
// pairs. Chunk by chunk out of shared memory these were bound by its passes (every byte, half and word of 32 rows meets four to a bank)
// and by the integers' conversions, and a tile's weights decode once a 256 tokens: 17408 x 5120 at 2048 tokens Q3_K 936 -> 400 us, Q5_1
// 655 -> 378, NVFP4 (its own way below) 625 -> 359, IQ4_XS 612 -> 456, IQ3_XXS 580 -> 457, IQ2_XXS 580 -> 431, Q2_K 563 -> 384, IQ1_M 542
// -> 403 (decoded into shared memory once a 512 tokens they took 488 to 534); 4096 x 4096 at 64 tokens 37-71 -> 23-35.
template <uint32_t T>
__device__ __forceinline__ void chunk_halves(const Chunk& c, uint32_t* r) {
  uint32_t lo = (uint32_t) c.lo, hi = (uint32_t) c.hi;
  float scale = c.d, plus;
  if constexpr (T == QTYPE_Q5_1) {
    plus = c.e;
  } else if constexpr (T == QTYPE_Q2_K) {
    scale = mul_rn(c.d, (float) c.s), plus = -mul_rn(c.e, (float) c.m);
  } else if constexpr (T == QTYPE_IQ1_S || T == QTYPE_IQ1_M) {  // -1, 0, 1 as 0, 1, 2; (d (2 s + 1)) (grid +- 1/8), exact
    scale = mul_rn(c.d, (float) (2 * c.s + 1)), plus = mul_rn(scale, c.m < 0 ? -1.125f : -0.875f);
    lo = (lo ^ kTops) - 0x7F7F7F7Fu, hi = (hi ^ kTops) - 0x7F7F7F7Fu;
  } else {  // a signed byte as it and 128
    if constexpr (T == QTYPE_Q3_K || T == QTYPE_IQ4_XS) scale = mul_rn(c.d, (float) c.s);
    else if constexpr (T == QTYPE_IQ3_XXS) scale = mul_rn(mul_rn(c.d, 0.5f + (float) c.s), 0.5f);
    else if constexpr (T == QTYPE_IQ2_XXS || T == QTYPE_IQ2_XS || T == QTYPE_IQ2_S) scale = mul_rn(mul_rn(c.d, 0.5f + (float) c.s), 0.25f);
    plus = mul_rn(scale, -128.0f), lo ^= kTops, hi ^= kTops;
  }
  const Affine a(scale, plus);
  a.bytes(lo, r[0], r[1]), a.bytes(hi, r[2], r[3]);
}
// The words of a row's block that hold step `sub`'s fields, each field where step 0's lies, so that the readers' offsets are known
// when compiled whatever the step is. (Four copies of the code, a step each - the four teams are on the four steps at once, and their
// instructions do not fit: IQ3_XXS 829 us where this takes 457.)
template <uint32_t T> constexpr int kFieldWords = (Fmt<T>::values == 32 ? 2 * Fmt<T>::bytes : Fmt<T>::bytes) / 4 + 2;
template <uint32_t T>
__device__ __forceinline__ void load_fields(const uint8_t* p, uint32_t sub, WordWindow<kFieldWords<T>, 0>& rd) {
  const uint32_t at = smem_addr(p);
  auto words = [&](int first, int n, uint32_t from, uint32_t shift) {  // words first .. first + n - 1, `from` bytes on
    const uint8_t* const src = p + from;
    const uint32_t lead = (at + from) & 3u;
    const uint32_t* const al = (const uint32_t*) (src - lead);
#pragma unroll
    for (int i = first; i < first + n; i++) rd.w[i] = __funnelshift_r(al[i], al[i + 1], 8u * lead) >> shift;
  };
  auto scale = [&]() { rd.w[0] = (rd.w[0] & 0xFFFF0000u) | lds_half(at); };
  if constexpr (T == QTYPE_IQ2_XXS) {
    words(0, 5, 16u * sub, 0), scale();
  } else if constexpr (T == QTYPE_IQ2_XS) {
    words(0, 5, 16u * sub, 0), scale(), rd.w[16] = lds_half(at + 66u + 2u * sub) << 16;
  } else if constexpr (T == QTYPE_IQ3_XXS) {
    words(0, 5, 16u * sub, 0), scale(), words(16, 3, 8u * sub, 0);
  } else if constexpr (T == QTYPE_IQ2_S) {
    words(0, 3, 8u * sub, 0), scale(), words(8, 3, 8u * sub, 0), rd.w[16] = lds_half(at + 66u + 2u * sub) << 16, rd.w[18] = lds_half(at + 74u + 2u * sub) << 16;
  } else if constexpr (T == QTYPE_IQ1_S) {
    words(0, 3, 8u * sub, 0), scale(), words(8, 2, 4u * sub, 0);
  } else if constexpr (T == QTYPE_IQ1_M) {
    words(0, 2, 8u * sub, 0), words(8, 1, 4u * sub, 0), words(12, 2, 0, 0);
  } else if constexpr (T == QTYPE_IQ4_XS) {
    rd.w[0] = lds_half(at) | (lds_half(at + 2u) >> (4u * sub)) << 16, rd.w[1] = lds8(at + 4u + sub), words(2, 8, 32u * sub, 0);
  } else if constexpr (T == QTYPE_Q2_K) {
    words(0, 1, 4u * sub, 0), words(4, 8, 32u * (sub >> 1), 4u * (sub & 1u)), words(20, 1, 0, 0);
  } else if constexpr (T == QTYPE_Q3_K) {
    words(0, 8, 0, 2u * sub), words(8, 8, 32u * (sub >> 1), 4u * (sub & 1u));
    words(24, 1, 4u * (sub & 1u), 4u * (sub >> 1)), words(26, 1, 0, 2u * sub), words(27, 1, 0, 0);
  } else {  // a block or two of the step's own
    words(0, kFieldWords<T> - 1, sub * (kStep / Fmt<T>::values) * Fmt<T>::bytes, 0);
  }
}
template <class Put>
__device__ __forceinline__ void nvfp4_step(const uint8_t* p, uint32_t sub, const Put& put) {
  WordWindow<kFieldWords<QTYPE_NVFP4>, 0> rd;
  load_fields<QTYPE_NVFP4>(p, sub, rd);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    // a UE4M3 byte's magnitude in an F16's exponent and mantissa is it times 2^-8, and the byte 0x7F is zero; an E2M1 code by an
    // F16 scale: at most six bits from 2^-10 to 2880, so every product here is exact
    const uint32_t c = rd.u8(q), h = c == 0x7Fu ? 0u : (c & 0x7Fu) << 7, h2 = h | h << 16;
    const __half2 f = __hmul2_rn(*(const __half2*) &h2, __float2half2_rn(256.0f)), one = __float2half2_rn(16384.0f);
    uint32_t r[8];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint32_t w = rd.u32(4 + 8 * q + 4 * k);
      e2m1_halves(((w << 1) & 0x0E0E0E0Eu) | ((w << 4) & kTops), one, r[2 * k], r[2 * k + 1]);
      e2m1_halves(((w >> 3) & 0x0E0E0E0Eu) | (w & kTops), one, r[4 + 2 * k], r[5 + 2 * k]);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const __half2 v = __hmul2_rn(*(const __half2*) &r[k], f);
      r[k] = *(const uint32_t*) &v;
    }
    put((uint32_t) q, r);
  }
}
// false: an odd scale, nothing put
template <uint32_t T, class Put>
__device__ __forceinline__ bool fields_step(const uint8_t* p, uint32_t sub, const Grids& g, const Put& put) {
  WordWindow<kFieldWords<T>, 0> rd;
  load_fields<T>(p, sub, rd);
  constexpr bool kTwo = Fmt<T>::values == 32;  // (the step is two blocks; else two sub-blocks of one)
  const PlainLuts lut{g};
  Sub sb[2];
  bool odd = false;
#pragma unroll
  for (int b = 0; b < 2; b++) {
    sb[b] = sub_of<T>(rd, kTwo ? b * Fmt<T>::bytes : 0, kTwo ? 0 : b);
    odd = odd || !(fabsf(sb[b].d) < __uint_as_float(0x7F800000u));
    if constexpr (T == QTYPE_IQ1_M) sb[b].a = ((sub & 2u) ? sb[b].b : sb[b].a) >> (16u * (sub & 1u));  // (the step's scale word)
  }
  if (__any_sync(0xFFFFFFFFu, odd)) return false;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int b = q >> 1;
    uint32_t r[8];
#pragma unroll
    for (int i = 0; i < 2; i++)
      chunk_halves<T>(chunk_of<T>(rd, kTwo ? b * Fmt<T>::bytes : 0, kTwo ? 0 : b, 2 * (q & 1) + i, sb[b], lut), r + 4 * i);
    put((uint32_t) q, r);
  }
  return true;
}

template <uint32_t T, class Put>
__device__ __forceinline__ void decode_step(uint32_t at, const uint8_t* p, uint32_t sub, const Grids& g, const Put& put) {
  if constexpr (T == QTYPE_Q4_K || T == QTYPE_Q5_K) {
    // the step is groups 2 sub and 2 sub + 1: the low and the high nibbles of the same 32 bytes
    const bool whole = __all_sync(0xFFFFFFFFu, (at & 15u) == 0);
    uint4 h = make_uint4(0x7C00u, 0, 0, 0);
    if (__all_sync(0xFFFFFFFFu, (at & 3u) == 0)) h = lds_16(at, whole);
    if (__any_sync(0xFFFFFFFFu, inf_or_nan(h.x) || inf_or_nan(h.x >> 16))) return decode_step_any<T>(p, sub, g, put);
    uint32_t sc, mn;
    k_scales(h.y, h.z, h.w, 16u * (sub & 1u), sub >= 2u, sc, mn);
    const float d = half_value(h.x & 0xFFFFu), m = -half_value(h.x >> 16);
    const float s0 = mul_rn(d, byte_value<0>(sc)), s1 = mul_rn(d, byte_value<1>(sc));
    const float m0 = mul_rn(m, byte_value<0>(mn)), m1 = mul_rn(m, byte_value<1>(mn));  // (minus the minimum)
    if constexpr (T == QTYPE_Q4_K) {  // (the high nibbles where they lie: 16 n under a sixteenth of the scale)
      const Affine a(s0, m0), b(mul_rn(s1, 0.0625f), m1);
#pragma unroll
      for (uint32_t i = 0; i < 2; i++) {
        const uint4 q = lds_16(at + 16u + 32u * sub + 16u * i, whole);
        const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t q8 = qw[k] >> 8;
          a.halves(qw[k] & 0x000F000Fu, q8 & 0x000F000Fu, lo[2 * k], lo[2 * k + 1]);
          b.halves(qw[k] & 0x00F000F0u, q8 & 0x00F000F0u, hi[2 * k], hi[2 * k + 1]);
        }
        put(i, lo), put(2u + i, hi);
      }
    } else {
      const Affine a(s0, m0), b(s1, m1);
#pragma unroll
      for (uint32_t i = 0; i < 2; i++) {
        const uint4 q = lds_16(at + 48u + 32u * sub + 16u * i, whole), f = lds_16(at + 16u + 16u * i, whole);
        const uint32_t qw[4] = {q.x, q.y, q.z, q.w};  // the fifth bits: bits 2 sub and 2 sub + 1 of the 32 bytes at 16
        const uint32_t fw[4] = {f.x >> (2u * sub), f.y >> (2u * sub), f.z >> (2u * sub), f.w >> (2u * sub)};
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          a.bytes((qw[k] & kLow4) | ((fw[k] << 4) & 0x10101010u), lo[2 * k], lo[2 * k + 1]);
          b.bytes(((qw[k] >> 4) & kLow4) | ((fw[k] << 3) & 0x10101010u), hi[2 * k], hi[2 * k + 1]);
        }
        put(i, lo), put(2u + i, hi);
      }
    }
  } else if constexpr (T == QTYPE_Q4_0 || T == QTYPE_MXFP4 || T == QTYPE_Q8_0) {
    // (rows of whole 16-byte pieces lie alike: the places of the step's bytes are then known when compiled)
    bool done;
    if (__all_sync(0xFFFFFFFFu, (at & 15u) == 0)) {
      done = two_blocks_in<T, 0>(at, sub, put);
    } else if (__all_sync(0xFFFFFFFFu, (at & 15u) == 8u)) {
      done = two_blocks_in<T, 8>(at & ~15u, sub, put);
    } else {
      Moved<2 * Fmt<T>::bytes> b;
      b.load(at + sub * 2u * Fmt<T>::bytes);
      done = two_blocks<T, 0>(b, put);
    }
    if (!done) decode_step_any<T>(p, sub, g, put);
  } else if constexpr (T == QTYPE_Q6_K) {
    const uint32_t h = lds_half(at + 208u);
    if (__any_sync(0xFFFFFFFFu, inf_or_nan(h))) return decode_step_any<T>(p, sub, g, put);
    if (sub & 1u) q6_step<true>(at, sub, half_value(h), put);
    else q6_step<false>(at, sub, half_value(h), put);
  } else if constexpr (T == QTYPE_NVFP4) {
    nvfp4_step(p, sub, put);
  } else if constexpr (T == QTYPE_MXFP8) {
    decode_step_any<T>(p, sub, g, put);
  } else {
    if (!fields_step<T>(p, sub, g, put)) decode_step_any<T>(p, sub, g, put);
  }
}

struct Args {
  const uint8_t* w;          // one matrix (wt NULL)
  const uint8_t* const* wt;  // grouped: the matrices
  const int32_t* cnt;        // grouped: tokens a matrix
  const uint32_t *xoff, *yoff;  // grouped: where a matrix's tokens start in x16 (halves) and y (floats)
  const __half* x16;
  float* y;
  uint32_t rows, cols, n, xts, ys;
  uint32_t n_mat, row_tiles;
  // a second matrix over the same tokens (w1 NULL: none), its row tiles after the first one's in the same launch: the shared
  // expert's gate and up, 16 row tiles each, 32 us one after the other
  const uint8_t* w1;
  float* y1;
  uint32_t rows1, ys1, row_tiles1;
  float scale1;
  uint32_t span;     // the most tokens a tile takes
  uint32_t use_tma;  // the activations come by tensor-map copies, else by 16-byte cp.async
  uint32_t early;    // the kernel ahead made x16 (mm_tokens): what does not need it starts before it has ended
  uint32_t raw_map;  // the weights too (Maps::raw); grouped: the matrices are those of one tensor, `bytes` apart from `base` on
  const uint8_t* base;
  uint64_t bytes;
  uint32_t n_base;
  float scale;
  uint32_t* status;
  // the epilogue (the kernel's EPI): kStore y = scale sum; kSilu y = silu(scale sum), and its f16 into x16_out (rows wide, tiled);
  // kGatedMean: the matrix is hc streams of dim rows, out[t][d] = (sum over s in order of xn[t][s][d]
  // sigmoid(sum_t[s dim + d])) / hc, and its f16 into x16_out (dim wide, token t at row out_row0 + t; NULL: none)
  __half* x16_out;
  int32_t* overflow;
  const float* xn;
  float* out;
  uint32_t hc, dim, per, out_row0;  // per: the dim values a tile takes (hc per <= 128 of its rows are used)
};
struct Maps {  // the tokens' maps: of a grouped launch map t a box of t + 1 token tiles, else the one map's box is a.span tokens
  CUtensorMap map[kMaxSpan / MM_TILE];
  CUtensorMap raw, raw1;  // the weights' bytes as [matrix][row][byte]; the second matrix's
};
enum : uint32_t { kStore = 0, kSilu = 1, kGatedMean = 2 };

struct Shared {
  // of a unit - one K step or two - full_a: their weights are in tensor memory; full_b: their tokens in shared memory; empty: their products
  // have run (so the weights' stages, and the tokens' slot of the token ring, are free)
  uint64_t full_a[kSteps], full_b[kSteps], empty[kSteps], full_raw[4], empty_raw[4], full_acc[2], empty_acc[2], drain;
  uint32_t tmem_base, max_tok, warp_tiles[kThreads / kWarp], warp_tok[kThreads / kWarp];
  int fail, epi_fail;
};

__host__ __device__ constexpr uint32_t whole16(uint32_t n) { return (n + 15u) & ~15u; }
__host__ __device__ constexpr uint32_t parts_of(uint32_t n, uint32_t of) { return (n + of - 1u) / of; }

// A wait on a raw slot names its phase by a parity, so it is right only where the phase before is known to be over. A producer team
// sees every phase of its slots but where a row of an odd multiple of 128 values ends in half a block of 256: that block has a step
// for two of the four teams, and the other two go past it. Whether, wherever a team waits for block b, block b - slots has landed by what
// the team has waited for before: that block itself; or block b' of its own, for which the loader had seen b' - slots and those before used up; or
// the products of step s - 8, s its last step (they end in order, and each step's block had landed). Rows of 2 .. 40 steps, `whole`
// at a time, tiles enough to repeat. (Three slots of 256 values do not hold - a team could take the phase before for its own and
// decode bytes that had not landed - so Q5_1, whose 256 values leave room for three, has blocks of 128.)
constexpr bool phases_known(uint32_t slots, uint32_t steps_raw, uint32_t whole) {
  for (uint32_t steps = whole; steps <= 40; steps += whole) {
    const uint32_t blocks = parts_of(steps, steps_raw);
    for (uint32_t team = 0; team < (uint32_t) kTeams; team++) {
      uint32_t own[64] = {}, n = 0, most = 0, last = 0;  // its blocks so far, less 1 the greatest; its last step
      for (uint32_t tile = 0; tile * blocks < 12 * slots; tile++) {
        const uint32_t s0 = tile * steps;
        for (uint32_t it = (team - s0) % (uint32_t) kTeams; it < steps; it += (uint32_t) kTeams) {
          const uint32_t b = tile * blocks + it / steps_raw;
          if (b >= slots) {
            const uint32_t before = b - slots;
            bool known = most > slots && before <= most - 1 - slots;
            for (uint32_t i = 0; i < n && i < 64; i++) known = known || own[i] == before + 1;
            if (last >= kSteps) {
              const uint32_t s = last - kSteps;
              known = known || before <= s / steps * blocks + s % steps / steps_raw;
            }
            if (!known) return false;
          }
          own[n++ % 64] = b + 1, most = b + 1, last = s0 + it;
        }
      }
    }
  }
  return true;
}

// Tile number t of the launch: tiles go matrix by matrix, row tile by row tile, a row tile's token tiles side by side (they
// share the weights' bytes in L2). first[m]: matrix m's first tile; m: where the last search ended (a role's tiles only
// go up). A matrix's tokens are dealt in equal whole tiles of 16.
struct Tile {
  uint32_t m, rt, c0, n;  // its matrix and row tile; its first token and their number
  bool second;            // the second matrix's
};
__device__ __forceinline__ Tile tile_at(const Args& a, const uint32_t* first, uint32_t t, uint32_t& m, uint32_t lane) {
  if (a.wt) {
    for (;;) {
      const uint32_t i = m + 1u + lane;
      const uint32_t past = __popc(__ballot_sync(0xFFFFFFFFu, first[i < a.n_mat ? i : a.n_mat] <= t && i <= a.n_mat));
      m += past;
      if (past < 32u) break;
    }
  }
  const uint32_t n = a.wt ? (uint32_t) a.cnt[m] : a.n, in = t - first[m], cols = parts_of(n, a.span);
  const uint32_t each = whole16(parts_of(n, cols));
  Tile r;
  r.m = m, r.rt = in / cols, r.c0 = (in - r.rt * cols) * each;
  r.second = r.rt >= a.row_tiles;
  if (r.second) r.rt -= a.row_tiles;
  r.n = r.c0 < n ? min(each, n - r.c0) : 0u;
  return r;
}

// EPI: the epilogue (kStore / kSilu / kGatedMean), a compile-time choice so that the plain product carries none of
// the others' code
template <uint32_t T, uint32_t EPI>
__global__ void __launch_bounds__(kThreads, 1) mm_tc_kernel(const Args a, const __grid_constant__ Maps maps) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ Shared sh;
  __shared__ __align__(16) uint8_t tables[grid_smem_bytes<T>() > 0 ? grid_smem_bytes<T>() : 16];
  const uint32_t tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
  const uint32_t steps = a.cols / kStep;
  const uint64_t row_bytes = (uint64_t) (a.cols / Fmt<T>::values) * Fmt<T>::bytes;
  constexpr uint32_t kStepsRaw = kRawK<T> / kStep, kSlot = kRawSlot<T>;
  const uint32_t kblocks = parts_of(steps, kStepsRaw);
  uint32_t* const first = (uint32_t*) (smem + kFirstAt<T, EPI>);
  uint8_t* const raw = smem + kRawAt<T, EPI>;
  const uint32_t pitch = a.raw_map ? kWindow<T> : kSlot;  // a row's bytes in the raw ring
  static_assert(kWindow<T> <= kSlot, "either fits");

  if (tid == 0) {
    for (uint32_t i = 0; i < kSteps; i++) bar_init(&sh.full_b[i], 1), bar_init(&sh.empty[i], 1);
    for (int i = 0; i < 4; i++)
      bar_init(&sh.full_raw[i], a.raw_map ? 1 : kRawWarps * kWarp), bar_init(&sh.empty_raw[i], (kProdWarps / kTeams) * kStepsRaw);
    for (int i = 0; i < 2; i++) bar_init(&sh.full_acc[i], 1), bar_init(&sh.empty_acc[i], kEpiWarps);
    bar_init(&sh.drain, 1);
    sh.fail = 0, sh.epi_fail = 0;
    bar_init_fence();
  }
  if (warp == (uint32_t) kIssuerWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem_base)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // (a dependent launch: the counts, x16 and the readers of y may be the kernel ahead's. Where that kernel is this call's own
  // conversion - launched the ordinary way, so that whatever wrote the weights is over - the weights' loads and their
  // decoding need not wait for it, only the tokens' loads and the stores. Passes of mm_tokens back to back, Q4_K 4096 x 2048 at
  // 2048 tokens: 41.4 -> 39.9 us; MXFP4 2560 x 1536, 126 tokens: 13.8 -> 12.7; elsewhere 0 to 4 %.)
  if (!a.early) pdl_wait();
  pdl_launch_next();
  // the matrices' first tiles, a thread each, and the most tokens a tile has
  const uint32_t n_mat = a.wt ? a.n_mat : 1u;
  static_assert(kMaxMats <= (uint32_t) kThreads, "a thread a matrix");
  {
    const uint32_t n = tid < n_mat ? (a.wt ? (uint32_t) max(a.cnt[tid], 0) : a.n) : 0u, cols = parts_of(n, a.span);
    const uint32_t mine = cols * (a.row_tiles + a.row_tiles1), most = __reduce_max_sync(0xFFFFFFFFu, n ? whole16(parts_of(n, cols)) : 0u);
    // (the pointers are the device's: one that is no matrix of the tensor comes through the map as another's rows, or as zeros)
    if (n && a.wt && a.raw_map) {
      const uint64_t at = (uint64_t) (a.wt[tid] - a.base), index = at / a.bytes;
      if (index >= a.n_base || index * a.bytes != at) atomicOr(a.status, kNotOfTensor);
    }
    uint32_t sum = mine;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, sum, o);
      if (lane >= (uint32_t) o) sum += v;
    }
    if (lane == kWarp - 1u) sh.warp_tiles[warp] = sum, sh.warp_tok[warp] = most;
    __syncthreads();
    uint32_t before = lane < warp ? sh.warp_tiles[lane] : 0u;
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    if (tid < n_mat) first[tid] = before + sum - mine;
    if (tid == n_mat - 1u) first[n_mat] = before + sum;
    const uint32_t tok = __reduce_max_sync(0xFFFFFFFFu, lane < (uint32_t) (kThreads / kWarp) ? sh.warp_tok[lane] : 0u);
    // the issuer goes by units: two steps where a tile is small and their products run shorter than a look at the barriers
    if (tid == 0) {
      sh.max_tok = tok;
      for (uint32_t i = 0; i < kSteps; i++) bar_init(&sh.full_a[i], (tok > (uint32_t) kN ? 1u : 2u) * kProdWarps / kTeams);
      bar_init_fence();
    }
  }
  const Grids g = stage_grids<T>(tables);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem_base;
  const uint32_t tiles = first[n_mat];
  // the token ring: slots of a unit's K steps of the largest tile's tokens, as many as fit, at most one a barrier (the products of
  // an odd number of token tiles read one past the last)
  const uint32_t slot_tiles = sh.max_tok ? sh.max_tok / MM_TILE : 1u, two = slot_tiles * MM_TILE > (uint32_t) kN ? 0u : 1u;  // (log2 of a unit's steps)
  const uint32_t units = kSteps >> two, unit_subs = kSubs << two;
  const uint32_t slot_bytes = (slot_tiles * unit_subs + (slot_tiles & 1u)) * 512u, slots = min(units, kTokenRing<EPI> / slot_bytes);
  uint32_t m_at = 0;  // (tile_at's)

  if (warp >= (uint32_t) kFirstProd && warp < (uint32_t) kIssuerWarp) {
    // ================= producers =================
    const uint32_t team = (warp - kFirstProd) / 4u, r = 32u * (warp % 4u) + lane;
    const uint32_t lane_cols = tmem + ((32u * (warp % 4u)) << 16) + kAccCols;
    uint32_t s0 = 0, rb0 = 0;  // the steps and raw blocks before this tile
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x, s0 += steps, rb0 += kblocks) {
      const Tile tl = tile_at(a, first, t, m_at, lane);
      const uint8_t* w = a.wt ? a.wt[tl.m] : tl.second ? a.w1 : a.w;
      const uint32_t rows = tl.second ? a.rows1 : a.rows;
      // (the weight row behind row r of the tile: see the raw loaders; here only where it starts in its 16-byte piece)
      uint32_t row;
      if constexpr (EPI == kGatedMean) {
        const uint32_t d0 = tl.rt * a.per, st = r / a.per, d = d0 + (r - st * a.per);
        row = (st < a.hc ? st : a.hc - 1) * a.dim + (d < a.dim ? d : a.dim - 1);
      } else {
        row = min(tl.rt * kM + r, rows - 1u);
      }
      const uint32_t base15 = (uint32_t) ((uintptr_t) (w + (uint64_t) row * row_bytes) & 15u);
      for (uint32_t it = (team - s0) % kTeams; it < steps; it += kTeams) {
        const uint32_t s = s0 + it, stage = s % kSteps, unit = stage >> two, kb = it / kStepsRaw, sub = it % kStepsRaw, rb = rb0 + kb, slot = rb % kRawStages<T>;
        if (!bar_wait_soon(&sh.full_raw[slot], (rb / kRawStages<T>) & 1u) ||  // (its parity: phases_known)
            (s >= kSteps && !bar_wait_soon(&sh.empty[unit], (s / kSteps - 1u) & 1u))) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t off = slot * (kM * kSlot) + r * pitch + ((base15 + kb * kRawBytes<T>) & 15u);
        const uint32_t col = lane_cols + stage * kStageCols;
        decode_step<T>(smem_addr(raw) + off, raw + off, sub, g, [&](uint32_t q, const uint32_t (&v)[8]) {
          asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(col + 8u * q), "r"(v[0]), "r"(v[1]),
                       "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                       : "memory");
        });
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          bar_arrive(&sh.full_a[unit]);
          // (the raw block's last step arrives for those a row's end leaves out)
          bar_arrive_n(&sh.empty_raw[slot], it == steps - 1u ? kStepsRaw - sub : 1u);
        }
      }
    }
    if (!ok) sh.fail = 1;
  } else if (warp >= (uint32_t) kFirstRaw && warp < (uint32_t) kTokenWarp) {
    // ================= the weights' loaders =================
    // The 16-byte pieces of the aligned span around each row's bytes (a block may start anywhere in a piece; every piece
    // asked for holds some of them): 64 threads take the pieces of kTogether rows in kRounds rounds whose places do not change
    // from block to block. (A loader that worked a row's address out for each copy held a K step to 1,000 cycles.)
    constexpr uint32_t kP = kRawPieces<T>, kLoaders = kRawWarps * kWarp;
    constexpr uint32_t kTogether = kP % 64u == 0 ? 1u : kP % 32u == 0 ? 2u : kP % 16u == 0 ? 4u : kP % 8u == 0 ? 8u : kP % 4u == 0 ? 16u : kP % 2u == 0 ? 32u : 64u;
    constexpr uint32_t kRounds = kTogether * kP / kLoaders;
    static_assert(kP <= 16u && kP * 16u <= kSlot && kRounds * kLoaders == kTogether * kP && kM % kTogether == 0, "the rows' pieces");
    const uint32_t lt = (warp - kFirstRaw) * kWarp + lane;
    uint32_t src_at[kRounds], dst_at[kRounds];
#pragma unroll
    for (uint32_t j = 0; j < kRounds; j++) {
      const uint32_t i = lt + j * kLoaders, r = i / kP, piece = i - r * kP;
      src_at[j] = r * (uint32_t) row_bytes + piece * 16u, dst_at[j] = r * kSlot + piece * 16u;
    }
    uint32_t rb = 0;
    bool ok = true;
    if (a.raw_map) {  // a copy a block: the second warp has nothing to do
      for (uint32_t t = blockIdx.x; t < tiles && ok && warp == (uint32_t) kFirstRaw; t += gridDim.x) {
        const Tile tl = tile_at(a, first, t, m_at, lane);
        const uint32_t mat = a.wt ? (uint32_t) ((uint64_t) (a.wt[tl.m] - a.base) / a.bytes) : 0u;
        for (uint32_t kb = 0; kb < kblocks; kb++, rb++) {
          const uint32_t slot = rb % kRawStages<T>;
          if (rb >= kRawStages<T> && !bar_wait_soon(&sh.empty_raw[slot], (rb / kRawStages<T> - 1u) & 1u)) {
            ok = false;
            break;
          }
          if (lane == 0) {  // (rows past the matrix, and bytes past a row's, are filled with zeros)
            bar_expect(&sh.full_raw[slot], kM * kWindow<T>);
            asm volatile(
                "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
                    smem_addr(raw) + slot * (kM * kSlot)),
                "l"(tl.second ? &maps.raw1 : &maps.raw), "r"((kb * kRawBytes<T>) & ~15u), "r"(tl.rt * kM), "r"(mat), "r"(smem_addr(&sh.full_raw[slot]))
                : "memory");
          }
          __syncwarp();
        }
      }
      if (!ok)  // (the copies in flight land before the block's shared memory is another's)
        for (uint32_t i = rb > kRawStages<T> ? rb - kRawStages<T> : 0u; i < rb; i++) bar_wait_warp(&sh.full_raw[i % kRawStages<T>], (i / kRawStages<T>) & 1u);
    }
    for (uint32_t t = blockIdx.x; t < tiles && ok && !a.raw_map; t += gridDim.x) {
      const Tile tl = tile_at(a, first, t, m_at, lane);
      const uint8_t* w = a.wt ? a.wt[tl.m] : tl.second ? a.w1 : a.w;
      const uint32_t rows = tl.second ? a.rows1 : a.rows;
      for (uint32_t kb = 0; kb < kblocks; kb++, rb++) {
        const uint32_t slot = rb % kRawStages<T>;
        if (rb >= kRawStages<T> && !bar_wait_soon(&sh.empty_raw[slot], (rb / kRawStages<T> - 1u) & 1u)) {
          ok = false;
          break;
        }
        const uint32_t dst = smem_addr(raw) + slot * (kM * kSlot);
        const uint64_t in_row = (uint64_t) kb * kRawBytes<T>;
        const uint32_t bytes = row_bytes - in_row < kRawBytes<T> ? (uint32_t) (row_bytes - in_row) : kRawBytes<T>;
        const uint32_t row0 = tl.rt * kM;
        auto copy = [&](uint32_t to, const uint8_t* from) {  // the piece `to` of a slot whose bytes start where `from` lies in its piece
          const uint32_t lead = (uint32_t) (uintptr_t) from & 15u;
          if (to % kSlot < lead + bytes)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + to), "l"(from - lead) : "memory");
        };
        if (EPI != kGatedMean && rows - row0 >= (uint32_t) kM && row_bytes < (1u << 24)) {
          const uint8_t* from = w + (uint64_t) row0 * row_bytes + in_row;
          for (uint32_t r0 = 0; r0 < (uint32_t) kM; r0 += kTogether, from += kTogether * row_bytes) {
#pragma unroll
            for (uint32_t j = 0; j < kRounds; j++) copy(r0 * kSlot + dst_at[j], from + src_at[j]);
          }
        } else {
          for (uint32_t r0 = 0; r0 < (uint32_t) kM; r0 += kTogether) {
#pragma unroll
            for (uint32_t j = 0; j < kRounds; j++) {
              // the weight row behind row r of the tile: the matrix's next 128 rows - or, for the gated mean, stream
              // r / per's row of value d0 + r % per, so the hc sums of one output value lie in one tile (a row past the
              // matrix, or past the streams, repeats a valid one and is never stored)
              const uint32_t to = r0 * kSlot + dst_at[j], r = to / kSlot;
              uint32_t row;
              if constexpr (EPI == kGatedMean) {
                const uint32_t d0 = tl.rt * a.per, st = r / a.per, d = d0 + (r - st * a.per);
                row = (st < a.hc ? st : a.hc - 1) * a.dim + (d < a.dim ? d : a.dim - 1);
              } else {
                row = min(row0 + r, rows - 1u);
              }
              copy(to, w + (uint64_t) row * row_bytes + in_row + to % kSlot);
            }
          }
        }
        arrive_when_copied(&sh.full_raw[slot]);
      }
    }
    if (!ok) sh.fail = 1;
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == (uint32_t) kTokenWarp) {
    // ================= the activations' loader =================
    if (a.early) pdl_wait();
    uint32_t s = 0, slot = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      const Tile tl = tile_at(a, first, t, m_at, lane);
      const uint32_t tok_tiles = whole16(tl.n) / MM_TILE;  // x16 holds whole tiles of 16 tokens
      const uint32_t sub_bytes = (a.wt ? tok_tiles : slot_tiles) * 512u;
      const uint32_t xoff = a.wt ? a.xoff[tl.m] : 0u, tile_halves = MM_TILE * a.xts;
      const uint32_t tile0 = xoff / tile_halves + tl.c0 / MM_TILE;
      const CUtensorMap* const map = &maps.map[a.wt ? tok_tiles - 1u : 0u];
      const bool mapped = a.use_tma && tile0 * tile_halves == xoff + (tl.c0 / MM_TILE) * tile_halves;
      const uint8_t* src0 = (const uint8_t*) (a.x16 + xoff + mm_x16_at(tl.c0, 0, a.xts)) + lane * 16u;
      const uint32_t dst0 = (lane >> 2) * 64u + (((lane & 3u) ^ ((lane >> 3) & 3u)) * 16u);
      for (uint32_t it = 0; it < steps; it += 1u << two, s++, src0 += MM_TILE * unit_subs * MM_TILE * 2u) {  // (s: units)
        if (s >= slots && !bar_wait_soon(&sh.empty[(s - slots) & (units - 1u)], ((s - slots) >> (3u - two)) & 1u)) {
          ok = false;
          break;
        }
        const uint32_t dst = smem_addr(smem) + slot * slot_bytes;
        uint64_t* const bar = &sh.full_b[s & (units - 1u)];
        if (mapped) {
          // the tiled x16 seen as [K fragment][token tile][two tokens][value]: one box is a step's four sub-tiles, swizzled as
          // the products read it (tiles past the last are filled with zeros); the barrier counts the bytes
          if (lane == 0) {
            bar_expect(bar, sub_bytes * unit_subs);
            for (uint32_t q = 0; q < unit_subs; q += kSubs)
              asm volatile(
                  "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
                      dst + q * sub_bytes),
                  "l"(map), "r"(0), "r"(0), "r"(tile0), "r"(it * kSubs + q), "r"(smem_addr(bar))
                  : "memory");
          }
          __syncwarp();
        } else {
          // tokens that start inside a tile of x16: a fragment a round, 512 bytes as they lie - lane = (two tokens, a quarter of
          // their 64 bytes), the quarter swizzled - waited for here and made visible to the tensor core
          const uint8_t* src = src0;
          uint32_t to = dst + dst0;
          for (uint32_t i = 0; i < tok_tiles; i++, src += tile_halves * 2u, to += 512u) {
            for (uint32_t q = 0; q < unit_subs; q++)
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + q * sub_bytes), "l"(src + q * 512u) : "memory");
          }
          asm volatile("cp.async.wait_all;" ::: "memory");
          fence_async_smem();
          __syncwarp();
          if (lane == 0) bar_arrive(bar);
        }
        if (++slot == slots) slot = 0;
      }
    }
    if (!ok) {  // (the copies in flight land before the block's shared memory is another's)
      sh.fail = 1;
      for (uint32_t i = s > slots ? s - slots : 0u; i < s; i++) bar_wait_warp(&sh.full_b[i & (units - 1u)], (i >> (3u - two)) & 1u);
    }
  } else if (warp == (uint32_t) kIssuerWarp) {
    // ================= issuer =================
    const uint32_t issuer = elect_one();
    uint32_t s = 0, slot = 0, acc = 0;  // acc: accumulators taken so far
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      const Tile tl = tile_at(a, first, t, m_at, lane);
      // a tile of up to 128 tokens has its even tokens' sums in an accumulator's first 64 columns, its odd ones' in the rest; a
      // larger one an accumulator of each
      const uint32_t uses = tl.n > (uint32_t) kN ? 2u : 1u, sub16 = (a.wt ? whole16(tl.n) / MM_TILE : slot_tiles) * (512u >> 4);
      for (uint32_t u = 0; u < uses && ok; u++)
        if (acc + u >= 2u && !bar_wait_soon(&sh.empty_acc[(acc + u) & 1u], ((acc + u) / 2u - 1u) & 1u)) ok = false;
      if (!ok) break;
      const uint32_t d0 = tmem + (acc & 1u) * kN, d1 = uses == 2u ? tmem + ((acc + 1u) & 1u) * kN : d0 + kN / 2;
      const uint32_t id = idesc(whole16((tl.n + 1u) / 2u));
      for (uint32_t it = 0; it < steps; it += 1u << two, s++) {  // (s: units)
        const uint32_t unit = s & (units - 1u), parity = (s >> (3u - two)) & 1u;
        if (!bar_wait_soon(&sh.full_b[unit], parity) || !bar_wait_soon(&sh.full_a[unit], parity)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t at = tmem + kAccCols + unit * (kStageCols << two);
        const uint64_t b0 = tile_desc_sw64(smem_addr(smem) + slot * slot_bytes);
        mma_f16_ts_k64(issuer, d0, d1, at, b0, sub16, id, it);
        if (two) mma_f16_ts_k64(issuer, d0, d1, at + kStageCols, b0 + 4u * sub16, sub16, id, 1u);
        mma_commit(issuer, &sh.empty[unit]);
        if (++slot == slots) slot = 0;
      }
      if (!ok) break;
      mma_commit(issuer, &sh.full_acc[acc & 1u]);
      if (uses == 2u) mma_commit(issuer, &sh.full_acc[(acc + 1u) & 1u]);
      acc += uses;
    }
    if (!ok) {  // (what has been issued ends before tensor memory is released)
      sh.fail = 1;
      mma_commit(issuer, &sh.drain);
      bar_wait_warp(&sh.drain, 0);
    }
  } else {
    // ================= epilogue =================
    if (a.early) pdl_wait();
    const uint32_t row = 32u * warp + lane;  // this thread's weight row of the tile = its TMEM lane
    uint32_t acc = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      const Tile tl = tile_at(a, first, t, m_at, lane);
      const uint32_t row0 = tl.rt * kM;
      const bool live = row0 + row < (tl.second ? a.rows1 : a.rows);
      const uint32_t ys = tl.second ? a.ys1 : a.ys;
      const float scale = tl.second ? a.scale1 : a.scale;
      const uint32_t uses = tl.n > (uint32_t) kN ? 2u : 1u;
      for (uint32_t u = 0; u < uses; u++, acc++) {  // the tile's accumulators
        const uint32_t buf = acc & 1u;
        ok = false;  // (a K loop's own waits are 0.2 s each and can queue up: look again while nobody has given up)
        for (uint32_t tries = 0; tries < 25u && !ok; tries++) {
          ok = bar_wait_long(&sh.full_acc[buf], (acc / 2u) & 1u);
          if (!ok && __any_sync(0xFFFFFFFFu, *(volatile int*) &sh.fail)) break;
        }
        if (!ok) sh.epi_fail = 1;
        // (the gated mean's warps meet below: all of them or none. Nobody writes the word between this barrier and the next.)
        if constexpr (EPI == kGatedMean) {
          asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * kWarp) : "memory");
          ok = *(volatile int*) &sh.epi_fail == 0;
        }
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        float* const y0 = (tl.second ? a.y1 : a.y) + (a.wt ? a.yoff[tl.m] : 0u) + (uint64_t) tl.c0 * ys + row0 + row;
#pragma unroll 1
        for (uint32_t c = 0; c < (uint32_t) kN; c += kChunkTok) {
          // column c of the accumulator is token 2 c + u, or (both halves in one) token 2 (c % 64) + c / 64
          const uint32_t t0 = uses == 2u ? 2u * c + u : 2u * (c % (kN / 2)) + c / (kN / 2);
          if (t0 >= tl.n) continue;
          uint32_t r[kChunkTok];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
              : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
              : "r"(tmem + ((32u * warp) << 16) + buf * kN + c)
              : "memory");
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if constexpr (EPI == kGatedMean) {
            // each thread gates its row's sums into the exchange ([token of the chunk][tile row]); then thread e adds value
            // e % per's streams in order for the tokens e / per, e / per + 128 / per, ...
            float* ex = (float*) (smem + kExAt<T, EPI>);
            const uint32_t d0 = tl.rt * a.per, st = row / a.per, d = d0 + (row - st * a.per);
            const bool mine = st < a.hc && d < a.dim;
#pragma unroll
            for (uint32_t i = 0; i < kChunkTok; i++) {
              float p = 0.0f;
              if (mine && t0 + 2u * i < tl.n)
                p = mul_rn(a.xn[((uint64_t) (tl.c0 + t0 + 2u * i) * a.hc + st) * a.dim + d], sigmoidf(__uint_as_float(r[i])));
              ex[i * kM + row] = p;
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * kWarp) : "memory");
            const uint32_t j = row % a.per, tg = row / a.per, groups = (uint32_t) kM / a.per;
            if (tg < groups && d0 + j < a.dim) {
              for (uint32_t i = tg; i < kChunkTok && t0 + 2u * i < tl.n; i += groups) {
                const uint32_t tk = tl.c0 + t0 + 2u * i;
                float sum = 0.0f;
                for (uint32_t q = 0; q < a.hc; q++) sum = __fadd_rn(sum, ex[i * kM + q * a.per + j]);
                const float v = __fdiv_rn(sum, (float) a.hc);
                a.out[(uint64_t) tk * a.dim + d0 + j] = v;
                if (a.x16_out) x16_store(a.x16_out, a.overflow, a.out_row0 + tk, d0 + j, a.dim, v);
              }
            }
            asm volatile("bar.sync 2, %0;" ::"n"(kEpiWarps * kWarp) : "memory");  // (the next tokens reuse ex)
          } else if (live) {
            float* y = y0 + (uint64_t) t0 * ys;
#pragma unroll
            for (uint32_t i = 0; i < kChunkTok; i++) {
              if (t0 + 2u * i < tl.n) {
                float v = mul_rn(__uint_as_float(r[i]), scale);
                if constexpr (EPI == kSilu) {
                  v = siluf(v);
                  x16_store(a.x16_out, a.overflow, tl.c0 + t0 + 2u * i, row0 + row, a.rows, v);
                }
                *y = v;
              }
              y += 2u * (uint64_t) ys;
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(&sh.empty_acc[buf]);
      }
    }
    if (!ok) sh.fail = 1;
  }
  // ================= common exit =================
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == (uint32_t) kIssuerWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
  if (tid == 0 && sh.fail) atomicOr(a.status, kWaitRanOut);
}

uint32_t* status_word() {
  static uint32_t* at[64];
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return nullptr;
  if (!at[d]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_status) != cudaSuccess) return nullptr;
    at[d] = (uint32_t*) p;
  }
  return at[d];
}

// the driver's tensor-map encoder, looked up once (no link against the driver library)
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encoder() {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiled) p;
  }
  return fn;
}

// the tiled x16 of `tiles` token tiles (rows xts values long) as [K fragment][token tile][two tokens][value in
// fragment]; a box: a K step's fragments of `tok` tokens
bool x16_map(const void* x16, uint32_t tiles, uint32_t xts, uint32_t tok, CUtensorMap* tm) {
  const EncodeTiled enc = encoder();
  if (!enc) return false;
  const cuuint64_t dims[4] = {2 * MM_TILE, MM_TILE / 2, tiles, xts / MM_TILE};
  const cuuint64_t strides[3] = {MM_TILE * 4, (cuuint64_t) MM_TILE * xts * 2, MM_TILE * MM_TILE * 2};
  const cuuint32_t box[4] = {2 * MM_TILE, MM_TILE / 2, tok / MM_TILE, kSubs}, unit[4] = {1, 1, 1, 1};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(x16), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// n_mat matrices of rows x row_bytes, `bytes` apart: a box is the block of a row tile's rows
bool raw_map(const void* w, uint64_t row_bytes, uint32_t rows, uint32_t n_mat, uint64_t bytes, uint32_t window, CUtensorMap* tm) {
  const EncodeTiled enc = encoder();
  if (!enc || ((uintptr_t) w | row_bytes | bytes) % 16 || row_bytes >> 32 || bytes >> 40 || row_bytes < window) return false;
  const cuuint64_t dims[3] = {row_bytes, rows, n_mat}, strides[2] = {row_bytes, bytes};
  const cuuint32_t box[3] = {window, kM, 1}, unit[3] = {1, 1, 1};
  return enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(w), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <uint32_t T, uint32_t EPI = kStore>
bool launch(Args a, uint32_t n_mat, uint32_t max_cnt, cudaStream_t s) {
  constexpr int kBytes = (int) kSmem<T, EPI>;
  static_assert(kBytes + grid_smem_bytes<T>() + (int) sizeof(Shared) + 64 <= 227 * 1024, "a block's shared memory");
  static_assert(phases_known(kRawStages<T>, kRawK<T> / kStep, Fmt<T>::values > 128 ? Fmt<T>::values / kStep : 2), "a producer's wait on a raw slot");
  a.status = status_word();
  if (!a.status) return false;
  int sms = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  a.row_tiles = EPI == kGatedMean ? parts_of(a.dim, a.per) : parts_of(a.rows, kM);
  a.row_tiles1 = a.w1 ? parts_of(a.rows1, kM) : 0u;
  static bool sized[64] = {};  // (one record a template instance, one flag a device)
  if (!allow_dynamic_smem(mm_tc_kernel<T, EPI>, kBytes, sized)) return false;
  alignas(64) Maps maps;
  memset(&maps, 0, sizeof maps);
  const uint64_t row_bytes = (uint64_t) (a.cols / Fmt<T>::values) * Fmt<T>::bytes;
  if (EPI != kGatedMean && (!a.wt || (a.base && a.bytes >= a.rows * row_bytes)))
    a.raw_map = a.wt ? raw_map(a.base, row_bytes, a.rows, a.n_base, a.bytes, kWindow<T>, &maps.raw)
                     : raw_map(a.w, row_bytes, a.rows, 1, a.rows * row_bytes, kWindow<T>, &maps.raw) &&
                           (!a.w1 || raw_map(a.w1, row_bytes, a.rows1, 1, a.rows1 * row_bytes, kWindow<T>, &maps.raw1));
  const uint64_t row_tiles = (uint64_t) a.row_tiles + a.row_tiles1;  // (of one matrix or two)
  if (a.wt) {
    a.span = max_cnt < kMaxSpan ? whole16(max_cnt) : kMaxSpan;
    // (where in x16 a matrix's tokens lie is on the device: the maps reach as far as its 32-bit offsets do, and a box has no
    // tile but the tokens')
    a.use_tma = 1;
    for (uint32_t t = 0; t < a.span / MM_TILE && a.use_tma; t++)
      if (!x16_map(a.x16, (uint32_t) (0xFFFFFFFFull / (MM_TILE * (uint64_t) a.xts)) + 1u + MM_MAX_TOKENS / MM_TILE, a.xts, (t + 1u) * MM_TILE, &maps.map[t])) a.use_tma = 0;
    for (uint32_t m0 = 0; m0 < n_mat; m0 += kMaxMats) {
      Args c = a;
      c.n_mat = n_mat - m0 < kMaxMats ? n_mat - m0 : kMaxMats;
      c.wt += m0, c.cnt += m0, c.xoff += m0, c.yoff += m0;
      const uint64_t tiles = (uint64_t) a.row_tiles * c.n_mat * parts_of(max_cnt, a.span);
      const dim3 grid((unsigned) (tiles < (uint64_t) sms ? tiles : (uint64_t) sms));
      if (launch_dependent(mm_tc_kernel<T, EPI>, grid, dim3(kThreads), kBytes, s, c, maps) != cudaSuccess) return false;
    }
    return true;
  }
  // tokens a tile: the split with the least estimated time - rounds of tiles over the SMs times a K step's cycles, which are
  // the decoders' or the products' (2 a token, and reading their operands), whichever is more
  uint64_t best = 0;
  // (of the gated mean too, although its ring has three slots of 256 tokens, not four: up to 192 a tile Q8_0 4 x 2560 x 512, 200 tokens,
  // took 74.7 us and 2 x 4096 x 2048, 500 tokens, 138.4, against 67.8 and 128.3; 4 x 7168 x 1536 at 2048 2117 and 2124)
  for (uint32_t cols = parts_of(a.n, kMaxSpan); cols <= parts_of(a.n, MM_TILE); cols++) {
    const uint32_t tok = whole16(parts_of(a.n, cols)), step = 60u + 9u * tok / 4u;
    const uint64_t rounds = (row_tiles * parts_of(a.n, tok) + (uint32_t) sms - 1u) / (uint32_t) sms;
    const uint64_t cost = rounds * (step > 320u ? step : 320u);
    if (!best || cost < best) best = cost, a.span = tok;
  }
  a.use_tma = x16_map(a.x16, parts_of(a.n, MM_TILE), a.xts, a.span, &maps.map[0]) ? 1u : 0u, a.n_mat = 1;
  const uint64_t tiles = row_tiles * parts_of(a.n, a.span);
  if (tiles > 0xFFFFFFFFull) return false;
  const dim3 grid((unsigned) (tiles < (uint64_t) sms ? tiles : (uint64_t) sms));
  return launch_dependent(mm_tc_kernel<T, EPI>, grid, dim3(kThreads), kBytes, s, a, maps) == cudaSuccess;
}

}  // namespace

bool shape_ok(uint32_t type, uint32_t rows, uint32_t cols) {
  const OsmosQTypeInfo* t = qtype_row(type);
  return t && rows && rows % MM_TILE == 0 && cols && cols % 128 == 0 && cols % t->values == 0;
}

namespace {
template <uint32_t EPI>
bool run_with(uint32_t type, const Args& a, void* stream) {
#define CASE(T) return launch<T, EPI>(a, 1, a.n, stream_of(stream));
  OSMOS_SWITCH_QUANT(type, CASE, return false)
#undef CASE
}
}  // namespace

bool run(uint32_t type, const void* w, uint32_t rows, uint32_t cols, const void* x16, uint32_t n, float* y, uint32_t ys,
         float scale, void* stream, bool early) {
  if (!w || !x16 || !y || !n || n > MM_MAX_TOKENS || !shape_ok(type, rows, cols) || (n > 1 && ys < rows)) return false;
  if ((uintptr_t) x16 & 15u) return false;
  Args a{};
  a.w = (const uint8_t*) w, a.x16 = (const __half*) x16, a.y = y, a.rows = rows, a.cols = cols, a.n = n, a.xts = cols;
  a.ys = ys, a.scale = scale, a.early = early ? 1u : 0u;
  return run_with<kStore>(type, a, stream);
}

// two matrices of a type and width over the same tokens in one launch, each the bits `run` gives it alone; both have been checked
bool run_pair(uint32_t type, const void* w0, uint32_t rows0, float* y0, uint32_t ys0, float s0, const void* w1, uint32_t rows1, float* y1,
              uint32_t ys1, float s1, uint32_t cols, const void* x16, uint32_t n, void* stream, bool early) {
  Args a{};
  a.w = (const uint8_t*) w0, a.x16 = (const __half*) x16, a.y = y0, a.rows = rows0, a.cols = cols, a.n = n, a.xts = cols;
  a.ys = ys0, a.scale = s0, a.early = early ? 1u : 0u;
  a.w1 = (const uint8_t*) w1, a.y1 = y1, a.rows1 = rows1, a.ys1 = ys1, a.scale1 = s1;
  return run_with<kStore>(type, a, stream);
}

bool run_silu(uint32_t type, const void* w, uint32_t rows, uint32_t cols, const void* x16, uint32_t n, float* y, uint32_t ys,
              float scale, void* x16_out, int32_t* overflow, void* stream) {
  if (!w || !x16 || !y || !x16_out || x16_out == x16 || !overflow || !n || n > MM_SILU_MAX_TOKENS ||
      !shape_ok(type, rows, cols) || (n > 1 && ys < rows) || (((uintptr_t) x16 | (uintptr_t) x16_out) & 15u))
    return false;
  Args a{};
  a.w = (const uint8_t*) w, a.x16 = (const __half*) x16, a.y = y, a.rows = rows, a.cols = cols, a.n = n, a.xts = cols;
  a.ys = ys, a.scale = scale, a.x16_out = (__half*) x16_out, a.overflow = overflow;
  return run_with<kSilu>(type, a, stream);
}

bool run_gated_mean(uint32_t type, const void* w, uint32_t hc, uint32_t dim, uint32_t cols, const void* x16, uint32_t n,
                    const float* xn, float* out, void* out16, uint32_t row0, int32_t* overflow, void* stream) {
  if (!w || !x16 || !xn || !out || out16 == x16 || (out16 && !overflow) || !n || n > MM_MAX_TOKENS || !hc ||
      hc > MM_GATED_MEAN_MAX_HC || !dim || dim % MM_TILE || (uint64_t) hc * dim > 0xFFFFFFFFull ||
      !shape_ok(type, hc * dim, cols) || ((uintptr_t) x16 & 15u))
    return false;
  Args a{};
  a.w = (const uint8_t*) w, a.x16 = (const __half*) x16, a.rows = hc * dim, a.cols = cols, a.n = n, a.xts = cols;
  a.scale = 1.0f, a.x16_out = (__half*) out16, a.overflow = overflow, a.xn = xn, a.out = out;
  a.hc = hc, a.dim = dim, a.out_row0 = row0;
  a.per = ((uint32_t) kM / hc) & ~(uint32_t) (MM_TILE - 1);  // whole tiles of 16 values: 128, 64, 32, 32, 16, ... for 1 - 8 streams
  return run_with<kGatedMean>(type, a, stream);
}

}  // namespace mm_tc
}  // namespace osmos

using namespace osmos;

extern "C" bool mm_known(uint32_t type) { return qtype_row(type) != nullptr; }
extern "C" bool mm_fits(uint32_t type, uint32_t rows, uint32_t cols) { return mm_tc::shape_ok(type, rows, cols); }
extern "C" uint32_t mm_col_tiles(uint32_t type, uint32_t n) {
  if (!qtype_row(type)) return 0;
  return n <= (uint32_t) mm_tc::kN ? 1u : n <= 2u * mm_tc::kN ? 2u : (uint32_t) mm_tc::kMaxAcc;
}
extern "C" uint32_t mm_status(void) {
  uint32_t* at = mm_tc::status_word();
  if (!at) return 0x80000000u;
  uint32_t v = 0, zero = 0;
  if (cudaMemcpy(&v, at, sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess) return 0x80000000u;
  cudaMemcpy(at, &zero, sizeof zero, cudaMemcpyHostToDevice);
  return v | fp4_tc::read_status();  // (the block-scaled FP4 product's record beside the f16 product's)
}

extern "C" bool mm_run(uint32_t type, const void* w, uint32_t rows, uint32_t cols, const void* x16, uint32_t n, float* y,
                       uint32_t ys, void* stream) {
  return mm_tc::run(type, w, rows, cols, x16, n, y, ys, 1.0f, stream);
}

extern "C" bool mm_run_silu(uint32_t type, const void* w, uint32_t rows, uint32_t cols, const void* x16, uint32_t n,
                            float* y, uint32_t ys, float scale, void* x16_out, int32_t* overflow, void* stream) {
  return mm_tc::run_silu(type, w, rows, cols, x16, n, y, ys, scale, x16_out, overflow, stream);
}

extern "C" bool mm_run_gated_mean(uint32_t type, const void* w, uint32_t hc, uint32_t dim, uint32_t cols, const void* x16,
                                  uint32_t n, const float* xn, float* out, void* out16, uint32_t row0, int32_t* overflow,
                                  void* stream) {
  return mm_tc::run_gated_mean(type, w, hc, dim, cols, x16, n, xn, out, out16, row0, overflow, stream);
}

extern "C" bool mm_run2(uint32_t type, const void* w0, uint32_t rows0, float* y0, uint32_t ys0, const void* w1,
                        uint32_t rows1, float* y1, uint32_t ys1, uint32_t cols, const void* x16, uint32_t n, void* stream) {
  if (!w0 || !w1 || !y0 || !y1 || !x16 || !n || n > MM_MAX_TOKENS || !mm_tc::shape_ok(type, rows0, cols) ||
      !mm_tc::shape_ok(type, rows1, cols) || (n > 1 && (ys0 < rows0 || ys1 < rows1)) || ((uintptr_t) x16 & 15u))
    return false;  // (decided for both before either is queued)
  return mm_tc::run_pair(type, w0, rows0, y0, ys0, 1.0f, w1, rows1, y1, ys1, 1.0f, cols, x16, n, stream, false);
}

extern "C" bool mm_tokens_scaled(uint32_t type, const void* w0, uint32_t rows0, float* y0, uint32_t ys0, float s0,
                                 const void* w1, uint32_t rows1, float* y1, uint32_t ys1, float s1, uint32_t cols,
                                 const float* x, uint32_t xs, uint32_t n, void* x16, int32_t* overflow, bool ready,
                                 void* stream) {
  if (!w0 || !y0 || !x || !x16 || !overflow || !n || !mm_tc::shape_ok(type, rows0, cols) || (n > 1 && (xs < cols || ys0 < rows0)))
    return false;
  if (w1 && (!y1 || !mm_tc::shape_ok(type, rows1, cols) || (n > 1 && ys1 < rows1))) return false;
  if ((uintptr_t) x16 & 15u) return false;
  for (uint32_t t0 = 0; t0 < n; t0 += MM_MAX_TOKENS) {  // MM_MAX_TOKENS a time through the one x16
    const uint32_t c = n - t0 < MM_MAX_TOKENS ? n - t0 : MM_MAX_TOKENS;
    const bool convert = !(ready && n <= MM_MAX_TOKENS);
    if (convert && !mm_x16(x + (uint64_t) t0 * xs, xs, c, cols, x16, overflow, stream)) return false;
    float* const to0 = y0 + (uint64_t) t0 * ys0;
    if (w1 ? !mm_tc::run_pair(type, w0, rows0, to0, ys0, s0, w1, rows1, y1 + (uint64_t) t0 * ys1, ys1, s1, cols, x16, c, stream, convert)
           : !mm_tc::run(type, w0, rows0, cols, x16, c, to0, ys0, s0, stream, convert))
      return false;
  }
  return true;
}

extern "C" bool mm_tokens(uint32_t type, const void* w0, uint32_t rows0, float* y0, uint32_t ys0, const void* w1,
                          uint32_t rows1, float* y1, uint32_t ys1, uint32_t cols, const float* x, uint32_t xs, uint32_t n,
                          void* x16, int32_t* overflow, bool ready, void* stream) {
  return mm_tokens_scaled(type, w0, rows0, y0, ys0, 1.0f, w1, rows1, y1, ys1, 1.0f, cols, x, xs, n, x16, overflow, ready, stream);
}

extern "C" bool mm_group_of(uint32_t type, const void* base, uint64_t bytes, uint32_t n_base, const void* const* w, const int32_t* cnt, uint32_t n_mat,
                            uint32_t max_cnt, uint32_t rows, uint32_t cols, const void* x16, const uint32_t* xoff, uint32_t xts, float* y,
                            const uint32_t* yoff, uint32_t ys, void* stream) {
  if (!w || !cnt || !x16 || !xoff || !y || !yoff || !n_mat || n_mat > 65535 || !max_cnt || max_cnt > MM_MAX_TOKENS ||
      !mm_tc::shape_ok(type, rows, cols) || xts < cols || xts % MM_TILE || ys < rows || ((uintptr_t) x16 & 15u))
    return false;
  mm_tc::Args a{};
  a.wt = (const uint8_t* const*) w, a.cnt = cnt, a.xoff = xoff, a.yoff = yoff, a.x16 = (const __half*) x16, a.y = y;
  a.rows = rows, a.cols = cols, a.xts = xts, a.ys = ys, a.scale = 1.0f;
  a.base = (const uint8_t*) base, a.bytes = bytes, a.n_base = n_base;
#define CASE(T) return mm_tc::launch<T>(a, n_mat, max_cnt, stream_of(stream));
  OSMOS_SWITCH_QUANT(type, CASE, return false)
#undef CASE
}

extern "C" bool mm_group(uint32_t type, const void* const* w, const int32_t* cnt, uint32_t n_mat, uint32_t max_cnt,
                         uint32_t rows, uint32_t cols, const void* x16, const uint32_t* xoff, uint32_t xts, float* y,
                         const uint32_t* yoff, uint32_t ys, void* stream) {
  return mm_group_of(type, nullptr, 0, 0, w, cnt, n_mat, max_cnt, rows, cols, x16, xoff, xts, y, yoff, ys, stream);
}
