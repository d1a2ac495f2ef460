// The F32-activation matvec (mv_run / mv_strided up to 8 tokens, mv_group, mv_group_tok) for the types whose 8-value
// chunks pair up on the same bytes: Q4_0, Q8_0, Q4_K, Q5_K, Q6_K, IQ4_XS, MXFP4. The sums are mv.cu's: of a row, lane l
// of 32 runs one fmaf chain over chunks l, l + 32, ... in value order, then the xor tree 16, 8, 4, 2, 1.
//
// What differs from mv_staged.cu is who computes a lane: a thread runs TWO of a row's 32 lanes side by side, lanes A and
// B whose chunks are the low and the high nibbles of the same eight bytes (of Q8_0: two chunks of one block). So a
// chunk's bytes, its scale fields and their unpacking are read and done once for 16 values, and every F32 operation of the two
// chains - the code made a float, its scale, the fmaf into the sum - is one packed instruction (add / mul / fma
// .rn.f32x2: element by element the same IEEE operation, so the same bits). Sixteen threads are a row, a warp two rows
// (RT of them a thread: 2 RT a warp), each with up to 8 tokens' chains. The two rows sit in even and odd lanes: a 16-byte
// read of x whose neighbouring lanes ask for the same piece takes two passes of shared memory, one whose halves do takes
// four, like 32 different pieces (measured: 2.0 against 4.0 cycles a warp).
//
// Bound by instruction issue at one token - 6.8 instructions a value all told (Q6_K 98304 x 2048, 60.3 us: 68 % of the issue slots,
// the integer pipe 66 %, shared memory 28 %, DRAM 34 %: what is left is four warps a scheduler with a chain each, and 9 %
// of the launch before the first slot and after the last) - and from three tokens on by x's reads. Measured, against a lane a
// thread (mv_staged.cu): 49152 x 2048 at one token Q6_K 41.1 -> 29.5 us (2.8 TB/s), Q5_K 45.1 -> 33.4, Q4_K 39.6 -> 29.9, IQ4_XS
// 42.1 -> 27.7; at eight tokens 80-85 -> 64-69; Q4_K 2048 x 7168 at five 22.6 -> 12.0; 1536 x 4096 MXFP4 matrices of 64 experts
// at 64 picks 239 -> 111 us; without MXFP4's table of pairs 128 experts top-4, 32 tokens, 620 -> 510 us the layer.
//
// A warp owns a ring of slots; a slot holds the same run of up to 8 256-value stretches of its 2 RT rows, a bulk copy a
// row of the 16-byte pieces around the row's bytes - so a row may start anywhere (Q6_K's 210-byte blocks: rows are
// multiples of 16 bytes only at every eighth width) and the ring does not grow with the row. x lies in shared memory
// in the order the threads read it: [256-value stretch][values 2 q, 2 q + 1 of the chunk][pair], a 16-byte piece (A's two
// values and B's, interleaved) each.
#include "mv_pair_api.h"

#include "decode.cuh"
#include "dispatch.cuh"
#include "mv_room.h"
#include "packed.cuh"
#include "tma.cuh"

namespace osmos {
namespace mvp {
namespace {

using namespace tma;

constexpr int kWarps = 16, kThreads = kWarps * kWarp;
constexpr uint32_t kMaxSlots = 4;
// 256-value stretches of a row a slot holds at most: with two rows a thread half as many (a slot's bytes stay)
template <int RT> constexpr uint32_t kSegOf = RT == 1 ? 8u : 4u;
constexpr uint32_t kMaxTok = 8;

__device__ uint32_t g_status;

struct Args {
  const uint8_t* w;
  const float* x;
  float* y;
  uint32_t rows, cols, xs, ys, n_tok;
  uint32_t seg;       // stretches a slot holds of a row
  uint32_t fit;       // tokens whose x a pass holds
  uint32_t smem;      // dynamic shared memory, bytes: x of a pass, then the rings
  uint32_t* status;
  // grouped forms: a block finds its entry and its part of that entry's rows (find_entry)
  const uint8_t* const* wt;
  const int32_t *cnt, *xrow;
  uint32_t n_entries, x_mat, x_div;
  uint32_t parts;  // blocks an entry
  uint32_t wave;   // blocks that the live entries are dealt anew over when they have fewer; 0: a block has the entry of its place
};

// parts of an entry's units, `most` at most: as few as leave a warp of the largest no more units than that many would
__host__ __device__ inline uint32_t even_parts(uint32_t units, uint32_t most) {
  const uint32_t rounds = (units + kWarps * most - 1) / (kWarps * most);
  return (units + kWarps * rounds - 1) / (kWarps * rounds);
}

// the eight bytes sh / 8 bytes into the aligned word at `al`, out of it and the two after it
__device__ __forceinline__ uint2 lds_8_bytes(uint32_t al, uint32_t sh) {
  const uint32_t r0 = lds32(al), r1 = lds32(al + 4), r2 = lds32(al + 8);
  return make_uint2(__funnelshift_r(r0, r1, sh), __funnelshift_r(r1, r2, sh));
}
__device__ __forceinline__ uint2 low_nibbles(uint2 q) { return make_uint2(q.x & kLow4, q.y & kLow4); }
__device__ __forceinline__ uint2 high_nibbles(uint2 q) { return make_uint2((q.x >> 4) & kLow4, (q.y >> 4) & kLow4); }

// ---- the types: what of a 256-value stretch thread p (0 .. 15) of a row reads --------------------------------------------
// kD: the distance of the pair's lanes (B = A + kD); lane(p): lane A. values(): the eight (A, B) values of the stretch at
// shared address `at` - the bits chunk_values gives (each product and difference rounded once, in its order).
template <uint32_t T> struct Pair;

template <uint32_t T> __host__ __device__ constexpr uint32_t stretch_bytes() { return Fmt<T>::bytes * (256 / Fmt<T>::values); }
// types whose rows and stretches are whole 16-byte pieces wherever a matrix starts on one (the others: Q6_K's 210 bytes, and
// the 136 of MXFP4 and IQ4_XS, where an odd stretch starts 8 bytes into a piece)
template <uint32_t T> constexpr bool kWhole = stretch_bytes<T>() % 16 == 0;
// types whose two nibbles go through a table of 256 (low, high) value pairs, two bf16 (the values are exact in it)
template <uint32_t T> constexpr bool kPairTable = (T == QTYPE_IQ4_XS);
constexpr uint32_t kTableBytes = 256u * 128u;  // a copy a lane: every lookup its own bank
struct Table {
  const uint8_t* at;
  uint32_t copy;  // this lane's, 4 lane bytes on
};

// byte j of w as a byte offset into the table (an entry's 32 copies are 128 bytes), this lane's copy
template <int J> __device__ __forceinline__ uint64_t table_pair(uint32_t w, const uint8_t* tbl, uint32_t copy) {
  const uint32_t e = *(const uint32_t*) (tbl + (((J == 0 ? w << 7 : w >> (J ? 8 * J - 7 : 0)) & 0x7F80u) | copy));
  return pack2u(e << 16, e & 0xFFFF0000u);
}
__device__ __forceinline__ void table_pairs(uint2 q, const Table& t, uint64_t* v) {
  v[0] = table_pair<0>(q.x, t.at, t.copy), v[1] = table_pair<1>(q.x, t.at, t.copy), v[2] = table_pair<2>(q.x, t.at, t.copy), v[3] = table_pair<3>(q.x, t.at, t.copy);
  v[4] = table_pair<0>(q.y, t.at, t.copy), v[5] = table_pair<1>(q.y, t.at, t.copy), v[6] = table_pair<2>(q.y, t.at, t.copy), v[7] = table_pair<3>(q.y, t.at, t.copy);
}

// the 32-value blocks: block p / 2 of the stretch's eight, lanes 4 (p / 2) + p % 2 and two on
template <> struct Pair<QTYPE_Q4_0> {
  static constexpr uint32_t kD = 2;
  uint32_t off, sh, doff;  // (a stretch starts on a word: where the bytes lie in theirs is the thread's own)
  __device__ __forceinline__ explicit Pair(uint32_t p) : off((p >> 1) * 18u + 2u + 8u * (p & 1u)), sh(off % 4u * 8u), doff((p >> 1) * 18u) { off &= ~3u; }
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 1) * 4u + (p & 1u); }
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    const uint2 q = lds_8_bytes(at + off, sh);
    const float d = half_value(lds16(at + doff));
    const uint64_t dd = pack2(d, d);
    code_pairs(low_nibbles(q), high_nibbles(q), -32776.0f, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = mul2(dd, v[j]);
  }
};
template <> struct Pair<QTYPE_Q8_0> {
  static constexpr uint32_t kD = 2;
  uint32_t off, sh, doff;
  __device__ __forceinline__ explicit Pair(uint32_t p) : off((p >> 1) * 34u + 2u + 8u * (p & 1u)), sh(off % 4u * 8u), doff((p >> 1) * 34u) { off &= ~3u; }
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 1) * 4u + (p & 1u); }
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    uint2 a = lds_8_bytes(at + off, sh), b = lds_8_bytes(at + off + 16u, sh);
    a.x ^= kTops, a.y ^= kTops, b.x ^= kTops, b.y ^= kTops;
    const float d = half_value(lds16(at + doff));
    const uint64_t dd = pack2(d, d);
    code_pairs(a, b, -32896.0f, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = mul2(dd, v[j]);
  }
};
template <> struct Pair<QTYPE_MXFP4> {
  static constexpr uint32_t kD = 2;
  uint32_t off, sh, eoff;
  __device__ __forceinline__ explicit Pair(uint32_t p) : off((p >> 1) * 17u + 1u + 8u * (p & 1u)), sh(off % 4u * 8u), eoff((p >> 1) * 17u) { off &= ~3u; }
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 1) * 4u + (p & 1u); }
  // An E2M1 code's bits as an F16's sign, exponent's low two bits and mantissa's top one are its value times 2^-14 (a subnormal
  // code is a subnormal F16); to F32 exactly, times 2^(e - 113): one rounding, of the value itself, as decode8's product. Past
  // e = 240 that factor is no F32: half the scale times the doubled code, as there. (Against a table of 256 pairs in shared memory, a copy
  // a lane, which took most of its passes; the scale has to be one addition and a shift for it: with its ranges told apart long rows were
  // slower than the table, 8192 x 4096 at one token 11.2 -> 11.7 us, now 10.2; 49152 x 7168 92.5 -> 95.5, now 82.7.)
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    const uint2 q = lds_8_bytes(at + off, sh);
    const uint32_t e = lds8(at + eoff);
    const bool large = e > 240u;
    const float d = __uint_as_float((e + (large ? 0xFFFFFFFFu : 14u)) << 23);  // (either is a normal F32, whatever e)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const uint32_t w = i ? q.y : q.x;
      const uint32_t lo = ((w << 1) & 0x0E0E0E0Eu) | ((w << 4) & kTops), hi = ((w >> 3) & 0x0E0E0E0Eu) | (w & kTops);
      const uint32_t le = __byte_perm(lo, 0, 0x2404), lp = lo & 0xFF00FF00u, he = __byte_perm(hi, 0, 0x2404), hp = hi & 0xFF00FF00u;
      v[4 * i] = pack2(low_half(le), low_half(he)), v[4 * i + 1] = pack2(low_half(lp), low_half(hp));
      v[4 * i + 2] = pack2(high_half(le), high_half(he)), v[4 * i + 3] = pack2(high_half(lp), high_half(hp));
    }
    const uint64_t dd = pack2(d, d);
    if (large) {
#pragma unroll
      for (int j = 0; j < kChunk; j++) v[j] = mul2(v[j], pack2(32768.0f, 32768.0f));
    }
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = mul2(dd, v[j]);
  }
};
// 256-value blocks from here on (of Q4_K and Q5_K thread p has groups 2 (p / 4) and the next: the low and the high nibbles of
// the same 32 bytes)
template <> struct Pair<QTYPE_IQ4_XS> {
  static constexpr uint32_t kD = 2;
  uint32_t off, so, s4, s2;
  __device__ __forceinline__ explicit Pair(uint32_t p) : off(8u + 8u * p), so(4u + (p >> 2)), s4(4u * ((p >> 1) & 1u)), s2(p & 14u) {}
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 1) * 4u + (p & 1u); }
  static __device__ __forceinline__ float entry(uint32_t n) { return (float) (int) (int8_t) iq4nl4(n); }
  __device__ __forceinline__ void values(uint32_t at, const Table& tbl, uint64_t* v) const {
    const uint2 q = lds64(at + off);
    const uint32_t hd = lds32(at), s = ((lds8(at + so) >> s4) & 0x0Fu) | ((hd >> (16u + s2)) & 3u) << 4;
    const float ds = mul_rn(half_value(hd & 0xFFFFu), __fadd_rn(__uint_as_float(0x4B000000u | s), -8388640.0f));  // d (s - 32)
    const uint64_t dd = pack2(ds, ds);
    table_pairs(q, tbl, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = mul2(dd, v[j]);
  }
};
template <> struct Pair<QTYPE_Q4_K> {
  static constexpr uint32_t kD = 4;
  uint32_t off, s;
  bool upper;
  __device__ __forceinline__ explicit Pair(uint32_t p) : off(16u + 8u * p), s(16u * ((p >> 2) & 1u)), upper(p >= 8u) {}
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 2) * 8u + (p & 3u); }
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    const int4 h = lds128(at);
    const uint2 q = lds64(at + off);
    uint32_t sc, mn;
    k_scales((uint32_t) h.y, (uint32_t) h.z, (uint32_t) h.w, s, upper, sc, mn);
    const float d = half_value((uint32_t) h.x & 0xFFFFu), m = -half_value((uint32_t) h.x >> 16);
    const uint64_t ds = mul2(pack2(d, d), pack2(byte_value<0>(sc), byte_value<1>(sc)));
    const uint64_t dm = mul2(pack2(m, m), pack2(byte_value<0>(mn), byte_value<1>(mn)));  // (minus the minimum)
    code_pairs(low_nibbles(q), high_nibbles(q), -32768.0f, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = add2(mul2(ds, v[j]), dm);
  }
};
template <> struct Pair<QTYPE_Q5_K> {
  static constexpr uint32_t kD = 4;
  uint32_t off, foff, s, b;
  bool upper;
  __device__ __forceinline__ explicit Pair(uint32_t p)
      : off(48u + 8u * p), foff(16u + 8u * (p & 3u)), s(16u * ((p >> 2) & 1u)), b(2u * (p >> 2)), upper(p >= 8u) {}
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return (p >> 2) * 8u + (p & 3u); }
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    const int4 h = lds128(at);
    const uint2 q = lds64(at + off), f = lds64(at + foff);
    uint32_t sc, mn;
    k_scales((uint32_t) h.y, (uint32_t) h.z, (uint32_t) h.w, s, upper, sc, mn);
    const float d = half_value((uint32_t) h.x & 0xFFFFu), m = -half_value((uint32_t) h.x >> 16);
    const uint64_t ds = mul2(pack2(d, d), pack2(byte_value<0>(sc), byte_value<1>(sc)));
    const uint64_t dm = mul2(pack2(m, m), pack2(byte_value<0>(mn), byte_value<1>(mn)));
    // the fifth bits: bit 2 g of a position's byte for A, bit 2 g + 1 for B
    const uint32_t f0 = f.x >> b, f1 = f.y >> b;
    const uint2 a = make_uint2((q.x & kLow4) | (f0 & kOnes) << 4, (q.y & kLow4) | (f1 & kOnes) << 4);
    const uint2 c = make_uint2(((q.x >> 4) & kLow4) | ((f0 << 3) & 0x10101010u), ((q.y >> 4) & kLow4) | ((f1 << 3) & 0x10101010u));
    code_pairs(a, c, -32768.0f, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = add2(mul2(ds, v[j]), dm);
  }
};
template <> struct Pair<QTYPE_Q6_K> {
  // p = 8 h + 4 r + kk: half h of the block, sub-blocks r (A: low nibbles) and r + 2 (B: high ones), chunk kk
  static constexpr uint32_t kD = 8;
  uint32_t off, toff, soff, s;
  __device__ __forceinline__ explicit Pair(uint32_t p)
      : off(64u * (p >> 3) + 8u * (p & 7u)), toff(128u + 32u * (p >> 3) + 8u * (p & 3u)), soff(192u + 8u * (p >> 3) + 2u * ((p >> 2) & 1u) + ((p >> 1) & 1u)),
        s(2u * ((p >> 2) & 1u)) {}
  static __device__ __forceinline__ uint32_t lane(uint32_t p) { return 16u * (p >> 3) + (p & 7u); }
  __device__ __forceinline__ void values(uint32_t at, const Table&, uint64_t* v) const {
    const uint32_t al = at & ~3u, sh = (at & 3u) * 8u;  // (the offsets are whole words)
    const uint2 q = lds_8_bytes(al + off, sh), t = lds_8_bytes(al + toff, sh);
    const float d = half_value(lds16(at + 208u));
    // a signed scale byte: 2^23 + (s ^ 0x80), less 2^23 + 128
    const float sa = __fadd_rn(__uint_as_float(0x4B000080u ^ lds8(at + soff)), -8388736.0f);
    const float sb = __fadd_rn(__uint_as_float(0x4B000080u ^ lds8(at + soff + 4u)), -8388736.0f);
    const uint64_t ds = mul2(pack2(d, d), pack2(sa, sb));
    // the top bit pairs: bits 2 r of a position's byte for A, 2 r + 4 for B
    const uint32_t t0 = t.x >> s, t1 = t.y >> s;
    const uint2 a = make_uint2((q.x & kLow4) | ((t0 << 4) & 0x30303030u), (q.y & kLow4) | ((t1 << 4) & 0x30303030u));
    const uint2 b = make_uint2(((q.x >> 4) & kLow4) | (t0 & 0x30303030u), ((q.y >> 4) & kLow4) | (t1 & 0x30303030u));
    code_pairs(a, b, -32800.0f, v);
#pragma unroll
    for (int j = 0; j < kChunk; j++) v[j] = mul2(ds, v[j]);
  }
};

// ---- the kernel --------------------------------------------------------------------------------------------------------
// A slot's row: the 16-byte pieces around up to `seg` stretches, and a piece more (the last 8-byte read may touch the word
// past the last byte).
// An odd number of 64-byte halves, so that the two rows' reads of a place lie on different halves of the banks.
template <uint32_t T> __host__ __device__ constexpr uint32_t slot_row_bytes(uint32_t cols, uint32_t seg) {
  const uint32_t n = cols / 256u < seg ? cols / 256u : seg;
  const uint32_t need = (n * stretch_bytes<T>() + 15u + 15u) / 16u * 16u + 16u;
  return (need + 63u) / 128u * 128u + 64u;
}
__host__ __device__ inline uint32_t x_bytes(uint32_t tokens, uint32_t cols) { return tokens * cols * 4u; }

template <uint32_t T, int RT>
struct Warp {  // one warp's view of a block's work on one matrix and one pass of tokens
  static constexpr uint32_t kRows = 2 * RT;
  const uint8_t* mat;
  uint8_t* ring;
  uint64_t* full;
  Table table;
  uint32_t lane, p, half, x0, row_bytes, seg_n, nseg, last_n, slots, slot_row, u0, u_hi, rows, cols;
  // the next place of the warp's sequence to be asked for - segment iseg of unit iu, into slot islot - and, for lanes
  // 0 .. kRows - 1, their row of it and its first byte in the matrix; kept by those lanes
  uint32_t iu, iseg, islot = 0, irow;
  uint64_t iat;
  uint32_t slot = 0, phase = 0;  // the next place to be read (a pass reads every place it asks for: both go on where it ends)

  __device__ __forceinline__ void start() {
    iu = u0, iseg = 0, irow = u0 * kRows + lane, iat = (uint64_t) irow * row_bytes;
    if (lane < kRows)
      for (uint32_t s = 0; s < slots; s++) issue();
  }
  __device__ __forceinline__ void issue() {  // lanes 0 .. kRows - 1, a row each
    if (iu >= u_hi) return;
    const bool last = iseg == nseg - 1;
    const uint64_t at = iat + iseg * (seg_n * stretch_bytes<T>());
    uint64_t from = at;
    uint32_t bytes = (last ? last_n : seg_n) * stretch_bytes<T>();
    if constexpr (!kWhole<T>) {
      const uint64_t all = (uint64_t) rows * row_bytes & ~(uint64_t) 15;
      uint64_t to = (at + bytes + 15u) & ~(uint64_t) 15;
      if (to > all) to = all;  // (the matrix's last bytes past a multiple of 16 are brought by the readers)
      from = at & ~(uint64_t) 15, bytes = (uint32_t) (to - from);
    }
    if (irow >= rows) bytes = 0;
    bar_expect(&full[islot], bytes);  // (the barrier counts kRows arrivals)
    if (bytes) bulk_load(ring + (islot * kRows + lane) * slot_row, mat + from, bytes, &full[islot]);
    if (last) iseg = 0, iu += kWarps, irow += kWarps * kRows, iat += (uint64_t) (kWarps * kRows) * row_bytes;
    else iseg++;
    islot = islot + 1 == slots ? 0 : islot + 1;
  }

  // the warp's units for NT tokens, token t's sums to y + t * ys; false when a copy never landed
  template <int NT>
  __device__ __forceinline__ bool run(float* y, uint32_t ys) {
    const Pair<T> pair(p);
    for (uint32_t u = u0; u < u_hi; u += kWarps) {
      const uint32_t r0 = u * kRows + half;  // this thread's rows: r0, r0 + 2, ...
      uint64_t acc[RT][NT];
#pragma unroll
      for (int k = 0; k < RT; k++)
#pragma unroll
        for (int t = 0; t < NT; t++) acc[k][t] = 0;
      uint32_t xa = x0;
      for (uint32_t seg = 0; seg < nseg; seg++) {
        if (!bar_wait_warp(&full[slot], phase)) return false;
        const uint32_t sa = smem_addr(ring) + slot * (kRows * slot_row);
        const uint32_t n = seg == nseg - 1 ? last_n : seg_n;
        uint32_t at[RT];
#pragma unroll
        for (int k = 0; k < RT; k++) {
          at[k] = sa + (2 * k + half) * slot_row;
          if constexpr (!kWhole<T>) at[k] += ((r0 + 2 * k) * row_bytes + seg * seg_n * stretch_bytes<T>()) & 15u;  // where the row's bytes start in a piece
        }
        if constexpr (!kWhole<T>) {
          if (seg == nseg - 1 && u == (rows - 1) / kRows) {
            // the matrix's last bytes, when it is not whole 16-byte pieces: by bytes
            const uint64_t total = (uint64_t) rows * row_bytes;
            const uint32_t tail = (uint32_t) (total & 15u);
            const uint32_t dst = sa + (rows - 1 - u * kRows) * slot_row + (((rows - 1) * row_bytes + seg * seg_n * stretch_bytes<T>()) & 15u) + n * stretch_bytes<T>() - tail;
            for (uint32_t b = lane; b < tail; b += kWarp) {
              const uint32_t v = mat[total - tail + b];
              asm volatile("st.shared.u8 [%0], %1;" ::"r"(dst + b), "r"(v) : "memory");
            }
            __syncwarp();
          }
        }
#pragma unroll(NT <= 2 ? 2 : 1)
        for (uint32_t it = 0; it < n; it++, xa += 1024u) {
          uint64_t v[RT][kChunk];
#pragma unroll
          for (int k = 0; k < RT; k++) pair.values(at[k] + it * stretch_bytes<T>(), table, v[k]);
#pragma unroll
          for (int t = 0; t < NT; t++) {
#pragma unroll
            for (int c = 0; c < 4; c++) {
              uint64_t xl, xh;
              asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(xl), "=l"(xh) : "r"(xa + t * (cols * 4u) + c * 256u));
#pragma unroll
              for (int k = 0; k < RT; k++) acc[k][t] = fma2(v[k][2 * c + 1], xh, fma2(v[k][2 * c], xl, acc[k][t]));
            }
          }
        }
        if (++slot == slots) slot = 0, phase ^= 1u;
        __syncwarp();  // every lane is done reading the slot: refill it
        if (lane < kRows) {
          fence_async_smem();
          issue();
        }
      }
#pragma unroll
      for (int k = 0; k < RT; k++)
#pragma unroll
        for (int t = 0; t < NT; t++) {
          const float s = tree(acc[k][t]);
          if (p == 0 && r0 + 2 * k < rows) y[(uint64_t) t * ys + r0 + 2 * k] = s;
        }
    }
    return true;
  }

  // the xor tree over the row's 32 lanes: lane A's index is p's bits with a zero put in at kD, and p the warp lane's without its
  // lowest bit - so a step past kD is a shuffle at its own distance for both sums, the step kD the thread's own two, a step
  // below it a shuffle of the one left at twice its distance
  static __device__ __forceinline__ float tree(uint64_t v) {
#pragma unroll
    for (int o = 16; o > (int) Pair<T>::kD; o >>= 1) v = add2(v, __shfl_xor_sync(0xFFFFFFFFu, v, o, kWarp));
    float a, b;
    unpack2(v, a, b);
    float s = __fadd_rn(a, b);
#pragma unroll
    for (int o = (int) Pair<T>::kD / 2; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xFFFFFFFFu, s, 2 * o, kWarp));
    return s;
  }
};

// a block's share of a matrix that does not start on 16 bytes: mv.cu's sums straight from global memory, a row a warp, a token
// at a time. (By value: with the kernel's arguments taken by reference every thread of the kernel copied them to its stack first -
// 12 Q4_K entries of 2048 x 512 at a token each 15.1 us, 12.7 so.)
template <uint32_t T>
__device__ __noinline__ void rows_in_place(const uint8_t* mat, uint32_t row_bytes, uint32_t cols, uint32_t lo, uint32_t hi, const float* x, uint32_t xs,
                                           float* y, uint32_t ys, uint32_t live) {
  const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp;
  for (uint32_t r = lo + warp; r < hi; r += kWarps)
    for (uint32_t t = 0; t < live; t++) {
      float s = 0.0f;
      for (uint32_t c = lane; c < cols / kChunk; c += kWarp) {
        float v[kChunk];
        decode8<T>(mat + (uint64_t) r * row_bytes + (c / Fmt<T>::chunks) * Fmt<T>::bytes, (int) (c % Fmt<T>::chunks), v, Grids{});
        const float* xc = x + (uint64_t) t * xs + c * kChunk;
#pragma unroll
        for (int j = 0; j < kChunk; j++) s = __fmaf_rn(v[j], xc[j], s);
      }
      s = xor_tree<kWarp>(s);
      if (lane == 0) y[(uint64_t) t * ys + r] = s;
    }
}

// A grouped launch's block finds its work. The blocks go to the entries that have tokens, `parts` to each in turn; where the live
// ones are so few that this leaves SMs idle - the host knows how many entries there are, not how many have tokens - a wave of
// blocks is dealt to them anew, down to a unit a warp (four live of 64, one token, Q6_K 2048 x 7168: 71.6 us without, 21.9 so; the
// kernels before this one 37). Every thread of the block calls it; false: a block too many. The look through the counts is two
// meetings of the block's warps (128 live of 128, Q4_K 1536 x 4096: 251.5 us without, 258 so): not for few entries, nor for more than
// the block has threads.
struct Work {
  const uint8_t* mat;
  uint32_t m, part, parts;
  int32_t cnt, xrow;  // (by token)
};
__device__ __forceinline__ bool find_entry(const Args& a, uint32_t units, Work& f) {
  f.parts = a.parts;
  if (a.wave) {
    __shared__ uint32_t s_live[kWarps];
    __shared__ Work s_found;
    const uint32_t tid = threadIdx.x, lane = tid % kWarp, warp = tid / kWarp;
    Work mine{nullptr, tid, 0, 0, 0, 0};
    if (tid < a.n_entries) mine.cnt = a.cnt[tid], mine.xrow = a.xrow[tid], mine.mat = a.wt[tid];  // (one trip for all the tables)
    const uint32_t on = __ballot_sync(0xFFFFFFFFu, mine.cnt > 0);
    if (lane == 0) s_live[warp] = __popc(on);
    __syncthreads();
    uint32_t live = 0, before = 0;
#pragma unroll
    for (uint32_t w = 0; w < (uint32_t) kWarps; w++) {
      if (w == warp) before = live;
      live += s_live[w];
    }
    uint32_t parts = a.parts;
    if (live && live * parts < a.wave) {
      const uint32_t most = units / kWarps, each = a.wave / live, to = each < most ? each : most;
      if (to > parts) parts = even_parts(units, to);
    }
    const uint32_t m = blockIdx.x / parts;
    if (m >= live) return false;
    if (mine.cnt > 0 && before + __popc(on & ((1u << lane) - 1u)) == m) s_found = mine;
    __syncthreads();
    f = s_found;
    f.parts = parts, f.part = blockIdx.x - m * parts;
    return true;
  }
  f.m = blockIdx.x / a.parts, f.part = blockIdx.x - f.m * a.parts, f.mat = a.wt[f.m], f.cnt = 1, f.xrow = 0;
  if (a.cnt) f.cnt = a.cnt[f.m], f.xrow = a.xrow[f.m];
  return f.cnt > 0;
}

template <uint32_t T, int RT, bool GROUP>
__global__ void __launch_bounds__(kThreads, 1) mv_pair_kernel(const Args a) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) uint32_t table[kPairTable<T> ? kTableBytes / 4 : 4];
  __shared__ __align__(8) uint64_t full[kWarps][kMaxSlots];
  const uint32_t tid = threadIdx.x, warp = tid / kWarp;
  Warp<T, RT> me;
  const uint32_t stretches = a.cols / 256u;
  me.lane = tid % kWarp, me.p = me.lane >> 1, me.half = me.lane & 1u;
  me.rows = a.rows, me.cols = a.cols, me.row_bytes = stretches * stretch_bytes<T>();
  me.seg_n = a.seg, me.nseg = (stretches + a.seg - 1) / a.seg, me.last_n = stretches - (me.nseg - 1) * a.seg;
  me.slot_row = slot_row_bytes<T>(a.cols, a.seg);
  me.full = full[warp], me.mat = a.w;
  me.table.at = (const uint8_t*) table, me.table.copy = me.lane * 4u;
  const float* xin = a.x;
  float* yout = a.y;
  uint32_t live = a.n_tok;
  [[maybe_unused]] uint32_t part, parts;  // (grouped: the block's share of its entry's rows)
  if (me.lane == 0) {
    for (uint32_t s = 0; s < kMaxSlots; s++) bar_init(&full[warp][s], 2 * RT);
    bar_init_fence();
  }
  __syncwarp();
  if constexpr (GROUP) {
    pdl_wait();  // (a dependent launch: the tables and x may be the output of the kernel ahead)
    pdl_launch_next();
    Work f;
    if (!find_entry(a, (a.rows + 2 * RT - 1) / (2 * RT), f)) return;  // (the whole block)
    part = f.part, parts = f.parts, me.mat = f.mat;
    if (a.cnt) {
      const uint64_t r0 = (uint64_t) f.xrow;
      xin = a.x + r0 * a.xs, yout = a.y + r0 * a.ys, live = (uint32_t) f.cnt < a.n_tok ? (uint32_t) f.cnt : a.n_tok;
    } else {
      xin = a.x + (uint64_t) (f.m / a.x_div) * a.x_mat, yout = a.y + (uint64_t) f.m * a.rows, live = 1;
    }
    if ((uintptr_t) me.mat & 15u) {  // such a matrix cannot be copied in bulk: read where it lies
      if (((uintptr_t) me.mat & 1u) && T != QTYPE_MXFP4) {  // (but for MXFP4's bytes a block is read by halves: reported, its rows left alone)
        if (tid == 0) atomicOr(a.status, 2u);
        return;
      }
      rows_in_place<T>(me.mat, me.row_bytes, a.cols, (uint32_t) ((uint64_t) part * a.rows / parts), (uint32_t) ((uint64_t) (part + 1) * a.rows / parts),
                       xin, a.xs, yout, a.ys, live);
      return;
    }
  }
  const uint32_t units = (a.rows + 2 * RT - 1) / (2 * RT);
  if constexpr (GROUP) me.u0 = (uint32_t) ((uint64_t) part * units / parts) + warp, me.u_hi = (uint32_t) ((uint64_t) (part + 1) * units / parts);
  else me.u0 = (uint32_t) ((uint64_t) blockIdx.x * units / gridDim.x) + warp, me.u_hi = (uint32_t) ((uint64_t) (blockIdx.x + 1) * units / gridDim.x);
  // the tokens in as few passes as their x allows, evenly; the rings take the rest of the block's shared memory
  const uint32_t passes = (live + a.fit - 1) / a.fit, per = (live + passes - 1) / passes;
  const uint32_t ring_off = (x_bytes(per, a.cols) + 127u) & ~127u, slot_bytes = 2 * RT * me.slot_row;
  me.slots = (a.smem - ring_off) / (kWarps * slot_bytes);
  if (me.slots > kMaxSlots) me.slots = kMaxSlots;
  me.ring = smem + ring_off + warp * me.slots * slot_bytes;
  me.start();
  if constexpr (kPairTable<T>) {
    for (uint32_t i = tid; i < 256u * 8u; i += kThreads) {  // a thread four copies of an entry
      const uint32_t e = i >> 3;
      const uint32_t v = __float_as_uint(Pair<T>::entry(e & 15u)) >> 16 | (__float_as_uint(Pair<T>::entry(e >> 4)) & 0xFFFF0000u);
      ((uint4*) table)[i] = make_uint4(v, v, v, v);
    }
  }
  if constexpr (!GROUP) {
    pdl_wait();  // (a dependent launch: x may be the output of the kernel ahead; the weight copies above are not)
    pdl_launch_next();
  }
  bool ok = true;
  for (uint32_t t0 = 0; t0 < live; t0 += per) {
    const uint32_t n = live - t0 < per ? live - t0 : per;
    if (t0) __syncthreads();  // another pass over the rows (its first slots were asked for at the end of the one before)
    // the pass's x, a (token, stretch, pair) a thread at a time
    for (uint32_t i = tid; i < n * stretches * 16u; i += kThreads) {
      const uint32_t p = i & 15u, ts = i >> 4, t = ts / stretches, it = ts - t * stretches;
      const float* from = xin + (uint64_t) (t0 + t) * a.xs + it * 256u + Pair<T>::lane(p) * 8u;
      const float4 a0 = __ldg((const float4*) from), a1 = __ldg((const float4*) from + 1);
      const float4 b0 = __ldg((const float4*) (from + Pair<T>::kD * 8u)), b1 = __ldg((const float4*) (from + Pair<T>::kD * 8u) + 1);
      const uint32_t at = smem_addr(smem) + t * (a.cols * 4u) + it * 1024u + p * 16u;
      sts128(at, a0.x, b0.x, a0.y, b0.y), sts128(at + 256u, a0.z, b0.z, a0.w, b0.w);
      sts128(at + 512u, a1.x, b1.x, a1.y, b1.y), sts128(at + 768u, a1.z, b1.z, a1.w, b1.w);
    }
    __syncthreads();  // x, the table, and the barriers' initialisation
    me.x0 = smem_addr(smem) + me.p * 16u;
    float* y = yout + (uint64_t) t0 * a.ys;
    switch (n) {
      case 1: ok = me.template run<1>(y, a.ys); break;
      case 2: ok = me.template run<2>(y, a.ys); break;
      case 3: ok = me.template run<3>(y, a.ys); break;
      case 4: ok = me.template run<4>(y, a.ys); break;
      case 5: ok = me.template run<5>(y, a.ys); break;
      case 6: ok = me.template run<6>(y, a.ys); break;
      case 7: ok = me.template run<7>(y, a.ys); break;
      default: ok = me.template run<8>(y, a.ys); break;
    }
    if (!__syncthreads_and(ok ? 1 : 0)) break;  // a copy never landed: report it and leave
    if (t0 + per < live) {  // the next pass's copies: every copy of this one has landed and been read
      fence_async_smem();
      me.start();
    }
  }
  if (!ok && me.lane == 0) atomicOr(a.status, 1u);
}

struct Device {
  int sms = 0;
  uint32_t* status = nullptr;
};

const Device* device_info() {
  static Device devs[64];
  int d = -1;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return nullptr;
  if (!devs[d].status) {
    void* at = nullptr;
    int sms = 0;
    if (cudaGetSymbolAddress(&at, g_status) != cudaSuccess || !at) return nullptr;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d) != cudaSuccess || sms <= 0) return nullptr;
    devs[d].sms = sms, devs[d].status = (uint32_t*) at;
  }
  return &devs[d];
}

template <uint32_t T, int RT, bool GROUP>
int launch(const Request& r, const Device* dev, cudaStream_t s) {
  constexpr uint32_t kLimit = 225u * 1024u - (kPairTable<T> ? kTableBytes : 0u);
  Args a{};
  a.w = (const uint8_t*) r.w, a.x = r.x, a.y = r.y, a.rows = r.rows, a.cols = r.cols, a.xs = r.xs, a.ys = r.ys, a.n_tok = r.n_tok;
  a.status = dev->status;
  a.wt = (const uint8_t* const*) r.wt, a.cnt = r.cnt, a.xrow = r.xrow, a.x_mat = r.x_mat, a.x_div = r.x_div;
  // the tokens a pass holds beside rings of two slots; shorter slots where they save a pass over the weights (4096 x 4096
  // MXFP4, 8 tokens: 26.9 us in two passes of slots of eight stretches)
  const mv_room::Passes room = mv_room::pair_passes(kLimit, kSegOf<RT>, kMaxTok, r.n_tok, r.cols,
                                                    [&](uint32_t seg) { return 2u * kWarps * 2u * RT * slot_row_bytes<T>(r.cols, seg); });
  if (!room.seg) return 0;
  a.seg = room.seg, a.fit = room.fit;
  a.smem = kLimit;
  const uint32_t units = (r.rows + 2 * RT - 1) / (2 * RT);
  dim3 grid((uint32_t) dev->sms);
  if (units < grid.x) grid.x = units;
  if constexpr (GROUP) {
    // an entry's rows over a few blocks, about four units a warp each and at most eight - more, down to a unit a warp, where
    // the entries are too few for three blocks an SM (one token's four MXFP4 experts of 1536 x 4096, the
    // layer: 123 us with the first rule alone, 57 with this one; the staged kernel 162), but a quarter fewer or less where their warps
    // take no more units each for it (128 experts top-4 of that shape, six tokens: 177 us a layer without this, whose
    // warps take one unit or two, 163 with it; 68 experts top-3 159 and 155, staged 172)
    const uint32_t sms = (uint32_t) dev->sms;
    const uint32_t some = units / (4u * kWarps) > 8u ? 8u : units / (4u * kWarps), most = units / kWarps;
    const uint32_t want = (3u * sms + r.n_entries - 1) / r.n_entries, more = want < most ? want : most;
    a.parts = some > more ? some : more;
    if (a.parts < 1u) a.parts = 1u;
    if (const uint32_t even = even_parts(units, a.parts); more > some && 4u * even <= 3u * a.parts) a.parts = even;
    const uint64_t blocks = (uint64_t) r.n_entries * a.parts;
    if (blocks > 0x7FFFFFFFull) return 0;
    grid.x = (uint32_t) blocks, a.n_entries = r.n_entries;
    if (r.cnt && r.n_entries > 12u && r.n_entries <= (uint32_t) kThreads) a.wave = grid.x < sms ? grid.x : sms;
  }
  static bool sized[64] = {};  // (one record a template instance, one flag a device)
  auto kernel = mv_pair_kernel<T, RT, GROUP>;
  if (!allow_dynamic_smem(kernel, (int) kLimit, sized)) return 0;
  return launch_dependent(kernel, grid, dim3(kThreads), kLimit, s, a) == cudaSuccess ? 1 : -1;
}

template <uint32_t T>
int by_shape(const Request& r, cudaStream_t s) {
  const Device* dev = device_info();
  if (!dev) return 0;
  if (r.wt) {
    if (const int st = launch<T, 2, true>(r, dev, s)) return st;
    return launch<T, 1, true>(r, dev, s);
  }
  // The kernel with a lane a thread (mv_staged.cu) where it is the faster one. Q8_0 has nothing to unpack, and with one or two
  // tokens that kernel's packed row pairs use half the instructions (49152 x 2048: 27.1 us against 34.0, two tokens 37.4
  // against 39.4; three 72.8 against 45.7). A matrix of few rows leaves most warps here without any - two rows a warp, not
  // one - which at the token counts that kernel has an instance for is felt in the types that unpack little (1024 x 8192, one
  // token: Q4_0 4.5 against 5.6, IQ4_XS 6.1 against 6.4, MXFP4 4.9 against 6.6; Q4_K, Q5_K and Q6_K are faster here at every
  // size). MXFP4's line, that kernel against this: at one token 2048 x 4096 4.8 / 5.1, 2368 x 4096 5.1 / 5.1; at two and more 1536
  // x 4096 5.2 / 5.7 (two), 7.1 / 7.4 (four), 10.9 / 10.9 (eight), 2048 x 4096 6.1 / 5.7, 8.4 / 7.5, 13.3 / 11.0, 2048 x 2048 4.0 / 4.0,
  // 5.3 / 4.8, 7.9 / 6.7.
  if (T == QTYPE_Q4_0 || T == QTYPE_Q8_0 || T == QTYPE_IQ4_XS || T == QTYPE_MXFP4) {
    const bool whole = (r.n_tok & (r.n_tok - 1)) == 0;
    const uint64_t few = (T == QTYPE_Q8_0 ? 16ull : T == QTYPE_MXFP4 ? (r.n_tok == 1 ? 16ull : 12ull) : 8ull) * dev->sms;
    if ((T == QTYPE_Q8_0 && r.n_tok <= 2) || (whole && r.rows <= few))
      if (const int st = mvs::try_launch(T, r, s)) return st;
  }
  // two rows a thread (they share x's reads) when every warp has units to spare
  if ((uint64_t) r.rows >= 8ull * kWarps * dev->sms)
    if (const int st = launch<T, 2, false>(r, dev, s)) return st;
  return launch<T, 1, false>(r, dev, s);
}

}  // namespace

int try_launch(uint32_t type, const Request& r, void* stream) {
  if (!r.rows || !r.n_tok || r.n_tok > kMaxTok || !r.cols || r.cols % 256) return 0;
  if (r.rows > 0x7FFFFFFFu) return 0;  // (a unit's rows in 32 bits; a row's bytes are where a token's x fits)
  if (r.wt) {  // every entry's x row starts on 16 bytes when the first does and the strides are whole words of 16
    if (((uintptr_t) r.x & 15u) || r.xs % 4 || r.x_mat % 4 || !r.n_entries || r.n_entries > 65535u) return 0;
  } else if ((((uintptr_t) r.w | (uintptr_t) r.x) & 15u) || (r.n_tok > 1 && r.xs % 4)) {
    return 0;
  }
  const cudaStream_t s = (cudaStream_t) stream;
  switch (type) {
    case QTYPE_Q4_0: return by_shape<QTYPE_Q4_0>(r, s);
    case QTYPE_Q8_0: return by_shape<QTYPE_Q8_0>(r, s);
    case QTYPE_Q4_K: return by_shape<QTYPE_Q4_K>(r, s);
    case QTYPE_Q5_K: return by_shape<QTYPE_Q5_K>(r, s);
    case QTYPE_Q6_K: return by_shape<QTYPE_Q6_K>(r, s);
    case QTYPE_IQ4_XS: return by_shape<QTYPE_IQ4_XS>(r, s);
    case QTYPE_MXFP4: return by_shape<QTYPE_MXFP4>(r, s);
    default: return 0;
  }
}

uint32_t read_status() {
  const Device* dev = device_info();
  if (!dev) return 0x80000000u;
  uint32_t v = 0, zero = 0;
  if (cudaMemcpy(&v, dev->status, sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess) return 0x80000000u;
  cudaMemcpy(dev->status, &zero, sizeof zero, cudaMemcpyHostToDevice);
  return v;
}

}  // namespace mvp
}  // namespace osmos
