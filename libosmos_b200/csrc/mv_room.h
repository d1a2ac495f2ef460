// How the F32-activation matvecs' blocks share out their shared memory (mv_staged.cu, mv_pair.cu): host arithmetic, in 64 bits
// throughout - a row that is wider than any block must come out as "no room", never as a product that has wrapped round.
#pragma once
#include <cstdint>

namespace osmos {
namespace mv_room {

// the slots a warp's ring has beside the tokens' x: `most` at most, 0 where x alone does not fit
inline uint32_t staged_slots(uint64_t budget, uint32_t warps, uint32_t most, uint64_t slot_bytes, uint32_t x_tokens, uint32_t cols) {
  const uint64_t x = ((uint64_t) x_tokens * cols * 4u + 127u) & ~(uint64_t) 127u;
  if (x >= budget || !slot_bytes) return 0;
  const uint64_t n = (budget - x) / (warps * slot_bytes);
  return n > most ? most : (uint32_t) n;
}

// The paired kernel's passes: the tokens a pass holds (`fit`, at most max_tok) beside rings of two slots of `seg` stretches of a
// row - the longest slots that need the fewest passes over the weights. seg 0: not even one token's x fits beside the shortest.
// ring_bytes(seg): the block's rings.
struct Passes {
  uint32_t seg, fit;
};
template <class F>
Passes pair_passes(uint64_t limit, uint32_t max_seg, uint32_t max_tok, uint32_t n_tok, uint32_t cols, F ring_bytes) {
  Passes best{0, 0};
  uint64_t fewest = 0;
  const uint64_t x = (uint64_t) cols * 4u;  // a token's
  for (uint32_t seg = max_seg; seg && x; seg >>= 1) {
    const uint64_t rings = (uint64_t) ring_bytes(seg) + 128u;  // (x ends on 128 bytes)
    if (rings + x > limit) continue;
    uint64_t fit = (limit - rings) / x;
    if (fit > max_tok) fit = max_tok;
    const uint64_t passes = (n_tok + fit - 1) / fit;
    if (!fewest || passes < fewest) fewest = passes, best.seg = seg, best.fit = (uint32_t) fit;
  }
  return best;
}

}  // namespace mv_room
}  // namespace osmos
