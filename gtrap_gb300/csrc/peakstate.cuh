// States of listed peak candidates, shared by warps that decide them at the same time.
//
// The states of 32 consecutive candidates are one 64-bit word: bit c of the low half, candidate c is
// undecided; bit c of the high half, it is kept; neither, it is deleted.  A word is read and written by
// one 64-bit access, so a reader sees, for each candidate, a state that it has had, whatever else is in
// flight: undecided (wait for it), kept or deleted, and the last two never change.  Two words, one for
// each bit, would need their two loads ordered as the writer orders its stores: a reader that saw a
// neighbour no longer undecided and not yet kept would take it for deleted and keep a peak too many.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GTRAP_PEAK_FN __host__ __device__ __forceinline__
#else
#define GTRAP_PEAK_FN inline
#endif

namespace gtrap {

GTRAP_PEAK_FN uint32_t undecided_of(uint64_t s) { return (uint32_t)s; }
GTRAP_PEAK_FN uint32_t kept_of(uint64_t s) { return (uint32_t)(s >> 32); }
GTRAP_PEAK_FN uint64_t peak_word(uint32_t undecided, uint32_t kept) { return (uint64_t)kept << 32 | undecided; }

// Bits of the kReach (8 or 16) candidates on either side of candidate `lane` of the word `mid`: bit j
// below kReach is entry lane - kReach + j, bit kReach + j is entry lane + 1 + j.
template <int kReach>
GTRAP_PEAK_FN uint32_t bits_around(uint32_t before, uint32_t mid, uint32_t behind, int lane) {
  constexpr uint32_t kMask = (1u << kReach) - 1u;
  const uint64_t lo = (uint64_t)mid << 32 | before, hi = (uint64_t)behind << 32 | mid;
  return ((uint32_t)(lo >> (32 - kReach + lane)) & kMask) | ((uint32_t)(hi >> (lane + 1)) & kMask) << kReach;
}

// What the higher-ranking candidates around `lane` (bits of `higher`, as above) do to it, from one view
// of its own word and of the words on either side: a kept one deletes it, an undecided one holds it up.
template <int kReach>
GTRAP_PEAK_FN void peak_decide(uint64_t before, uint64_t mid, uint64_t behind, uint32_t higher, int lane,
                               bool &deleted, bool &blocked) {
  deleted = higher & bits_around<kReach>(kept_of(before), kept_of(mid), kept_of(behind), lane);
  blocked = higher & bits_around<kReach>(undecided_of(before), undecided_of(mid), undecided_of(behind), lane);
}

}  // namespace gtrap
