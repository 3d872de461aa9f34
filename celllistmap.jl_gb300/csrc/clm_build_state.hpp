// What a particle set remembers from one build to the next, and the decisions taken from it, apart from the device
// buffers and launches that they govern (so that the CPU tests run them without a GPU).
#pragma once

#include <cstdint>

namespace clm {

struct BuildState {
  bool dirty = true;
  bool built = false;
  bool pending = false;      // the device totals of the last build were not read back yet
  // k_build_small: two halves of per-cell counters.  A launch counts in one half and clears the other for the next.
  int64_t small_cells = 0;   // cells that they are laid out and cleared for (0: none)
  unsigned small_epoch = 0;  // launches since they were cleared
};

// Before a launch of k_build_small that counts `ncells` cells (`moved`: in a new allocation): true when both halves have
// to be cleared first.
inline bool small_needs_clear(BuildState& S, int64_t ncells, bool moved) {
  if (S.small_cells == ncells && !moved) return false;
  S.small_cells = 0;
  S.small_epoch = 0;
  return true;
}
// The half that the next launch counts in.  It advances with a launch (small_launched) and not when one is prepared: a
// prepared launch that another set's failure drops has cleared nothing.
inline int small_half(const BuildState& S) { return (int)(S.small_epoch + 1) & 1; }
// After the launch, or its failure.
inline void small_launched(BuildState& S, int64_t ncells, bool ok) {
  S.small_cells = ok ? ncells : 0;
  S.small_epoch = ok ? S.small_epoch + 1 : 0;
}

// A build that was not enqueued to its end is not used: the next call builds the set again.
inline void drop_build(BuildState& S) {
  S.pending = false;
  S.dirty = true;
}

}  // namespace clm
