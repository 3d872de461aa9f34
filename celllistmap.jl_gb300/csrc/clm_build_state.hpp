// What a particle set remembers from one build to the next, and the decisions taken from it, apart from the device
// buffers and launches that they govern (so that the CPU tests run them without a GPU).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "clm_device.cuh"

namespace clm {

enum Status {
  RERUN_BUILD = -1,  // internal: the copies overflowed the capacity; rebuild with the exact size and rerun
  OK = 0, ERR_ARG = 1, ERR_CELL_TOO_SMALL = 2, ERR_NAN = 3, ERR_DIM = 4, ERR_CUDA = 5, ERR_CAPACITY = 6,
  ERR_STATE = 7, ERR_TIMEOUT = 8, ERR_NOMEM = 9, ERR_LCELL = 10, ERR_NONPERIODIC_CELL = 11, ERR_INTERNAL = 12
};

// Cells of more copies than this are built by radix (the counting build ranks each copy against its cell).
constexpr int kRadixAbovePerCell = 1024;
// Places per cell of the build of few particles, and the most that the bucket build takes.
constexpr int kBucket = 128;
constexpr int kBucketMost = 256;

struct BuildState {
  bool dirty = true;
  bool built = false;
  bool pending = false;      // the device totals of the last build were not read back yet
  int64_t n_copies = 0;      // valid once the build was synchronized (pending == false)
  int64_t n_real_cells = 0;
  int64_t copy_cap = 0;      // capacity for copies learned from previous builds
  int64_t cap_used = 0;      // capacity used by the last build
  bool counted = false;      // the last build counted its cells' copies (their number and its largest cell are read back)
  bool prefer_radix = false; // one met a cell of more than kRadixAbovePerCell copies
  int tile_mult = 0;         // counting build: staging slots per particle of a tile (0: from the estimate)
  size_t cell_count_zero = 0;  // bytes of the scan words and counters left cleared by the last build (0: clear before use)
  bool small = false;        // the last build was that of few particles (k_small_place)
  bool small_off = false;    // one met a cell with more copies than kBucket
  int bucket_used = 0;       // bucket build: places per cell of the last build (0: another build)
  int bucket = 0;            // places that an earlier build's largest cell called for
  bool bucket_off = false;   // a build met a cell with more copies than kBucketMost leaves room for
  // k_small_place: two halves of per-cell counters.  A launch counts in one half and clears the other for the next.
  int64_t small_cells = 0;   // cells that they are laid out and cleared for (0: none)
  unsigned small_epoch = 0;  // launches since they were cleared
};

// Before a launch of k_small_place that counts `ncells` cells (`moved`: in a new allocation): true when both halves have
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

// Places per cell for cells of up to `most` copies, a quarter more.
inline int bucket_places(int most) { return (most + most / 4 + 7) / 8 * 8; }

// A set (or a batch) whose fullest cells are no longer those of earlier builds.
inline void forget_crowding(BuildState& S) {
  S.small_off = S.bucket_off = S.prefer_radix = false;
  S.bucket = 0;
}

struct BuildCheck {
  int status;
  bool overflow;    // the builds are repeated with larger capacities
  const char* msg;  // of an error status
};

// After the host has the words of the last builds: `words` is the pinned area that build_totals fills (number of copies
// of set s at 32 + 2 s, of real cells at 33 + 2 s, the largest cell's copies at 44 + s, the error word at 40).
inline BuildCheck check_builds(BuildState* const* sets, int nsets, const int* words) {
  BuildCheck r{OK, false, nullptr};
  const int errw = words[40];
  if (errw & DERR_SCAN) {
    // blocks that gave up waiting left cells unwritten, and words that a later build would find cleared
    for (int s = 0; s < nsets; s++) {
      sets[s]->small_cells = 0;
      sets[s]->cell_count_zero = 0;
    }
  }
  if (errw & DERR_NAN) {
    for (int s = 0; s < nsets; s++) sets[s]->dirty = true;
    return {ERR_NAN, false, "Invalid coordinates found (NaN) in the particle positions."};
  }
  for (int s = 0; s < nsets; s++) {
    BuildState& S = *sets[s];
    if (!S.pending) continue;
    if (words[32 + 2 * s] < 0) {  // the 32-bit copy-offset scan wrapped: more than 2^31 - 1 copies
      drop_build(S);
      return {ERR_ARG, r.overflow,
              "too many particle copies for one set (particles and their periodic images exceed 2^31 - 1)"};
    }
    S.n_copies = words[32 + 2 * s];
    S.n_real_cells = words[33 + 2 * s];
    // the largest cell's copies (k_small_cells: 0 when every cell fits its bucket)
    const int most = S.counted ? words[44 + s] : 0;
    if (most > kRadixAbovePerCell) S.prefer_radix = true;
    if (errw & tile_overflow(s)) {
      if (S.small || S.bucket_used) {
        // more places than the largest cell's copies, or the builds without buckets
        if (S.small) S.small_off = true;
        if (bucket_places(most) <= kBucketMost) S.bucket = std::max(S.bucket, bucket_places(most));
        else S.bucket_off = true;
      } else {
        // a tile had more copies than its staging slots: more slots per particle, and build again
        S.tile_mult = std::min(27, 2 * S.tile_mult);
      }
      S.dirty = true;
      r.overflow = true;
    } else if (S.counted && !S.small) {
      // Cells that have become emptier: the builds given up are taken again once the fullest cell leaves a quarter of
      // their places free, so that a set near the line does not overflow every other step.
      if (4 * most <= 3 * kBucket) S.small_off = false;
      if (S.bucket_off && 4 * most <= 3 * kBucketMost) {
        S.bucket_off = false;
        S.bucket = bucket_places(most);
      }
      if (2 * most <= S.bucket) S.bucket = bucket_places(most);
    }
    S.pending = false;
    if (S.n_copies > S.cap_used || (errw & DERR_COPY_OVERFLOW)) {
      S.copy_cap = S.n_copies + S.n_copies / 8 + 1024;
      S.dirty = true;
      r.overflow = true;
    } else if (S.n_copies > S.copy_cap) {
      S.copy_cap = S.n_copies;
    }
  }
  // A list that a failed build left is not used by a later call: the sets are built again.
  const bool scan = errw & DERR_SCAN, range = !r.overflow && (errw & DERR_CELL_RANGE);
  for (int s = 0; (scan || range) && s < nsets; s++) drop_build(*sets[s]);
  if (scan) return {ERR_INTERNAL, r.overflow, "cell-list build: a scan tile gave up waiting for an earlier tile"};
  if (range)
    return {ERR_INTERNAL, false, "cell-list build consistency check failed (particle outside the computing box)"};
  return r;
}

}  // namespace clm
