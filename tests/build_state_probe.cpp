// Test infrastructure: the state that a set carries from build to build (clm_build_state.hpp), driven on the host with
// a model of the launches (built by tests/test_build_state.py).
#include <cstdint>
#include <vector>

#include "clm_build_state.hpp"

// Builds of one set with the counters of k_small_place: step k of `script` is 0 (prepared and launched), 1 (prepared, dropped
// because the other set failed), 2 (prepared, the launch failed), 3 (launched with another number of cells) or 4
// (launched in a new allocation).  Returns the first step whose launch found counters that were not clear, or -1.
extern "C" int small_counters_probe(const int* script, int n) {
  clm::BuildState S;
  std::vector<int> half(2, 99);  // what each half holds; the memory starts uncleared
  int64_t cells = 100;
  for (int k = 0; k < n; k++) {
    if (script[k] == 3) cells = cells == 100 ? 64 : 100;
    if (script[k] == 4) half.assign(2, 99);
    if (clm::small_needs_clear(S, cells, k == 0 || script[k] == 4)) half.assign(2, 0);
    if (script[k] == 1) {
      clm::drop_build(S);
      if (!S.dirty || S.pending) return k;
      continue;
    }
    const bool ok = script[k] != 2;
    const int h = clm::small_half(S);
    if (ok) {
      if (half[(size_t)h] != 0) return k;
      half[(size_t)h] = 7;  // the copies of this build
      half[(size_t)(1 - h)] = 0;
    }
    clm::small_launched(S, cells, ok);
  }
  return -1;
}

// check_builds on two sets built together (kind: 0 counting, 1 few particles, 2 bucket), with the given words of the
// device: out = {status, overflow, then for each set dirty, pending, counters to be cleared}.
extern "C" void check_probe(int kind, int errw, int copies, int largest, int* out) {
  clm::BuildState S[2];
  int words[64] = {};
  words[40] = errw;
  for (int s = 0; s < 2; s++) {
    S[s].built = S[s].counted = S[s].pending = true;
    S[s].dirty = false;
    S[s].small = kind == 1;
    S[s].bucket_used = kind == 2 ? 24 : 0;
    S[s].tile_mult = 2;
    S[s].cap_used = S[s].copy_cap = 1000;
    S[s].small_cells = 100;
    S[s].cell_count_zero = 800;
    words[32 + 2 * s] = copies;
    words[33 + 2 * s] = 10;
    words[44 + s] = largest;
  }
  clm::BuildState* sets[2] = {&S[0], &S[1]};
  const clm::BuildCheck c = clm::check_builds(sets, 2, words);
  out[0] = c.status;
  out[1] = c.overflow;
  for (int s = 0; s < 2; s++) {
    out[2 + 3 * s] = S[s].dirty;
    out[3 + 3 * s] = S[s].pending;
    out[4 + 3 * s] = S[s].small_cells == 0 && S[s].cell_count_zero == 0;
  }
}

// A sequence of steps of two sets built together: step k has the builds kind[k][s] (0 counting, 1 few particles, 2 bucket
// of 24 places, 3 none) and the largest cells most[k][s]; each flags an overflow of its own set when the cell does not
// fit.  state[k][s] after the step: small_off, bucket_off, bucket, dirty, tile_mult.
extern "C" void crowding_probe(int n, const int* kind, const int* most, int* state) {
  clm::BuildState S[2];
  clm::BuildState* sets[2] = {&S[0], &S[1]};
  for (int k = 0; k < n; k++) {
    int words[64] = {};
    for (int s = 0; s < 2; s++) {
      const int kd = kind[2 * k + s], m = most[2 * k + s];
      S[s].built = true;
      S[s].dirty = false;
      S[s].pending = kd != 3;
      S[s].counted = true;
      S[s].small = kd == 1;
      S[s].bucket_used = kd == 2 ? std::max(24, S[s].bucket) : 0;
      if (S[s].tile_mult == 0) S[s].tile_mult = 2;
      S[s].cap_used = 1000;
      words[32 + 2 * s] = 900;
      words[44 + s] = kd == 1 && m <= clm::kBucket ? 0 : m;
      if ((kd == 1 && m > clm::kBucket) || (kd == 2 && m > S[s].bucket_used)) words[40] |= clm::tile_overflow(s);
    }
    clm::check_builds(sets, 2, words);
    for (int s = 0; s < 2; s++) {
      int* o = state + 10 * k + 5 * s;
      o[0] = S[s].small_off;
      o[1] = S[s].bucket_off;
      o[2] = S[s].bucket;
      o[3] = S[s].dirty;
      o[4] = S[s].tile_mult;
    }
  }
}
