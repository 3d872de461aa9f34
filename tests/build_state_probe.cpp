// Test infrastructure: the state that a set carries from build to build (clm_build_state.hpp), driven on the host with
// a model of the launches (built by tests/test_build_state.py).
#include <cstdint>
#include <vector>

#include "clm_build_state.hpp"

// Builds of one set with k_build_small's counters: step k of `script` is 0 (prepared and launched), 1 (prepared, dropped
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
