// Host model of a ring of buffers with mbarrier phases: whatever is in flight when a
// pipeline stops, for_pending_copies (csrc/tc_util.cuh) waits for all of it and for
// nothing that was never issued.
#include <stdio.h>

#include <vector>

#include "tc_util.cuh"

int main() {
  int bad = 0;
  for (int stages = 1; stages <= 4; ++stages)
    for (int issued = 0; issued <= 4 * stages + 1; ++issued)
      for (int arrived = issued > stages ? issued - stages : 0; arrived <= issued; ++arrived) {
        // copies 0 .. arrived - 1 have arrived; a buffer's barrier is in phase
        // (copies of it that have arrived)
        std::vector<int> phase(stages, 0), waits(stages, 0);
        for (int c = 0; c < arrived; ++c) ++phase[c % stages];
        std::vector<bool> in_flight(stages, false);
        for (int c = arrived; c < issued; ++c) in_flight[c % stages] = true;
        smx::tc::for_pending_copies(issued, stages, [&](int s, unsigned parity) {
          ++waits[s];
          const bool done = (phase[s] & 1) != int(parity);  // the phase of that parity is over
          if (in_flight[s] == done) ++bad;                  // returns at once with a copy in flight, or never
          if (!done) ++phase[s], in_flight[s] = false;      // (the copy arrives)
        });
        for (int s = 0; s < stages; ++s)
          if (in_flight[s] || waits[s] != (s < issued)) ++bad;
      }
  printf("%d\n", bad);
  return bad != 0;
}
