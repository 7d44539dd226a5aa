// query_outcome (graphzeppelin_b200/csrc/gz_status.h) over every combination of status bits and values that
// an out-of-samples word may hold, written or not.
#include <cstdio>

#include "gz_status.h"

int main() {
  using namespace gz;
  int bad = 0;
  const uint32_t words[] = {0u, 1u, 0xdeadbeefu, 0xffffffffu};
  for (uint32_t st = 0; st < 8; ++st)
    for (uint32_t oos : words) {
      const QueryOutcome o = query_outcome(st, oos);
      const QueryOutcome want = st & kStatusTimeout ? QueryOutcome::kTimeout
                                : oos               ? QueryOutcome::kOutOfSamples
                                : st & kStatusBadSample ? QueryOutcome::kBadSample
                                                        : QueryOutcome::kAnswer;
      if (o != want) {
        ++bad;
        std::printf("FAIL status %u word %u\n", st, oos);
      }
    }
  if (!bad) std::printf("query outcome ok\n");
  return bad ? 1 : 0;
}
