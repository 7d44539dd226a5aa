// FailedSize (graphzeppelin_b200/csrc/gz_ingest_plan.h): a buffer that could not be had is asked for again
// only in a smaller size.
#include <cstdio>

#include "gz_ingest_plan.h"

int main() {
  gz::FailedSize f;
  int bad = !f.may_try(0) + !f.may_try(1ull << 62);
  f.failed(1000);
  bad += !f.may_try(999) + f.may_try(1000) + f.may_try(1001) + f.may_try(~0ull);
  f.failed(5000);  // larger than what failed already: nothing changes
  bad += !f.may_try(999) + f.may_try(1000);
  f.failed(10);
  bad += !f.may_try(9) + f.may_try(10) + f.may_try(999);
  // a buffer too large for the memory, asked for by a hundred calls: one attempt
  gz::FailedSize g;
  int attempts = 0;
  for (int i = 0; i < 100; ++i)
    if (g.may_try(1 << 20)) {
      ++attempts;
      g.failed(1 << 20);
    }
  bad += attempts != 1;
  if (!bad) std::printf("failed size ok\n");
  return bad != 0;
}
