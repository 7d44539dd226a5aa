// Properties of DirectRoute (graphzeppelin_b200/csrc/gz_ingest_plan.h): which record calls go straight to
// the sketches, over streams of calls between two flushes.
#include <cstdio>
#include <cstdlib>

#include "gz_ingest_plan.h"

static int failures = 0;
#define CHECK(c)                                                        \
  do {                                                                  \
    if (!(c)) {                                                         \
      ++failures;                                                       \
      std::printf("FAIL %s:%d: %s\n", __FILE__, __LINE__, #c);          \
    }                                                                   \
  } while (0)

// A stream of `calls` calls of n records with nothing flushed in between; records that went direct.
static uint64_t stream(gz::DirectRoute &r, uint64_t n, int calls, double entries, uint64_t bytes) {
  uint64_t direct = 0, pending = 0;
  for (int i = 0; i < calls; ++i) {
    if (r.take(n, entries, pending, bytes)) direct += n;
    else pending += 2 * n;
  }
  return direct;
}

int main() {
  const uint64_t kSizes[] = {1ull << 20, 1ull << 27, (1ull << 27) + 1, 400ull << 20, 1ull << 29, 1ull << 30, 16ull << 30};
  const uint64_t kCalls[] = {1, 16, 500, 16384, 16385, 20000, 200000, 1000000, 2000000};
  for (uint64_t bytes : kSizes) {
    const double entries = (double)(bytes / 8192) * 4;  // 4 entries a vertex, sketches of 8 KB
    const double limit = entries * (bytes > gz::kWideSketchBytes ? 0.25 : 0.5);
    for (uint64_t n : kCalls) {
      gz::DirectRoute r;
      // one call alone: by the limit only
      CHECK(r.take(n, entries, 0, bytes) == ((double)n < limit));
      r.flushed();
      CHECK(r.sent == 0);
      // however long the stream, calls whose direct form costs more than a gutter pass send no more
      // than the limit together; the others always go direct below the limit
      const uint64_t direct = stream(r, n, 1000, entries, bytes);
      const bool cheap = n <= gz::kDirectAlways || 4.0 * (double)n <= limit || bytes <= gz::kResidentSketchBytes;
      if ((double)n >= limit) CHECK(direct == 0);
      else if (cheap) CHECK(direct == 1000 * n);
      else CHECK(direct >= n && (double)direct < limit);
      // the gutter waits with entries: only cheap calls go direct
      gz::DirectRoute p;
      CHECK(p.take(n, entries, 2, bytes) == (cheap && (double)n < limit));
      CHECK(p.sent == 0);
      // a flush starts the interval anew
      r.flushed();
      CHECK(stream(r, n, 1000, entries, bytes) == direct);
      CHECK(!r.take(n, 0.0, 0, bytes));  // factor 0
    }
  }
  if (!failures) std::printf("direct route ok\n");
  return failures ? 1 : 0;
}
