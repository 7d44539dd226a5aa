// Plans of record ingest, host-only C++ shared by the library and its CPU unit tests: how a host
// call's records are cut into host->device copies and when the gutter is folded into the sketches
// (IngestPlan), which calls go straight to the sketches instead of the gutter (DirectRoute), and which
// optional buffers are not asked for again (FailedSize).
//
// The copies run on a second stream into kStageBuffers device buffers while the gutter and the
// sketch update run on the handle's stream. A long call is cut so that the sketch update overlaps
// the copies from start to end: the first chunk is kFirstChunk records and the chunks double up to
// kStageRecords, and every chunk is folded into the sketches as soon as it lands (a wave of its
// own). The last kTailRecords records come as a tail of halving chunks (about 8, 4 and 2 Mi
// records) with no wave of their own: a wave re-reads and re-writes every vertex sketch it
// touches, which costs more than a small chunk's copy, so their gutter passes keep pace with the
// copies and one wave folds the whole tail at the next flush or query, when the last and
// smallest chunk has landed. This shape is used only while all sketches together are at most
// kShapeSketchBytes (a pass over them then costs a fraction of a millisecond, and a chunk's
// sketch update keeps pace with the copy of the next); other calls copy kStageRecords-record
// chunks and fold one wave per kWaveEntries endpoint updates.
#pragma once

#include <algorithm>
#include <cstdint>

namespace gz {

constexpr uint64_t kStageRecords = 1ull << 24;  // records per host->device copy, at most
constexpr int kStageBuffers = 4;                 // device staging buffers of the copy pipeline
constexpr uint64_t kWaveEntries = 1ull << 26;    // endpoint updates per wave of an unshaped call
constexpr uint64_t kFirstChunk = 1ull << 23;
constexpr uint64_t kLastChunk = 1ull << 21;                       // the tail's last chunk
constexpr uint64_t kTailRecords = (1ull << 23) + (1ull << 22) + kLastChunk;  // the tail
constexpr uint64_t kShapeSketchBytes = 3ull << 29;
static_assert(kFirstChunk <= kStageRecords && kTailRecords <= kStageRecords, "shaped chunks fit a stage");

struct IngestPlan {
  uint64_t n = 0;       // records of the call
  uint64_t chunk = 0;   // largest chunk (= the staging buffers' capacity in records)
  uint64_t ramp = 0;    // size of the next chunk before the end-of-call rule
  bool shaped = false;  // doubling first chunks, a wave per chunk, a tail of halving chunks

  // in_place: the handle applies records straight to the sketches (no gutter, no waves);
  // sketch_bytes_total: every vertex sketch of the handle together.
  IngestPlan(uint64_t n_, bool in_place, uint64_t sketch_bytes_total)
      : n(n_), chunk(std::min<uint64_t>(kStageRecords, n_)) {
    shaped = n > 2 * kStageRecords && !in_place && sketch_bytes_total <= kShapeSketchBytes;
    ramp = shaped ? std::min(kFirstChunk, chunk) : chunk;
  }

  // Records of the chunk that starts at record off (off < n); at least 1, at most chunk.
  uint64_t next(uint64_t off) {
    const uint64_t left = n - off;
    uint64_t m = std::min(ramp, left);
    if (shaped) {
      if (left > kTailRecords) {
        m = std::min(m, left - kTailRecords);  // the full chunks end where the tail starts
      } else {
        // the tail: what is left above 2 Mi + 4 Mi, then 4 Mi, then 2 Mi
        const uint64_t rest = kLastChunk + (kLastChunk << 1);
        m = left > rest ? left - rest : left > kLastChunk ? left - kLastChunk : left;
      }
    }
    ramp = std::min(2 * ramp, chunk);
    return m;
  }

  // Whether to fold the gutter into the sketches after the chunk that ends at record end, with
  // pending endpoint updates buffered. The last chunk (and in the shaped form the whole tail) is
  // left to the next flush or query.
  bool wave_after(uint64_t end, uint64_t pending) const {
    if (shaped) return n - end >= kTailRecords && end < n;
    return end < n && pending >= kWaveEntries;
  }
};

// Calls that skip the gutter. A record XORed straight into both endpoints' sketches costs about 60
// L2 reductions -- 0.3 ns of the GPU while all sketches lie in L2, 1.2 to 2.4 ns past that -- but no
// gutter pass (25 to 50 us) and no wave (a pass over the touched tiles). Which is cheaper depends on
// everything that arrives before the next flush, not on one call:
//   limit   records between two flushes (a query is one) that are cheaper direct than as a wave of
//           their own: the in-place break-even of every tile, entries_in_place entries together;
//           half of that past kWideSketchBytes, where reductions miss L2 (call and flush, direct
//           against gutter: 50,021 vertices, 420 MB of sketches, 100,042 records 133 and 144 us,
//           150,063 189 and 153; 2^18 vertices, 3 GB, 131,072 records 299 and 454 us, 262,144 571 and
//           503, 393,216 840 and 535; 2^20, 524,288 1.26 and 1.64 ms, 1,572,864 3.73 and 1.98).
//   always  records of a call that cost no more direct than the call's own gutter pass and its chunk's
//           part in a wave of many, whatever came before: a quarter of the limit, kDirectAlways at
//           least, and with resident sketches all below the limit (a call direct, against gutter pass
//           plus a twentieth of the flush of 20: 16,384 vertices, 100,000 records 31 and 37 us;
//           50,021, 20,000 21 and 46, 50,000 60 and 47; 2^17, 20,000 34 and 69, 50,000 99 and 74;
//           2^20, 200,000 483 and 528, 500,000 1184 and 581).
// A call above `always` goes direct only while nothing waits in the gutter and the interval's calls
// of this kind stay below the limit together; after that the stream fills the gutter (2^17 vertices, 60
// calls of 200,000 records and one flush: 22.0 ms judged call by call, 5.6 judged together; 2^20, 13 of
// 1e6: 30.3 and 10.9).
constexpr uint64_t kResidentSketchBytes = 1ull << 27;
constexpr uint64_t kWideSketchBytes = 1ull << 29;
constexpr uint64_t kDirectAlways = 1ull << 14;

struct DirectRoute {
  uint64_t sent = 0;  // records of calls above `always` that went direct since the last flush

  // Whether the n records of a call go direct (counted as sent when they do).
  // entries_in_place: entries that all tiles together take in place (0: no call goes direct);
  // entries_pending: entries waiting in the gutter; sketch_bytes_total: as for IngestPlan.
  bool take(uint64_t n, double entries_in_place, uint64_t entries_pending, uint64_t sketch_bytes_total) {
    const double limit = entries_in_place * (sketch_bytes_total > kWideSketchBytes ? 0.25 : 0.5);
    if (!((double)n < limit)) return false;
    if (n <= kDirectAlways || 4.0 * (double)n <= limit || sketch_bytes_total <= kResidentSketchBytes) return true;
    if (entries_pending || !((double)(sent + n) < limit)) return false;
    sent += n;
    return true;
  }
  void flushed() { sent = 0; }
};

// Sizes at which an optional buffer could not be had. The caller then takes the form that does without, and
// does not ask for as much again: a failed allocation costs milliseconds, and a growing buffer gives
// its old block up first.
struct FailedSize {
  uint64_t least = ~0ull;
  bool may_try(uint64_t size) const { return size < least; }
  void failed(uint64_t size) { least = std::min(least, size); }
};

}  // namespace gz
