// Status bits that kernels raise, and what a finished query answers. Host-only C++ apart from the
// constants, shared by the library and its CPU unit test.
#pragma once
#include <cstdint>

namespace gz {

// Status bits a kernel may raise in the handle's device status word.
enum : uint32_t {
  kStatusBadVertex = 1u << 0,
  kStatusTimeout = 1u << 1,
  kStatusBadSample = 1u << 2,
};

enum class QueryOutcome { kAnswer, kTimeout, kOutOfSamples, kBadSample };

// Outcome of a query from the device status as it left it and from its out-of-samples word. A query
// whose wait gave up returned without writing that word, the rounds, the labels or the component
// count, so the status comes first: none of them is looked at after a timeout. (The bit may also be
// an earlier update's: the sketches are then not to be trusted either.)
inline QueryOutcome query_outcome(uint32_t status, uint32_t out_of_samples) {
  if (status & kStatusTimeout) return QueryOutcome::kTimeout;
  if (out_of_samples) return QueryOutcome::kOutOfSamples;
  if (status & kStatusBadSample) return QueryOutcome::kBadSample;
  return QueryOutcome::kAnswer;
}

}  // namespace gz
