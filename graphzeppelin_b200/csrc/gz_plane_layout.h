// Places in a sketch that the plane updates touch ahead of time. Usable on the host and on the device,
// shared with the CPU unit test.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GZ_HD __host__ __device__
#else
#define GZ_HD
#endif

namespace gz {

// A column of B buckets is brought to L2 by its first word and by this one, 64 bytes on, or by its last word
// where it is shorter: nothing past the sketch is named, which a caller's own buffer may end with.
GZ_HD constexpr uint32_t column_second_word(uint32_t B) { return 3 * B - 1 < 16 ? 3 * B - 1 : 16; }

}  // namespace gz
