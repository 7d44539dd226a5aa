// gz_planes.cuh -- bucket planes: device code of the sketch updates that accumulate a tile's entries in
// shared memory (single graphs, gz_planes.cu; many graphs, gz_batch.cu).
//
// Bucket planes. A warp takes 32 entries, one per lane. At step t = 0..31 lane l handles slot
// l ^ t of its entry: slot s < C is column s, slot C the deterministic bucket, higher slots are
// unused (sketches of more columns go in groups of 32 slots, one pass over the entries each). A
// plane row holds 32 slots, so slot s is shared-memory bank s and the 32 lanes of a step hit 32
// different banks whatever their vertices and depths: the red.shared.xor never conflict (the
// per-entry ordering, every lane on column c at once, concentrates lanes on a few banks because
// depth 0 takes half the updates). Each bucket is kept as four words,
//   A = XOR of (neighbour | 1 << 31) over the entries whose neighbour is above the vertex,
//   GA = XOR of their checksums,
//   B and GB = the same over the other entries (the bucket's gamma is GA ^ GB),
// so one update XORs two words (A and GA, or B and GB) instead of three. With idx = (min << 32) | max
// (concat_pairing_fn, src/util.cpp:45-51) the bucket's alpha is recovered as
//   alpha low  = low31(A) ^ (top bit of B ? vertex : 0),
//   alpha high = low31(B) ^ (top bit of A ? vertex : 0),
// the top bits holding the parity of each kind's entry count (vertex ids are below 2^31).
// Rows hold depths 0 .. kPlaneRows - 2; the last row collects the depths at or above it (2^-11 of
// the column updates), which are XORed into the sketch in HBM with global atomics; the write-back changes
// only the buckets of the rows above it (CubeSketch, whose buckets take every depth from their own on,
// counts the last row in).
//
// What bounds the update: shared-memory issue. A slot step is two red.shared.xor, one wavefront
// each, 64 wavefronts per 32 entries and SM. The address of a step is made by one byte permute
// and one XOR: a row is 256 bytes -- 32 slots of A (or B), then the same slots' checksums, reached with
// an immediate offset of 128 -- so that address byte 0 is the slot, byte 1 the row (the code plus the
// plane's first row, added to four codes at once; planes never straddle a 64 KB boundary), and the
// rest the plane's 64 KB block.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "gz_common.cuh"
#include "gz_device.cuh"
#include "gz_kernels.cuh"
#include "gz_plane_layout.h"

namespace gz {
namespace dev {

constexpr uint32_t kPlaneThr = kPlaneRows - 1;  // first depth not held in the planes
constexpr uint32_t kRowBytes = 256;             // 32 slots, then their checksums
constexpr uint32_t kGOff = kPlaneSlots * 4;     // a slot's checksum sits this far behind it
constexpr uint32_t kQueueSlots = 64;            // per-warp queue of filtered entries

constexpr uint32_t kPairRows = 2 * kPlaneRows;  // planes A and B of one vertex, back to back

// Bytes of the planes of 1 << tile_shift vertices, the unused rows before 64 KB boundaries included,
// when they start within the first 4 KB of the block's shared memory: 10 pairs fit before the first
// boundary and 10 between boundaries, and 4 KB at most are left over.
__host__ __device__ constexpr uint32_t planes_bytes(uint32_t tile_shift) {
  const uint32_t n = 1u << tile_shift;
  return n * kPairRows * kRowBytes + (n - 1) / 10 * 4096u;
}

// Depth codes of up to 32 columns into the nibble words w (column c of kcol in bits 4 (c % 8) of
// word c / 8; nibbles past nc are zero); pm = premixed edge index. min(depth, 11) of a hash is the
// place of the lowest bit of (hash | cap), 31 - clz of that bit alone (a quarter-rate bit reverse
// less than counting trailing zeros: 1.48e12 against 1.34e12 codes/s on a register-only kernel).
// The clz values, 16 .. 31 each, are summed at nibble distances; taking 16 per nibble off and
// complementing turns all of a word's nibbles into codes at once. LO columns are known to exist.
template <int LO>
__device__ __forceinline__ void all_codes(uint64_t pm, const uint64_t *kcol, uint32_t nc, uint32_t cap,
                                          uint32_t (&w)[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t x = 0;
    if (8 * q < LO || 8u * q < nc) {
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        const int c = 8 * q + k;
        if (c + 1 < LO || (uint32_t)c < nc) {
          const uint32_t y0 = tail_lo32(pm ^ kcol[c]) | cap, y1 = tail_lo32(pm ^ kcol[c + 1]) | cap;
          x += (uint32_t)__clz(y0 & (0u - y0)) << (4 * k);
          x += (uint32_t)__clz(y1 & (0u - y1)) << (4 * k + 4);
        }
      }
      x = ~(x - 0x11111110u);
      const uint32_t n = 8 * q + 8 <= LO ? 8u : min(nc - 8u * q, 8u);
      if (8 * q + 8 > LO && n < 8) x &= (1u << (4 * n)) - 1u;
    }
    w[q] = x;
  }
}

// Coded entry of vertex a (neighbour b): the codes, then the payload (b << bin_shift) | (a & bin
// mask): in the last word where the codes leave it free (every sketch up to 2^17 vertices; taking
// an entry apart then needs no 64-bit shifts), else from bit 4C on.
constexpr uint32_t kWordCodes = 24;  // columns whose codes leave the last word free
__device__ __forceinline__ uint4 pack_entry(const uint32_t (&w)[4], uint32_t a, uint32_t b,
                                            uint32_t C, uint32_t bin_shift) {
  if (C <= kWordCodes) return make_uint4(w[0], w[1], w[2], (b << bin_shift) | (a & ((1u << bin_shift) - 1u)));
  const uint64_t pay = ((uint64_t)b << bin_shift) | (a & ((1u << bin_shift) - 1u));
  const uint64_t hi = (((uint64_t)w[3] << 32) | w[2]) | (pay << (4 * C - 64));
  return make_uint4(w[0], w[1], (uint32_t)hi, (uint32_t)(hi >> 32));
}

// Vertex, neighbour and codes of a coded entry lying in gutter bin `bin`.
__device__ __forceinline__ void unpack_entry(uint4 e, uint32_t bin, uint32_t C, uint32_t bin_shift,
                                             uint32_t &v, uint32_t &u, uint32_t (&w)[4]) {
  if (C <= kWordCodes) {
    v = (bin << bin_shift) | (e.w & ((1u << bin_shift) - 1u));
    u = e.w >> bin_shift;
    w[0] = e.x;
    w[1] = e.y;
    w[2] = e.z;
    w[3] = 0;
    return;
  }
  const uint64_t hi = ((uint64_t)e.w << 32) | e.z;
  const uint32_t sh = 4 * C - 64;
  const uint64_t pay = hi >> sh;
  const uint64_t codes_hi = hi & ((1ull << sh) - 1ull);
  v = (bin << bin_shift) | ((uint32_t)pay & ((1u << bin_shift) - 1u));
  u = (uint32_t)(pay >> bin_shift);
  w[0] = e.x;
  w[1] = e.y;
  w[2] = (uint32_t)codes_hi;
  w[3] = (uint32_t)(codes_hi >> 32);
}

// 3-bit codes (kEntryCoded3). Eight nibbles holding values <= 7 <-> their low 3 bits packed into
// 24 bits (nibble k at bits 3k .. 3k + 2), in three steps of pairs.
__device__ __forceinline__ uint32_t squeeze3(uint32_t w) {
  w = (w & 0x07070707u) | ((w >> 1) & 0x38383838u);
  w = (w & 0x003f003fu) | ((w >> 2) & 0x0fc00fc0u);
  return (w & 0x00000fffu) | ((w >> 4) & 0x00fff000u);
}
__device__ __forceinline__ uint32_t spread3(uint32_t x) {
  x = (x & 0x00000fffu) | ((x << 4) & 0x0fff0000u);
  x = (x & 0x003f003fu) | ((x << 2) & 0x3f003f00u);
  return (x & 0x07070707u) | ((x << 1) & 0x70707070u);
}

// Coded entry with 3-bit codes of vertex a (neighbour b): codes (each <= 7, as nibbles in w) in
// bits 0 .. 3C - 1, then from bit 3C the payload (b << bin_shift) | (a & bin mask). 3C >= 54.
__device__ __forceinline__ uint4 pack_entry3(const uint32_t (&w)[4], uint32_t a, uint32_t b,
                                             uint32_t C, uint32_t bin_shift) {
  const uint64_t z2 = squeeze3(w[2]);
  uint64_t lo = (uint64_t)squeeze3(w[0]) | ((uint64_t)squeeze3(w[1]) << 24) | (z2 << 48);
  uint64_t hi = (z2 >> 16) | ((uint64_t)squeeze3(w[3]) << 8);
  const uint64_t pay = ((uint64_t)b << bin_shift) | (a & ((1u << bin_shift) - 1u));
  const uint32_t sh = 3 * C;
  if (sh >= 64) {
    hi |= pay << (sh - 64);
  } else {
    lo |= pay << sh;
    hi |= pay >> (64 - sh);
  }
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}

// Payload (bits from 3C on) of a 3-bit coded entry.
__device__ __forceinline__ uint64_t payload3(uint4 e, uint32_t C) {
  const uint64_t lo = ((uint64_t)e.y << 32) | e.x, hi = ((uint64_t)e.w << 32) | e.z;
  const uint32_t sh = 3 * C;
  return sh >= 64 ? hi >> (sh - 64) : (lo >> sh) | (hi << (64 - sh));
}

// Vertex, neighbour and codes (as nibbles, escapes = 7 left in place) of a 3-bit coded entry
// lying in gutter bin `bin`.
__device__ __forceinline__ void unpack_entry3(uint4 e, uint32_t bin, uint32_t C, uint32_t bin_shift,
                                              uint32_t &v, uint32_t &u, uint32_t (&w)[4]) {
  uint64_t lo = ((uint64_t)e.y << 32) | e.x, hi = ((uint64_t)e.w << 32) | e.z;
  const uint32_t sh = 3 * C;
  const uint64_t pay = sh >= 64 ? hi >> (sh - 64) : (lo >> sh) | (hi << (64 - sh));
  v = (bin << bin_shift) | ((uint32_t)pay & ((1u << bin_shift) - 1u));
  u = (uint32_t)(pay >> bin_shift);
  if (sh >= 64) {
    hi &= (1ull << (sh - 64)) - 1ull;
  } else {
    lo &= (1ull << sh) - 1ull;
    hi = 0;
  }
  w[0] = spread3((uint32_t)lo & 0xffffffu);
  w[1] = spread3((uint32_t)(lo >> 24) & 0xffffffu);
  w[2] = spread3((uint32_t)((lo >> 48) | (hi << 16)) & 0xffffffu);
  w[3] = spread3((uint32_t)(hi >> 8) & 0xffffffu);
}

// The 4-bit codes of a 3-bit coded entry: every escaped column (code 7: depth 7 or more) hashed
// again for min(depth, 11). Out of line: about one entry in five at 28 columns has an escape.
static __device__ __noinline__ uint4 fix_escapes3(uint4 w4, uint64_t pm, const uint64_t *kcol, uint32_t cap) {
  uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    // nibbles <= 7: adding 1 carries into bit 3 of a nibble exactly when it is 7
    for (uint32_t f = (w[g] + 0x11111111u) & 0x88888888u; f; f &= f - 1) {
      const uint32_t k = (__ffs(f) - 1) >> 2;  // nibble index in the word
      const uint32_t code = depth_code(pm ^ kcol[8 * g + k], cap);
      w[g] = (w[g] & ~(15u << (4 * k))) | (code << (4 * k));
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// ------------------------------------------------------------------------------------------------
// bucket-plane sketch update
// ------------------------------------------------------------------------------------------------
// (No memory clobber: the planes are touched by assembly alone, ordered by its volatility and the CTA
// barriers, and other loads may move across.)
__device__ __forceinline__ void red_xor_shared(uint32_t addr, uint32_t v) {
  asm volatile("red.shared.xor.b32 [%0], %1;" ::"r"(addr), "r"(v));
}
// The same slot's checksum.
__device__ __forceinline__ void red_xor_shared_g(uint32_t addr, uint32_t v) {
  asm volatile("red.shared.xor.b32 [%0+%2], %1;" ::"r"(addr), "r"(v), "n"(kGOff));
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// First row (shared-memory address / 256) of the planes of vertex vl of a tile whose planes start at
// row r0: pairs of planes back to back, none across a 64 KB boundary.
__device__ __forceinline__ uint32_t pair_row(uint32_t r0, uint32_t vl) {
  uint32_t r = r0;
  for (;;) {
    const uint32_t fit = (256u - (r & 255u)) / kPairRows;  // pairs before the boundary
    if (vl < fit) return r + vl * kPairRows;
    vl -= fit;
    r = (r | 255u) + 1;
  }
}

// Bits 4n + 3 of the nibbles n holding the escape code (codes do not exceed it).
__device__ __forceinline__ uint32_t deep_codes(uint32_t w) {
  static_assert(kDepthEscape == 11 && kDepthEscape == kPlaneThr, "11: bits 3, 1 and 0; the last plane row");
  return w & (w << 2) & (w << 3) & 0x88888888u;
}

// Bucket of a sketch in HBM, three 32-bit atomics (alpha low, alpha high, gamma).
__device__ __forceinline__ void xor_bucket_global(uint32_t *sk, uint32_t bucket, uint32_t lo,
                                                  uint32_t hi, uint32_t chk) {
  uint32_t *p = sk + 3 * bucket;
  atomicXor(p, lo);
  atomicXor(p + 1, hi);
  atomicXor(p + 2, chk);
}

// The columns of an entry whose code is the escape (depth 11 or more): XORed into HBM at their exact
// depth (CubeSketch: at every depth from the last row's on). They went to the planes' last row,
// which CubeSketch needs to hold exactly the depths below B: a depth of B is taken out of it again
// (last_row: address of slot 0 of that row). kcol and c0: the group's columns.
template <bool CUBE>
__device__ __forceinline__ void apply_deep(const uint32_t (&c4)[4], uint64_t pm, uint32_t v, uint32_t u,
                                           uint32_t chk, uint32_t *sk, const uint64_t *kcol, uint32_t c0,
                                           uint32_t B, uint32_t last_row) {
  const uint32_t lo = max(u, v), hi = min(u, v);
#pragma unroll 1
  for (int w = 0; w < 4; ++w) {
    for (uint32_t f = deep_codes(w == 0 ? c4[0] : w == 1 ? c4[1] : w == 2 ? c4[2] : c4[3]); f; f &= f - 1) {
      const uint32_t c = 8 * w + ((__ffs(f) - 1) >> 2);
      const uint32_t d = depth_exact(pm ^ kcol[c], B);
      if (CUBE) {
        if (d < B) {
          for (uint32_t j = kPlaneThr; j <= d; ++j) xor_bucket_global(sk, (c0 + c) * B + j, lo, hi, chk);
        } else {
          red_xor_shared(last_row + 4 * c, u | 0x80000000u);
          red_xor_shared_g(last_row + 4 * c, chk);
        }
      } else if (d < B) {
        xor_bucket_global(sk, (c0 + c) * B + d, lo, hi, chk);
      }
    }
  }
}

// nibble t of the result = nibble t ^ (lane & 30) of the input (byte in the word, word; the lowest
// index bit is taken where the nibbles are widened)
__device__ __forceinline__ void permute_codes(uint32_t (&c4)[4], uint32_t lane) {
  const uint32_t q = (lane >> 1) & 3u;
  const uint32_t sel = q | ((1u ^ q) << 4) | ((2u ^ q) << 8) | ((3u ^ q) << 12);
#pragma unroll
  for (int w = 0; w < 4; ++w) c4[w] = prmt(c4[w], 0, sel);
  if (lane & 8) {
    uint32_t x = c4[0]; c4[0] = c4[1]; c4[1] = x;
    x = c4[2]; c4[2] = c4[3]; c4[3] = x;
  }
  if (lane & 16) {
    uint32_t x = c4[0]; c4[0] = c4[2]; c4[2] = x;
    x = c4[1]; c4[1] = c4[3]; c4[3] = x;
  }
}

// The 32 slot steps of one entry per lane: codes c4 (already permuted), plane starting at row `row`.
__device__ __forceinline__ void slot_steps(const uint32_t (&c4)[4], uint32_t row, uint32_t val,
                                           uint32_t chk, uint32_t lane) {
  const uint32_t radd = (row & 255u) * 0x01010101u;
  const uint32_t base = ((row >> 8) << 16) | (lane << 2), odd = 4 * (lane & 1);
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    // one byte per step: the row inside the plane's 64 KB block
    const uint32_t ev = ((c4[w] >> odd) & 0x0f0f0f0fu) + radd, od = ((c4[w] >> (4 - odd)) & 0x0f0f0f0fu) + radd;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t t = 8 * w + j;
      // byte 1: the row; byte 0: the slot; the plane's block
      const uint32_t a = prmt((j & 1) ? od : ev, base ^ (t << 2), 0x7604u | ((uint32_t)(j >> 1) << 4));
      red_xor_shared(a, val);
      red_xor_shared_g(a, chk);
    }
  }
}

// Vertex, neighbour, premixed index and codes (of the group's nc columns, constants kcol) of a gutter
// entry of bin `bin`: unpacked from a coded entry (3-bit codes: escapes hashed again), or hashed here
// for a plain {vertex, neighbour} entry.
template <int KIND>
__device__ __forceinline__ void decode_entry(uint4 e, uint32_t bin, const PlaneGeom &g, uint32_t cap,
                                             const uint64_t *kcol, uint32_t nc, uint32_t &v, uint32_t &u,
                                             uint64_t &pm, uint32_t (&c4)[4]) {
  if (KIND == kEntryCoded) {
    unpack_entry(e, bin, g.C, g.bin_shift, v, u, c4);
  } else if (KIND == kEntryCoded3) {
    unpack_entry3(e, bin, g.C, g.bin_shift, v, u, c4);
  } else {
    v = e.x;
    u = e.y;
  }
  pm = xxh3_premix(((uint64_t)max(u, v) << 32) | min(u, v));  // idx = (min << 32) | max
  if (KIND == kEntryCoded3) {
    const uint32_t esc = ((c4[0] + 0x11111111u) | (c4[1] + 0x11111111u) | (c4[2] + 0x11111111u) |
                          (c4[3] + 0x11111111u)) & 0x88888888u;
    if (esc) {
      const uint4 w = fix_escapes3(make_uint4(c4[0], c4[1], c4[2], c4[3]), pm, kcol, cap);
      c4[0] = w.x;
      c4[1] = w.y;
      c4[2] = w.z;
      c4[3] = w.w;
    }
  } else if (KIND == kEntryPlain) {
    all_codes<0>(pm, kcol, nc, cap, c4);
  }
}

// Vertex of a gutter entry of bin `bin` (for filtering a bin's entries by tile).
template <int KIND>
__device__ __forceinline__ uint32_t entry_vertex(uint4 e, uint32_t bin, const PlaneGeom &g) {
  if (KIND == kEntryPlain) return e.x;
  if (KIND == kEntryCoded && g.C <= kWordCodes) return (bin << g.bin_shift) | (e.w & ((1u << g.bin_shift) - 1u));
  const uint64_t pay = KIND == kEntryCoded3 ? payload3(e, g.C)
                                            : (((uint64_t)e.w << 32) | e.z) >> (4 * g.C - 64);
  return (bin << g.bin_shift) | ((uint32_t)pay & ((1u << g.bin_shift) - 1u));
}

template <int KIND>
__device__ __forceinline__ uint4 load_entry(const uint8_t *cb, uint32_t i) {
  if (KIND != kEntryPlain) return reinterpret_cast<const uint4 *>(cb)[i];
  const uint2 k = reinterpret_cast<const uint2 *>(cb)[i];
  return make_uint4(k.x, k.y, 0, 0);
}

// What a CTA works on: one group of columns of one tile.
struct PlaneItem {
  uint32_t t, bin, c0, nc;  // tile, its bin, the group's first column and number of columns
  const uint64_t *kcol;     // the group's hash constants
  uint32_t *gsk;
  const uint32_t *row_of;   // first row of each vertex's planes
  uint32_t *deep;           // bit l of word j: entry 32 j + l of the segment has an escape code
};
// Entries are taken in segments of 64 groups of 32 a warp; each warp looks at the escapes among its entries of
// a segment (about 1 entry in 85 at 24 columns) together, after its last slot step.
__host__ __device__ constexpr uint32_t deep_words(uint32_t threads) { return 2 * threads; }

// An entry ready for its slot steps.
struct Ready {
  uint32_t c4[4], row, val, chk;
};

// A coded entry's escape codes are flagged (deep); a plain entry's, whose codes would have to be
// hashed again later, are applied here.
template <int KIND, bool CUBE>
__device__ __forceinline__ Ready ready_entry(uint4 en, bool valid, const PlaneItem &x, const PlaneGeom &g,
                                             uint64_t kchk, uint32_t cap, uint32_t tile_mask, uint32_t lane,
                                             bool &deep) {
  Ready r;
  uint32_t v, u;
  uint64_t pm;
  decode_entry<KIND>(en, x.bin, g, cap, x.kcol, x.nc, v, u, pm, r.c4);
  r.chk = tail_lo32(pm ^ kchk);
  r.val = u | 0x80000000u;
  r.row = x.row_of[v & tile_mask] + (u > v ? 0u : kPlaneRows);  // plane A or B
  deep = (deep_codes(r.c4[0]) | deep_codes(r.c4[1]) | deep_codes(r.c4[2]) | deep_codes(r.c4[3])) != 0;
  if (KIND == kEntryPlain) {
    if (deep && valid)
      apply_deep<CUBE>(r.c4, pm, v, u, r.chk, x.gsk + (uint64_t)v * g.sketch_words, x.kcol, x.c0, g.B,
                       (r.row + kPlaneThr) * kRowBytes);
    deep = false;
  }
  permute_codes(r.c4, lane);
  return r;
}

// Entries [b, e) of one gutter chunk (at cb; coded ones: at most 32 deep_words(threads) of them) into the planes of the
// item's tile.
template <int KIND, bool CUBE>
__device__ __forceinline__ void plane_chunk(const PlaneItem &x, const PlaneGeom &g, uint64_t kchk, uint32_t cap,
                                            const uint8_t *cb, uint32_t b, uint32_t e, uint32_t *queue) {
  const uint32_t nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tile_mask = (1u << g.tile_shift) - 1, step = nwarps * 32;
  // word j of this warp's escape mask: bit l of word warp + j nwarps, entry b + 32 word + l
  auto deep_entries = [&]() {
    __syncwarp();
    for (uint32_t j = warp + lane * nwarps; j < (e - b + 31) / 32; j += step)
      for (uint32_t m = x.deep[j]; m; m &= m - 1) {
        uint32_t v, u, c4[4];
        uint64_t pm;
        decode_entry<KIND>(load_entry<KIND>(cb, b + 32 * j + __ffs(m) - 1), x.bin, g, cap, x.kcol, x.nc, v, u, pm,
                           c4);
        if ((v >> g.tile_shift) != x.t) continue;
        const uint32_t row = x.row_of[v & tile_mask] + (u > v ? 0u : kPlaneRows);
        apply_deep<CUBE>(c4, pm, v, u, tail_lo32(pm ^ kchk), x.gsk + (uint64_t)v * g.sketch_words, x.kcol, x.c0,
                         g.B, (row + kPlaneThr) * kRowBytes);
      }
    __syncwarp();
  };
  if (g.bin_shift == g.tile_shift) {
    // the bin is this tile: every entry applies. A warp's slot steps of one group of 32 entries (LSU)
    // are issued between the arithmetic that makes the next group ready (ALU), and the group after
    // that is being loaded. Lanes past the end repeat the last entry with nothing to XOR.
    uint32_t i = b + warp * 32 + lane;
    if (i - lane >= e) return;
    uint32_t word = warp;
    bool deep, any = false;
    auto load = [&](uint32_t k) { return load_entry<KIND>(cb, min(k, e - 1)); };
    uint4 nx = load(i);
    Ready r = ready_entry<KIND, CUBE>(nx, i < e, x, g, kchk, cap, tile_mask, lane, deep);
    nx = load(i + step);
    for (;; i += step, word += nwarps) {
      if (KIND != kEntryPlain) {
        const uint32_t m = __ballot_sync(kFull, deep && i < e);
        if (lane == 0) x.deep[word] = m;
        any = any || m;
      }
      if (i - lane + step >= e) break;
      const Ready q = r;
      r = ready_entry<KIND, CUBE>(nx, i + step < e, x, g, kchk, cap, tile_mask, lane, deep);
      nx = load(i + 2 * step);
      slot_steps(q.c4, q.row, q.val, q.chk, lane);
    }
    const bool in = i < e;
    slot_steps(r.c4, r.row, in ? r.val : 0u, in ? r.chk : 0u, lane);
    if (KIND != kEntryPlain && any) deep_entries();
  } else {
    // the bin holds several tiles: each warp ballots its group, queues the indices of this tile's
    // entries, and applies full warps of queued ones; two groups are in flight ahead of the one
    // ballotted. The escape mask has the word of the group that an entry was found in.
    uint32_t i0 = b + warp * 32, qn = 0;
    if (KIND != kEntryPlain)
      for (uint32_t j = warp + lane * nwarps; j < (e - b + 31) / 32; j += step) x.deep[j] = 0;
    __syncwarp();
    bool any = false;
    auto apply = [&](uint32_t i, bool valid) {
      bool deep;
      const Ready r = ready_entry<KIND, CUBE>(load_entry<KIND>(cb, i), valid, x, g, kchk, cap, tile_mask, lane, deep);
      if (KIND != kEntryPlain) {
        if (valid && deep) atomicOr(&x.deep[(i - b) >> 5], 1u << ((i - b) & 31));
        any = __any_sync(kFull, any || (valid && deep));
      }
      slot_steps(r.c4, r.row, valid ? r.val : 0u, valid ? r.chk : 0u, lane);
    };
    auto tile_at = [&](uint32_t i) {
      return i < e ? entry_vertex<KIND>(load_entry<KIND>(cb, i), x.bin, g) >> g.tile_shift : ~x.t;
    };
    uint32_t nx = tile_at(i0 + lane), nx2 = tile_at(i0 + step + lane);
    for (; i0 < e; i0 += step) {
      const bool mine = nx == x.t;
      nx = nx2;
      nx2 = tile_at(i0 + 2 * step + lane);
      const uint32_t m = __ballot_sync(kFull, mine);
      if (mine) queue[qn + __popc(m & ((1u << lane) - 1u))] = i0 + lane;
      qn += __popc(m);
      __syncwarp();
      if (qn >= 32) {
        const uint32_t q = queue[lane];
        __syncwarp();
        qn -= 32;
        if (lane < qn) queue[lane] = queue[32 + lane];
        __syncwarp();
        apply(q, true);
      }
    }
    if (qn) {
      const uint32_t q = queue[lane < qn ? lane : 0];
      __syncwarp();
      apply(q, lane < qn);
    }
    if (KIND != kEntryPlain && any) deep_entries();
  }
}

// One endpoint update XORed into the sketch sk in HBM by a whole warp: lane l < nc holds the depth
// of column l (nothing to do when it is B or more), lane nc stands for the deterministic bucket.
// The buckets' words are dealt over the lanes three to a bucket, so a bucket is one request to L2
// instead of three.
__device__ __forceinline__ void warp_update_global(uint32_t *sk, uint32_t nc, uint32_t depth,
                                                   uint32_t B, uint32_t lo, uint32_t hi, uint32_t chk) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t off = lane < nc ? (depth < B ? 3 * (lane * B + depth) : 0xffffffffu) : 3 * nc * B;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const uint32_t f = i * 32 + lane, bk = f / 3, kk = f - 3 * bk;
    const uint32_t o = __shfl_sync(kFull, off, bk);
    if (bk <= nc && o != 0xffffffffu) atomicXor(sk + o + kk, kk == 0 ? lo : kk == 1 ? hi : chk);
  }
}

// A whole record (u != v) by a warp: hashed once -- kc is the constant of the lane's column (lanes past
// the columns: any) -- and XORed into both endpoints' sketches su and sv.
__device__ __forceinline__ void warp_record_global(uint32_t *su, uint32_t *sv, uint32_t u, uint32_t v, uint32_t C,
                                                   uint32_t B, uint64_t kc, uint64_t kchk) {
  const uint32_t lo = max(u, v), hi = min(u, v);
  const uint64_t pm = xxh3_premix(((uint64_t)lo << 32) | hi);
  const uint32_t depth = depth_exact(pm ^ kc, B), chk = tail_lo32(pm ^ kchk);
  warp_update_global(su, C, depth, B, lo, hi, chk);
  warp_update_global(sv, C, depth, B, lo, hi, chk);
}

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v));
}

// Write-back of one vertex's planes (A at shared address pa, B behind it) by one warp, and their
// clearing for the next tile. col: the group's first column in the sketch; its nc columns start 3 B
// words apart, and rows 0 .. R - 1 come from the planes, 3 R words a column; the deterministic bucket
// is the first row of slot det (none in this group when det is 32 or more). Lane by column, a lane
// turns its slot's rows into sketch words (every lane its own bank); the words are then laid down in
// the order of the sketch over the planes themselves and taken in that order, so that a warp's
// reductions go to consecutive words of HBM. Zero words are left alone. (6e7 records at 2^17 vertices /
// 1.28e7 at 2^20: 1.51 / 2.86 ms; a read-modify-write with 13 words in flight per lane 1.62 / 3.47,
// with 6 1.58 / 3.12. Reading the planes in the order of the sketch is a 14-way bank conflict: 16 us a
// tile of 32 vertices.)
// sparse: few entries, so the rows past the deepest one in use are looked for and left out.
template <bool CUBE>
__device__ __forceinline__ void write_back(uint32_t pa, uint32_t vg, uint32_t *col, uint32_t nc, uint32_t det,
                                           uint32_t B, uint32_t lane, bool sparse) {
  constexpr uint32_t pb = kPlaneRows * kRowBytes;
  uint32_t R = min(B, kPlaneThr), used = 0;
  const uint32_t at = pa + 4 * lane;
  const bool mine = lane < nc || lane == det;
  uint32_t w[3 * kPlaneThr];
  uint32_t s[4] = {0, 0, 0, 0};
  if (CUBE && B > kPlaneThr) {  // the depths from kPlaneThr to B - 1
    s[0] = lds32(at + kPlaneThr * kRowBytes);
    s[1] = lds32(at + kPlaneThr * kRowBytes + kGOff);
    s[2] = lds32(at + pb + kPlaneThr * kRowBytes);
    s[3] = lds32(at + pb + kPlaneThr * kRowBytes + kGOff);
  }
#pragma unroll
  for (int r = kPlaneThr - 1; r >= 0; --r) {
    uint32_t a = 0, ga = 0, b = 0, gb = 0;
    if (mine && (uint32_t)r < R) {
      const uint32_t o = at + r * kRowBytes;
      a = lds32(o);
      ga = lds32(o + kGOff);
      b = lds32(o + pb);
      gb = lds32(o + pb + kGOff);
    }
    if (CUBE && lane != det) {
      // CubeSketch: bucket d of a column takes every update of depth d or more
      // (src/sketch.cpp:50-67), the suffix XOR over the rows
      a = s[0] ^= a;
      ga = s[1] ^= ga;
      b = s[2] ^= b;
      gb = s[3] ^= gb;
    }
    w[3 * r] = (a & 0x7fffffffu) ^ ((b >> 31) ? vg : 0u);
    w[3 * r + 1] = (b & 0x7fffffffu) ^ ((a >> 31) ? vg : 0u);
    w[3 * r + 2] = ga ^ gb;
    used |= a | b | ga | gb ? 1u << r : 0u;
  }
  if (sparse) R = 32 - __clz(__reduce_or_sync(kFull, used));
  else __syncwarp();
  if (!R) return;
  const uint32_t run = 3 * R;
  const uint32_t list = nc * run + (det < 32 ? 3u : 0u);  // words; the deterministic bucket's last
#pragma unroll
  for (int i = 0; i < 3 * (int)kPlaneThr; ++i)
    if ((lane < nc && (uint32_t)i < run) || (lane == det && i < 3)) sts32(pa + 4 * (lane * run + i), w[i]);
  __syncwarp();
  // word k of its column, at offset off in the sketch; 32 words on, that is dc columns and dk words
  const uint32_t dc = 32 / run, dk = 32 - dc * run, doff = 3 * dc * B + dk, dwrap = 3 * B - run;
  const uint32_t c = lane / run;
  uint32_t k = lane - c * run, off = 3 * c * B + k;
#pragma unroll 4
  for (uint32_t i = lane; i < list; i += 32) {
    const uint32_t y = lds32(pa + 4 * i);
    if (y) atomicXor(col + off, y);
    k += dk;
    off += doff;
    if (k >= run) {
      k -= run;
      off += dwrap;
    }
  }
  __syncwarp();
#pragma unroll
  for (uint32_t i = 0; i < kPairRows * kRowBytes / 512; ++i)
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(pa + i * 512 + lane * 16), "r"(0u));
}

}  // namespace dev
}  // namespace gz
