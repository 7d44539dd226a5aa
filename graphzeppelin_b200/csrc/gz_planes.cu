// gz_planes.cu -- coded-entry record ingest for CameoSketch sketches of at most 31 columns.
//
// Sketch::update (src/sketch.cpp:69-83) XORs an edge index and its checksum into the
// deterministic bucket and into bucket (c, depth_c(idx)) of every column c, and
// CCSketchAlg::update / apply_update_batch (src/cc_sketch_alg.cpp:106-133) apply it to both
// endpoint sketches. Every vertex sketch uses the same seed (src/cc_sketch_alg.cpp:21), so the two
// endpoints get the same depths and the same checksum.
//
//   k_hash_sort_scatter  per tile of records: the two endpoint entries counting-sorted by gutter
//                        bin in shared memory, each record's C column depths hashed once into
//                        4-bit (or 3-bit) codes carried by both entries, the runs written out
//                        coalesced.
//   k_plane_update       per tile of W vertices: the tile's entries (filtered out of their gutter
//                        bin when a bin holds several tiles) XORed into bucket planes in shared
//                        memory that start at zero, then each vertex's rows XORed into its sketch
//                        in HBM. The checksum is hashed here, per entry.
// A coded entry is 128 bits: the C codes in bits 0 .. 4C - 1 (column c in bits 4c .. 4c + 3),
// then the neighbour shifted left by bin_shift bits OR the vertex's offset inside its gutter bin
// (the bin is known from where the entry lies). It is used when 4C + bin_shift + the neighbour's
// bits fit in 128 (every CameoSketch up to 2^18 vertices). Past that, codes of 3 bits (code 7 =
// depth 7 or more) fit larger graphs (3C + bin_shift + neighbour bits <= 128: 2^20 vertices and
// far beyond); an escaped column (1 in 128 column updates) is hashed again where the entry is
// applied, so the planes see the same 4-bit codes either way.
//
// Bucket planes. A warp takes 32 entries, one per lane. At step t = 0..31 lane l handles slot
// l ^ t of its entry: slot s < C is column s, slot C the deterministic bucket, higher slots are
// unused (sketches of more columns go in groups of 32 slots, one pass over the entries each). A
// plane row holds 32 slots, so slot s is shared-memory bank s and the 32 lanes of a step hit 32
// different banks whatever their vertices and depths: the red.shared.xor never conflict (the
// per-entry ordering, every lane on column c at once, concentrates lanes on a few banks because
// depth 0 takes half the updates). Each bucket is kept as three words,
//   A = XOR of (neighbour | 1 << 31) over the entries whose neighbour is above the vertex,
//   B = the same over the other entries,
//   G = XOR of their checksums,
// so one update XORs two words (A or B, and G) instead of three. With idx = (min << 32) | max
// (concat_pairing_fn, src/util.cpp:45-51) the bucket's alpha is recovered as
//   alpha low  = low31(A) ^ (top bit of B ? vertex : 0),
//   alpha high = low31(B) ^ (top bit of A ? vertex : 0),
// the top bits holding the parity of each kind's entry count (vertex ids are below 2^31).
// Rows hold depths 0 .. kPlaneRows - 2; the last row collects the depths at or above it (2^-11 of
// the column updates), which are XORed into the sketch in HBM with global atomics; those rows are
// never touched by the write-back, which changes only the rows the planes hold.
//
// What bounds the update: shared-memory issue. A slot step is two red.shared.xor, one wavefront
// each, 64 wavefronts per 32 entries and SM. The address of a step is made by one byte permute
// and one XOR: a row is 256 bytes -- 32 slots of A (or B), then the same slots' checksums, reached with
// an immediate offset of 128 -- so that address byte 0 is the slot, byte 1 the row (the code plus the
// plane's first row, added to four codes at once; planes never straddle a 64 KB boundary), and the
// rest the plane's 64 KB block.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "gz_common.cuh"
#include "gz_device.cuh"
#include "gz_kernels.cuh"

namespace gz {

namespace {

using namespace gz::dev;

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
__device__ __noinline__ uint4 fix_escapes3(uint4 w4, uint64_t pm, const uint64_t *kcol, uint32_t cap) {
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
// hash sort-scatter (records in, coded entries out)
// ------------------------------------------------------------------------------------------------
// Per tile of rec_tile records: stage them (coalesced 128-bit loads), count their endpoint entries
// per bin, reserve one run per non-empty bin in the gutter (one global atomic each), hash every
// record's C columns once, place both entries (and their bins) in bin order in shared memory,
// and write the runs out.
// Exclusive scan over the threads of a block of NT threads (a multiple of 32, <= 1024).
template <int NT>
__device__ __forceinline__ uint32_t block_scan(uint32_t x, uint32_t *ws /*32*/) {
  if (NT == 1024) return block_scan_1024(x, ws);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, inc, o);
    if (lane >= (uint32_t)o) inc += y;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < NT / 32 ? ws[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, w, o);
      if (lane >= (uint32_t)o) w += y;
    }
    ws[lane] = w;
  }
  __syncthreads();
  const uint32_t r = (warp ? ws[warp - 1] : 0u) + inc - x;
  __syncthreads();
  return r;
}

// C3: 3-bit codes (kEntryCoded3), else 4-bit (kEntryCoded).
template <int RPT, int NT, bool C3>
__global__ void __launch_bounds__(NT, 1024 / NT)
k_hash_sort_scatter(const uint8_t *__restrict__ rec, uint64_t n, GutterGeom g, PlaneHash ph,
                    uint32_t rec_tile, const uint64_t *__restrict__ base,
                    uint32_t *__restrict__ fill, uint4 *__restrict__ entries) {
  extern __shared__ __align__(16) uint8_t gsm[];
  __shared__ uint32_t ws[32];
  const uint32_t nb = g.nbins, nb4 = (nb + 3) & ~3u;
  uint32_t *s_cur = reinterpret_cast<uint32_t *>(gsm);  // counts, then placement cursors
  uint32_t *s_rel = s_cur + nb4;  // a bin's run: gutter position minus position in the tile
  uint4 *s_ent = reinterpret_cast<uint4 *>(s_rel + nb4);
  uint16_t *s_bin = reinterpret_cast<uint16_t *>(s_ent + 2 * (size_t)rec_tile);  // bin of each entry
  // the staged records share the entry area: they are parsed into registers before the first
  // entry is placed, and the next tile is staged only after the write-out
  uint8_t *s_rec = reinterpret_cast<uint8_t *>(s_ent);
  const uint32_t per_thread = (nb + NT - 1) / NT;  // bins per thread
  const uint32_t cap = 1u << min(ph.B, C3 ? kDepthEscape3 : kDepthEscape);
  for (uint64_t t0 = blockIdx.x * (uint64_t)rec_tile; t0 < n; t0 += (uint64_t)gridDim.x * rec_tile) {
    const uint32_t cnt = (uint32_t)(n - t0 < rec_tile ? n - t0 : rec_tile);
    for (uint32_t b = threadIdx.x; b < nb; b += blockDim.x) s_cur[b] = 0u;
    const uint32_t shift = stage_records(rec, t0, cnt, s_rec);
    __syncthreads();
    // 1. this thread's records into registers, then their per-bin counts
    uint32_t ru[RPT], rv[RPT];
#pragma unroll
    for (int k = 0; k < RPT; ++k) {
      const uint32_t i = threadIdx.x + k * blockDim.x;
      ru[k] = rv[k] = 0xffffffffu;
      if (i < cnt) {
        parse_record(s_rec, shift, i, ru[k], rv[k]);
        if (ru[k] >= g.V || rv[k] >= g.V) ru[k] = 0xffffffffu;  // dropped (the count pass flags it)
      }
    }
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (ru[k] != 0xffffffffu) {
        atomicAdd(&s_cur[ru[k] >> g.bin_shift], 1u);
        atomicAdd(&s_cur[rv[k] >> g.bin_shift], 1u);
      }
    __syncthreads();
    // 2. run offsets inside the tile (bins [tid*per_thread, +per_thread) per thread) and one run
    //    reserved per non-empty bin in the gutter
    uint32_t sum = 0;
    for (uint32_t k = 0; k < per_thread; ++k) {
      const uint32_t b = threadIdx.x * per_thread + k;
      sum += b < nb ? s_cur[b] : 0u;
    }
    uint32_t run = block_scan<NT>(sum, ws);
    for (uint32_t k = 0; k < per_thread; ++k) {
      const uint32_t b = threadIdx.x * per_thread + k;
      if (b < nb) {
        const uint32_t c = s_cur[b];
        s_rel[b] = c ? (uint32_t)base[b] + atomicAdd(&fill[b], c) - run : 0u;
        s_cur[b] = run;
        run += c;
      }
    }
    __syncthreads();
    // 3. slots claimed, each record hashed once, both endpoint entries placed in bin order
    uint32_t pu[RPT], pv[RPT];
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (ru[k] != 0xffffffffu) {
        pu[k] = atomicAdd(&s_cur[ru[k] >> g.bin_shift], 1u);
        pv[k] = atomicAdd(&s_cur[rv[k] >> g.bin_shift], 1u);
      }
#pragma unroll
    for (int k = 0; k < RPT; ++k)
      if (ru[k] != 0xffffffffu) {
        const uint32_t lo = max(ru[k], rv[k]), hi = min(ru[k], rv[k]);
        const uint64_t pm = xxh3_premix(((uint64_t)lo << 32) | hi);
        uint32_t w[4];
        all_codes<18>(pm, ph.kcol, ph.C, cap, w);
        s_ent[pu[k]] = C3 ? pack_entry3(w, ru[k], rv[k], ph.C, g.bin_shift)
                          : pack_entry(w, ru[k], rv[k], ph.C, g.bin_shift);
        s_ent[pv[k]] = C3 ? pack_entry3(w, rv[k], ru[k], ph.C, g.bin_shift)
                          : pack_entry(w, rv[k], ru[k], ph.C, g.bin_shift);
        s_bin[pu[k]] = (uint16_t)(ru[k] >> g.bin_shift);
        s_bin[pv[k]] = (uint16_t)(rv[k] >> g.bin_shift);
      }
    __syncthreads();
    // 4. coalesced write-out of the runs
    const uint32_t total = s_cur[nb - 1];
    for (uint32_t j = threadIdx.x; j < total; j += blockDim.x) entries[s_rel[s_bin[j]] + j] = s_ent[j];
    __syncthreads();
  }
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

template <int KIND>
__device__ __forceinline__ Ready ready_entry(uint4 en, const PlaneItem &x, const PlaneGeom &g, uint64_t kchk,
                                             uint32_t cap, uint32_t tile_mask, uint32_t lane, bool &deep) {
  Ready r;
  uint32_t v, u;
  uint64_t pm;
  decode_entry<KIND>(en, x.bin, g, cap, x.kcol, x.nc, v, u, pm, r.c4);
  r.chk = tail_lo32(pm ^ kchk);
  r.val = u | 0x80000000u;
  r.row = x.row_of[v & tile_mask] + (u > v ? 0u : kPlaneRows);  // plane A or B
  deep = (deep_codes(r.c4[0]) | deep_codes(r.c4[1]) | deep_codes(r.c4[2]) | deep_codes(r.c4[3])) != 0;
  permute_codes(r.c4, lane);
  return r;
}

// Entries [b, e) of one gutter chunk (at cb; at most 32 deep_words(threads) of them) into the planes of the
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
    Ready r = ready_entry<KIND>(nx, x, g, kchk, cap, tile_mask, lane, deep);
    nx = load(i + step);
    for (;; i += step, word += nwarps) {
      const uint32_t m = __ballot_sync(kFull, deep && i < e);
      if (lane == 0) x.deep[word] = m;
      any = any || m;
      if (i - lane + step >= e) break;
      const Ready q = r;
      r = ready_entry<KIND>(nx, x, g, kchk, cap, tile_mask, lane, deep);
      nx = load(i + 2 * step);
      slot_steps(q.c4, q.row, q.val, q.chk, lane);
    }
    const bool in = i < e;
    slot_steps(r.c4, r.row, in ? r.val : 0u, in ? r.chk : 0u, lane);
    if (any) deep_entries();
  } else {
    // the bin holds several tiles: each warp ballots its group, queues the indices of this tile's
    // entries, and applies full warps of queued ones; two groups are in flight ahead of the one
    // ballotted. The escape mask has the word of the group that an entry was found in.
    uint32_t i0 = b + warp * 32, qn = 0;
    for (uint32_t j = warp + lane * nwarps; j < (e - b + 31) / 32; j += step) x.deep[j] = 0;
    __syncwarp();
    bool any = false;
    auto apply = [&](uint32_t i, bool valid) {
      bool deep;
      const Ready r = ready_entry<KIND>(load_entry<KIND>(cb, i), x, g, kchk, cap, tile_mask, lane, deep);
      if (valid && deep) atomicOr(&x.deep[(i - b) >> 5], 1u << ((i - b) & 31));
      any = __any_sync(kFull, any || (valid && deep));
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
    if (any) deep_entries();
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

// Sparse calls (few updates for the graph's size): every record hashed once, a warp per record and
// a lane per column, and XORed into both endpoints' sketches in HBM: one launch, no gutter.
// (A self-loop XORs one sketch twice: no change, as through the gutter.)
__global__ void __launch_bounds__(256)
k_direct_records(const uint8_t *__restrict__ rec, uint64_t n, uint32_t V, uint32_t sketch_words,
                 PlaneHash ph, uint32_t *__restrict__ sk, uint32_t *__restrict__ status) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t kc = lane < ph.C ? ph.kcol[lane] : ph.kchk;
  for (uint64_t i = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; i < n; i += nwarps) {
    uint32_t u, v;
    load_record(rec, rec + 9 * n, i, u, v);
    if (u >= V || v >= V) {
      if (lane == 0) atomicOr(status, kStatusBadVertex);
      continue;
    }
    if (u == v) continue;
    const uint32_t lo = max(u, v), hi = min(u, v);
    const uint64_t pm = xxh3_premix(((uint64_t)lo << 32) | hi);
    const uint32_t depth = depth_exact(pm ^ kc, ph.B);
    const uint32_t chk = tail_lo32(pm ^ ph.kchk);
    warp_update_global(sk + (uint64_t)u * sketch_words, ph.C, depth, ph.B, lo, hi, chk);
    warp_update_global(sk + (uint64_t)v * sketch_words, ph.C, depth, ph.B, lo, hi, chk);
  }
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
// the order of the sketch over the planes themselves and taken in that order, so that the lanes read
// and write consecutive words in HBM, 13 of them in flight per lane. Zero words are left alone.
// (Global reductions instead run into L2's rate for them, about 45e9 sectors/s; reading the planes
// in the order of the sketch is a 14-way bank conflict: 16 us a tile of 32 vertices.)
template <bool CUBE>
__device__ __forceinline__ void write_back(uint32_t pa, uint32_t vg, uint32_t *col, uint32_t nc, uint32_t det,
                                           uint32_t B, uint32_t lane) {
  constexpr uint32_t pb = kPlaneRows * kRowBytes;
  const uint32_t R = min(B, kPlaneThr), run = 3 * R;
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
  }
  __syncwarp();
  const uint32_t list = nc * run + (det < 32 ? 3u : 0u);  // words; the deterministic bucket's last
#pragma unroll
  for (int i = 0; i < 3 * (int)kPlaneThr; ++i)
    if ((lane < nc && (uint32_t)i < run) || (lane == det && i < 3)) sts32(pa + 4 * (lane * run + i), w[i]);
  __syncwarp();
  uint32_t c = 0, k = lane;  // word k of column c
  while (k >= run) {
    k -= run;
    ++c;
  }
  for (uint32_t i0 = 0; i0 < list; i0 += 13 * 32) {
    uint32_t y[13], old[13], off[13];
#pragma unroll
    for (int j = 0; j < 13; ++j) {
      const uint32_t i = i0 + j * 32 + lane;
      y[j] = i < list ? lds32(pa + 4 * i) : 0u;
      off[j] = 3 * c * B + k;
      old[j] = y[j] ? __ldcg(col + off[j]) : 0u;
      k += 32;
      while (k >= run) {
        k -= run;
        ++c;
      }
    }
#pragma unroll
    for (int j = 0; j < 13; ++j)
      if (y[j]) col[off[j]] = old[j] ^ y[j];
  }
  __syncwarp();
#pragma unroll
  for (uint32_t i = 0; i < kPairRows * kRowBytes / 512; ++i)
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(pa + i * 512 + lane * 16), "r"(0u));
}

// The update kernel: persistent CTAs take (tile, group) items. CODED: entries of the coded path
// (sketches of one group of slots; plain entries come from apply_update_batch); otherwise plain
// entries only, hashed here. Threads and tile size come with the launch: one CTA of 1024 threads and
// 32 vertices per SM where the gutter's bins ask for large tiles; four of 256 threads and 8 vertices,
// whose phases overlap each other, otherwise.
template <bool CODED, bool CUBE, class Hash>
__global__ void __launch_bounds__(1024, 1)
k_plane_update(const __grid_constant__ PlaneGeom g, const __grid_constant__ Hash ph,
               uint8_t *__restrict__ sketches, const uint8_t *__restrict__ gutter,
               const __grid_constant__ ChunkTable chunks, const uint32_t *__restrict__ bin_off, int nchunks,
               uint32_t *work_counter) {
  extern __shared__ __align__(16) uint8_t dsm[];
  __shared__ uint32_t s_row[kPlaneMaxTile];
  __shared__ uint32_t s_claim[2][2];
  const uint32_t W = 1u << g.tile_shift;
  const uint32_t nwarps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t per_bin = g.bin_shift - g.tile_shift;  // log2(tiles per bin)
  const uint32_t s0 = (smem_u32(dsm) + kRowBytes - 1) & ~(kRowBytes - 1);
  // planes A and B of W vertices from s0 on, the escape mask, then the per-warp queues of filtered
  // entry indices
  uint32_t *deep = reinterpret_cast<uint32_t *>(dsm + (s0 - smem_u32(dsm)) + planes_bytes(g.tile_shift));
  uint32_t *queue = deep + deep_words(blockDim.x) + warp * kQueueSlots;
  const uint32_t C = g.C, B = g.B, cap = 1u << min(B, kDepthEscape);
  for (uint32_t q = threadIdx.x; q < W; q += blockDim.x) s_row[q] = pair_row(s0 >> 8, q);
  PlaneItem x;
  x.gsk = reinterpret_cast<uint32_t *>(sketches);
  x.row_of = s_row;
  x.deep = deep;
  const uint32_t stride = g.nbins + 1, nitems = g.ntiles * g.groups;
  for (uint32_t i = threadIdx.x; i < planes_bytes(g.tile_shift) / 16; i += blockDim.x)
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(s0 + i * 16), "r"(0u));
  auto claim = [&](uint32_t *to) {
    const uint32_t it = atomicAdd(work_counter, 1u);
    uint32_t total = 0;
    if (it < nitems) {
      const uint32_t bin = (it / g.groups) >> per_bin;
      for (int k = 0; k < nchunks; ++k)
        total += bin_off[(uint64_t)k * stride + bin + 1] - bin_off[(uint64_t)k * stride + bin];
    }
    to[0] = it;
    to[1] = total;  // entries of the tile's bin
  };
  if (threadIdx.x == 0) claim(s_claim[0]);
  for (uint32_t n = 0;; ++n) {
    __syncthreads();
    const uint32_t item = s_claim[n & 1][0], total = s_claim[n & 1][1];
    if (item >= nitems) break;
    if (threadIdx.x == 0) claim(s_claim[(n + 1) & 1]);  // while the others work on this one
    if (total == 0) continue;
    const uint32_t grp = g.groups == 1 ? 0u : item % g.groups;
    x.t = g.groups == 1 ? item : item / g.groups;
    x.bin = x.t >> per_bin;
    x.c0 = grp * kPlaneSlots;
    x.nc = min(C - x.c0, kPlaneSlots);
    x.kcol = ph.kcol + x.c0;
    const bool direct = !CUBE && total < (g.direct_max << per_bin);
    if (direct && grp) continue;
    for (int k = 0; k < nchunks; ++k) {
      const uint32_t b = bin_off[(uint64_t)k * stride + x.bin], e = bin_off[(uint64_t)k * stride + x.bin + 1];
      const uint8_t *cb = gutter + chunks.base[k];
      const uint32_t kind = CODED ? chunks.kind[k] : kEntryPlain;
      if (direct) {
        // few entries: each XORed in place in HBM by a warp, lane by column (no planes to write back)
        for (uint32_t i = b + warp; i < e; i += nwarps) {
          uint4 en;
          uint32_t v, u, w4[4];
          if (CODED && kind != kEntryPlain) {
            en = load_entry<kEntryCoded>(cb, i);
            if (kind == kEntryCoded) unpack_entry(en, x.bin, C, g.bin_shift, v, u, w4);
            else unpack_entry3(en, x.bin, C, g.bin_shift, v, u, w4);
          } else {
            en = load_entry<kEntryPlain>(cb, i);
            v = en.x;
            u = en.y;
          }
          if ((v >> g.tile_shift) != x.t) continue;
          const uint32_t lo = max(u, v), hi = min(u, v);
          const uint64_t pm = xxh3_premix(((uint64_t)lo << 32) | hi);
          warp_update_global(x.gsk + (uint64_t)v * g.sketch_words, C,
                             depth_exact(pm ^ x.kcol[min(lane, C - 1)], B), B, lo, hi, tail_lo32(pm ^ ph.kchk));
        }
        continue;
      }
      const uint32_t seg = 32 * deep_words(blockDim.x);
      for (uint32_t b1 = b; b1 < e; b1 += seg) {
        const uint32_t e1 = min(e, b1 + seg);
        if (CODED && kind == kEntryCoded) plane_chunk<kEntryCoded, CUBE>(x, g, ph.kchk, cap, cb, b1, e1, queue);
        else if (CODED && kind == kEntryCoded3) plane_chunk<kEntryCoded3, CUBE>(x, g, ph.kchk, cap, cb, b1, e1, queue);
        else plane_chunk<kEntryPlain, CUBE>(x, g, ph.kchk, cap, cb, b1, e1, queue);
      }
    }
    if (direct) continue;
    // the first lines of what the write-back reads are brought to L2 while the other warps finish
    for (uint32_t vl = warp; vl < W; vl += nwarps) {
      const uint32_t vg = (x.t << g.tile_shift) + vl;
      if (vg < g.V && lane < x.nc) {
        const uint32_t *p = x.gsk + (uint64_t)vg * g.sketch_words + 3 * (x.c0 + lane) * B;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
        if (total >= 64u << g.tile_shift) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 3 * min(B, kPlaneThr) - 1));
      }
    }
    __syncthreads();
    for (uint32_t vl = warp; vl < W; vl += nwarps) {
      const uint32_t vg = (x.t << g.tile_shift) + vl;
      if (vg >= g.V) break;
      write_back<CUBE>(s_row[vl] << 8, vg, x.gsk + (uint64_t)vg * g.sketch_words + 3 * (size_t)x.c0 * B, x.nc,
                       C - x.c0, B, lane);
    }
  }
}

// Register-only rate of the per-column hash above: eight independent chains per thread, each
// step a premixed input XOR a column constant, the rrmxmx tail and the depth code, the next input
// being this one XOR its code.
__global__ void k_plane_hash_peak(uint32_t iters, uint64_t *out) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  uint64_t y[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) y[k] = xxh3_premix(tid * 8 + k);
  uint32_t acc = 0;
  for (uint32_t i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t d = depth_code(y[k] ^ (0x9E3779B97F4A7C15ULL * (uint64_t)(k + 1)), 1u << kDepthEscape);
      acc += d;
      y[k] ^= d;
    }
  }
  uint64_t r = acc;
#pragma unroll
  for (int k = 0; k < 8; ++k) r ^= y[k];
  out[tid] = r;
}

// Rate of the plane update's shared-memory step alone: 32 vertices of planes, each thread one
// synthetic entry per iteration (codes 0..3, random vertex and plane), its 32 slot steps made
// exactly as the update makes them.
__global__ void __launch_bounds__(1024, 1) k_plane_update_peak(uint32_t iters, uint32_t *out) {
  extern __shared__ __align__(16) uint8_t dsm[];
  __shared__ uint32_t s_row[kPlaneMaxTile];
  const uint32_t s0 = (smem_u32(dsm) + kRowBytes - 1) & ~(kRowBytes - 1);
  const uint32_t lane = threadIdx.x & 31, words = planes_bytes(5) / 4;
  uint32_t *pw = reinterpret_cast<uint32_t *>(dsm + (s0 - smem_u32(dsm)));
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) pw[i] = 0;
  if (threadIdx.x < kPlaneMaxTile) s_row[threadIdx.x] = pair_row(s0 >> 8, threadIdx.x);
  __syncthreads();
  uint32_t z = fmix32_(blockIdx.x * 1024u + threadIdx.x);
  for (uint32_t it = 0; it < iters; ++it) {
    z = z * 1664525u + 1013904223u;
    uint32_t c4[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) c4[w] = fmix32_(z + (uint32_t)w) & 0x33333333u;
    slot_steps(c4, s_row[z >> 27] + ((z >> 26) & 1u) * kPlaneRows, z | 0x80000000u, z * 747796405u, lane);
  }
  __syncthreads();
  uint32_t acc = 0;
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) acc ^= pw[i];
  out[blockIdx.x * 1024u + threadIdx.x] = acc;
}

}  // namespace

// ================================================================================================
// host wrappers
// ================================================================================================
PlaneHash plane_hash(uint64_t seed, uint32_t C, uint32_t B) {
  PlaneHash ph{};
  ph.C = C;
  ph.B = B;
  for (uint32_t c = 0; c < C && c < kPlaneMaxColumns; ++c)
    ph.kcol[c] = xxh3_premix(xxh3_flip(seed + 5ull * c));  // column_seed (include/sketch.h:175-176)
  ph.kchk = xxh3_premix(xxh3_flip(seed));                  // checksum_seed
  return ph;
}

constexpr int kHashSortMaxRpt = 6;
constexpr int kHashSortThreads = 1024;  // one CTA per SM (every register of the SM)

uint32_t hash_sort_tile(uint32_t nbins, size_t smem_budget, uint64_t n) {
  const int nt = kHashSortThreads;
  const size_t fixed = (size_t)2 * ((nbins + 3) & ~3u) * 4 + 256;
  if (nbins > kSortBinsMax || fixed >= smem_budget) return 0;
  // 2 coded entries of 16 B per record, and their 2-byte bins
  const uint64_t most = std::min<size_t>((smem_budget - fixed) / 36, (size_t)kHashSortMaxRpt * nt) / nt * nt;
  if (!most) return 0;
  // an SM's share of the records in as few tiles as hold it, all alike: a short call then uses every
  // SM (8,528 records: 22 us in two tiles of 6144, 9 us in nine of 1024), a long one has no short last wave
  const uint64_t share = (n + num_sms() - 1) / num_sms(), k = std::max<uint64_t>(1, (share + most - 1) / most);
  return (uint32_t)std::min<uint64_t>(most, std::max<uint64_t>(nt, ((share + k - 1) / k + nt - 1) / nt * nt));
}

cudaError_t gutter_hash_sort(const void *d_rec, uint64_t n, GutterGeom g, const PlaneHash &ph,
                             uint32_t rec_tile, const uint64_t *base, uint32_t *fill,
                             uint4 *entries, uint32_t kind, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  constexpr int NT = kHashSortThreads;
  if (rec_tile < (uint32_t)NT || rec_tile > (uint32_t)(kHashSortMaxRpt * NT) || rec_tile % NT ||
      (kind != kEntryCoded && kind != kEntryCoded3))
    return cudaErrorInvalidValue;
  const size_t smem = (size_t)2 * ((g.nbins + 3) & ~3u) * 4 + (size_t)rec_tile * 36;
  const uint64_t tiles = (n + rec_tile - 1) / rec_tile;
  const uint8_t *rec = reinterpret_cast<const uint8_t *>(d_rec);
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e = smem_optin(kern);
    if (e != cudaSuccess) return e;
    const int G = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)num_sms(), tiles));
    kern<<<G, NT, smem, s>>>(rec, n, g, ph, rec_tile, base, fill, entries);
    add_launches(1);
    return cudaGetLastError();
  };
  auto by_rpt = [&](auto c3) -> cudaError_t {
    constexpr bool K = decltype(c3)::value;
    switch (rec_tile / NT) {
      case 1: return launch(k_hash_sort_scatter<1, NT, K>);
      case 2: return launch(k_hash_sort_scatter<2, NT, K>);
      case 3: return launch(k_hash_sort_scatter<3, NT, K>);
      case 4: return launch(k_hash_sort_scatter<4, NT, K>);
      case 5: return launch(k_hash_sort_scatter<5, NT, K>);
      default: return launch(k_hash_sort_scatter<6, NT, K>);
    }
  };
  return kind == kEntryCoded3 ? by_rpt(std::true_type{}) : by_rpt(std::false_type{});
}

size_t plane_update_smem(uint32_t tile_shift, int threads) {
  return kRowBytes + planes_bytes(tile_shift) + deep_words(threads) * 4 + (size_t)(threads / 32) * kQueueSlots * 4;
}

int plane_update_ctas_per_sm(uint32_t tile_shift, int threads) {
  int n = 0;
  auto kern = k_plane_update<true, false, PlaneHash>;
  if (smem_optin(kern) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads,
                                                    plane_update_smem(tile_shift, threads)) != cudaSuccess)
    return 1;
  return n > 0 ? n : 1;
}

cudaError_t plane_update(const PlaneGeom &g, const PlaneHash &ph, uint8_t *sketches,
                         const uint8_t *gutter, const ChunkTable &chunks, const uint32_t *bin_off,
                         int nchunks, uint32_t *work_counter, uint32_t * /*status*/, int grid,
                         int threads, cudaStream_t s) {
  if (g.C > kPlaneMaxColumns || g.C < 18 || g.groups != 1 || g.tile_shift > 5 ||
      g.bin_shift < g.tile_shift || threads % 32 || threads < 32 || threads > 1024)
    return cudaErrorInvalidValue;
  auto kern = k_plane_update<true, false, PlaneHash>;
  cudaError_t e = smem_optin(kern);
  if (e != cudaSuccess) return e;
  kern<<<grid, threads, plane_update_smem(g.tile_shift, threads), s>>>(g, ph, sketches, gutter, chunks, bin_off,
                                                                      nchunks, work_counter);
  add_launches(1);
  return cudaGetLastError();
}

// 32 threads a vertex: one warp each in the write-back. Four CTAs of 8 vertices share an SM, two of 16.
int plane_threads(uint32_t tile_shift) { return std::min(1024, 32 << tile_shift); }

PlaneHashWide plane_hash_wide(uint64_t seed, uint32_t C, uint32_t B) {
  PlaneHashWide ph{};
  ph.C = C;
  ph.B = B;
  for (uint32_t c = 0; c < C && c < kPlaneMaxColumnsWide; ++c) ph.kcol[c] = xxh3_premix(xxh3_flip(seed + 5ull * c));
  ph.kchk = xxh3_premix(xxh3_flip(seed));
  return ph;
}

cudaError_t plane_update_plain(const PlaneGeom &g, bool cube, const PlaneHashWide &ph, uint8_t *sketches,
                               const uint8_t *gutter, const ChunkTable &chunks, const uint32_t *bin_off,
                               int nchunks, uint32_t *work_counter, cudaStream_t s) {
  if (g.C > kPlaneMaxColumnsWide || g.groups != (g.C + kPlaneSlots) / kPlaneSlots || g.tile_shift > 5 ||
      g.bin_shift < g.tile_shift || (g.groups > 1 && g.direct_max))
    return cudaErrorInvalidValue;
  const int threads = plane_threads(g.tile_shift);
  const size_t smem = plane_update_smem(g.tile_shift, threads);
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e = smem_optin(kern);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
    if (e != cudaSuccess) return e;
    const int grid = (int)std::min<uint64_t>((uint64_t)g.ntiles * g.groups, (uint64_t)num_sms() * std::max(per_sm, 1));
    kern<<<grid, threads, smem, s>>>(g, ph, sketches, gutter, chunks, bin_off, nchunks, work_counter);
    add_launches(1);
    return cudaGetLastError();
  };
  return cube ? launch(k_plane_update<false, true, PlaneHashWide>)
              : launch(k_plane_update<false, false, PlaneHashWide>);
}

cudaError_t direct_records(const void *d_rec, uint64_t n, uint32_t V, uint32_t sketch_words,
                           const PlaneHash &ph, uint8_t *sketches, uint32_t *status, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (ph.C > kPlaneMaxColumns) return cudaErrorInvalidValue;
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 7) / 8, (uint64_t)num_sms() * 8);
  k_direct_records<<<grid, 256, 0, s>>>(reinterpret_cast<const uint8_t *>(d_rec), n, V, sketch_words, ph,
                                        reinterpret_cast<uint32_t *>(sketches), status);
  add_launches(1);
  return cudaGetLastError();
}

cudaError_t plane_hash_peak(uint32_t iters, int blocks, int threads, uint64_t *out, cudaStream_t s) {
  k_plane_hash_peak<<<blocks, threads, 0, s>>>(iters, out);
  add_launches(1);
  return cudaGetLastError();
}

cudaError_t plane_update_peak(uint32_t iters, int blocks, uint32_t *out, cudaStream_t s) {
  cudaError_t e = smem_optin(k_plane_update_peak);
  if (e != cudaSuccess) return e;
  k_plane_update_peak<<<blocks, 1024, kRowBytes + planes_bytes(5), s>>>(iters, out);
  add_launches(1);
  return cudaGetLastError();
}

}  // namespace gz
