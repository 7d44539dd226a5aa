// gz_planes.cu -- record ingest through bucket planes: coded entries (CameoSketch of at most 31 columns),
// plain entries (CubeSketch, more columns, large graphs), and records XORed straight into the sketches.
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
//                        in HBM. The checksum is hashed here, per entry (of a plain entry, the
//                        columns too).
//   k_direct_records     few records: each by a warp into both endpoints' sketches in HBM.
// A coded entry is 128 bits: the C codes in bits 0 .. 4C - 1 (column c in bits 4c .. 4c + 3),
// then the neighbour shifted left by bin_shift bits OR the vertex's offset inside its gutter bin
// (the bin is known from where the entry lies). It is used when 4C + bin_shift + the neighbour's
// bits fit in 128 (every CameoSketch up to 2^18 vertices). Past that, codes of 3 bits (code 7 =
// depth 7 or more) fit larger graphs (3C + bin_shift + neighbour bits <= 128: 2^20 vertices and
// far beyond); an escaped column (1 in 128 column updates) is hashed again where the entry is
// applied, so the planes see the same 4-bit codes either way.
//
// The planes themselves: gz_planes.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "gz_common.cuh"
#include "gz_device.cuh"
#include "gz_kernels.cuh"
#include "gz_planes.cuh"

namespace gz {

namespace {

using namespace gz::dev;

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

// Sparse calls (few updates for the graph's size): every record hashed once, a warp per record and
// a lane per column, and XORed into both endpoints' sketches in HBM: one launch, no gutter.
// (A self-loop XORs one sketch twice: no change, as through the gutter.)
__global__ void __launch_bounds__(256)
k_direct_records(const uint8_t *__restrict__ rec, uint64_t n, uint32_t V, uint32_t sketch_words,
                 PlaneHash ph, uint32_t *__restrict__ sk, uint32_t *__restrict__ status) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t kc = lane < ph.C ? ph.kcol[lane] : ph.kchk;
  // up to 32 consecutive records a warp, read by its lanes
  const uint32_t per = (uint32_t)min((n + nwarps - 1) / nwarps, (uint64_t)32);
  for (uint64_t i0 = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * per; i0 < n; i0 += nwarps * per) {
    uint32_t mu = 0, mv = 0;
    if (lane < per && i0 + lane < n) load_record(rec, rec + 9 * n, i0 + lane, mu, mv);
    if (mu >= V || mv >= V) {
      atomicOr(status, kStatusBadVertex);
      mu = mv;  // dropped
    }
    for (uint32_t m = __ballot_sync(kFull, mu != mv); m; m &= m - 1) {
      const uint32_t u = __shfl_sync(kFull, mu, __ffs(m) - 1), v = __shfl_sync(kFull, mv, __ffs(m) - 1);
      warp_record_global(sk + (uint64_t)u * sketch_words, sk + (uint64_t)v * sketch_words, u, v, ph.C, ph.B, kc,
                         ph.kchk);
    }
  }
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
  __shared__ uint4 s_claim[3];  // item, entries of its bin, and their range when there is one chunk
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
  auto claim = [&](uint4 &to) {
    uint4 c = make_uint4(atomicAdd(work_counter, 1u), 0, 0, 0);
    if (c.x < nitems) {
      const uint32_t bin = (c.x / g.groups) >> per_bin;
      for (int k = 0; k < nchunks; ++k) {
        c.z = bin_off[(uint64_t)k * stride + bin];
        c.w = bin_off[(uint64_t)k * stride + bin + 1];
        c.y += c.w - c.z;
      }
    }
    to = c;
  };
  const uint32_t esz = CODED ? 16 : 8;
  const uint32_t dense = 64u << g.tile_shift;  // entries of a tile whose rows are all in use
  if (threadIdx.x == 0) {
    claim(s_claim[0]);
    claim(s_claim[1]);
  }
  for (uint32_t n = 0;; ++n) {
    __syncthreads();
    const uint4 cl = s_claim[n % 3], ahead = s_claim[(n + 1) % 3];
    const uint32_t item = cl.x, total = cl.y;
    if (item >= nitems) break;
    if (threadIdx.x == 0) claim(s_claim[(n + 2) % 3]);  // while the others work on this one
    // a small tile is a chain of waits: what the next one will read is brought to L2 meanwhile
    if (ahead.x < nitems && ahead.y && ahead.y < dense && nchunks == 1) {
      for (uint32_t o = 128 * threadIdx.x; o < esz * (ahead.w - ahead.z); o += 128 * blockDim.x)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(gutter + chunks.base[0] + (uint64_t)esz * ahead.z + o));
      const uint32_t t2 = ahead.x / g.groups, c2 = (ahead.x - t2 * g.groups) * kPlaneSlots + lane;
      for (uint32_t vl = warp; vl < W; vl += nwarps)
        if (c2 < C && (t2 << g.tile_shift) + vl < g.V) {
          const uint32_t *p = x.gsk + (uint64_t)((t2 << g.tile_shift) + vl) * g.sketch_words + 3 * c2 * B;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p + column_second_word(B)));
        }
    }
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
      uint32_t b = cl.z, e = cl.w;
      if (nchunks > 1) {
        b = bin_off[(uint64_t)k * stride + x.bin];
        e = bin_off[(uint64_t)k * stride + x.bin + 1];
      }
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
    // (a large one's rows would not stay there that long: brought while the other warps finish)
    if (total >= dense)
      for (uint32_t vl = warp; vl < W; vl += nwarps) {
        const uint32_t vg = (x.t << g.tile_shift) + vl;
        if (vg < g.V && lane < x.nc) {
          const uint32_t *p = x.gsk + (uint64_t)vg * g.sketch_words + 3 * (x.c0 + lane) * B;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 3 * min(B, kPlaneThr) - 1));
        }
      }
    __syncthreads();
    for (uint32_t vl = warp; vl < W; vl += nwarps) {
      const uint32_t vg = (x.t << g.tile_shift) + vl;
      if (vg >= g.V) break;
      write_back<CUBE>(s_row[vl] << 8, vg, x.gsk + (uint64_t)vg * g.sketch_words + 3 * (size_t)x.c0 * B, x.nc,
                       C - x.c0, B, lane, total < dense);
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
                         int nchunks, uint32_t *work_counter, int grid, int threads, cudaStream_t s) {
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
