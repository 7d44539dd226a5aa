// gz_noalloc.cu -- gz_ingest_records_noalloc: the record-ingest pipeline (device gutter +
// sketch update) for callers that cannot allocate GPU memory.
//
// Some callers of this library are not allowed to allocate device memory: plugins running inside
// a host framework that hands out all GPU memory from its own pool (a library-side cudaMalloc
// would bypass that pool's accounting and can fail or fragment it), and latency-critical service
// loops where cudaMalloc / cudaFree would synchronize the device and stall every other stream.
// For them this entry point takes the caller's sketches and records (both already in device
// memory) and allocates nothing: its scratch memory (gutter entries, bin counts and offsets,
// status words) lives in one fixed, file-scope device array that every GPU which
// loads the library holds until the process exits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/gz_b200.h"
#include "gz_device.cuh"
#include "gz_kernels.cuh"

// gz_capi.cu: stores the text gz_last_error() returns on this thread
void gz_internal_set_error(const std::string &msg);

namespace {

// Limits of one call, and the scratch layout they need.
constexpr uint64_t kNoAllocMaxRecords = 1ull << 21;  // 2,097,152 records per call
constexpr uint32_t kNoAllocMaxVertices = 1u << 22;   // 4,194,304 vertices
constexpr uint32_t kNoAllocMaxBins = 1u << 16;
constexpr uint32_t kNoAllocMaxColumns = 127;

constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kOffEntries = 0;
constexpr size_t kOffCounts = align256(kOffEntries + kNoAllocMaxRecords * 2 * 8);
constexpr size_t kOffCursor = align256(kOffCounts + (size_t)kNoAllocMaxBins * 8);
constexpr size_t kOffScanTmp = align256(kOffCursor + (size_t)kNoAllocMaxBins * 8);
constexpr size_t kOffTotal = align256(kOffScanTmp + 64 * 8);
constexpr size_t kOffBinOff = align256(kOffTotal + 8);
constexpr size_t kOffFill = align256(kOffBinOff + ((size_t)kNoAllocMaxBins + 1) * 4);
constexpr size_t kOffStatus = align256(kOffFill + (size_t)kNoAllocMaxBins * 4);
constexpr size_t kScratchBytes = align256(kOffStatus + 16);  // about 34 MiB

// The scratch array. Host code must not use this name as a device address: the address comes
// from cudaGetSymbolAddress, once per device (see scratch_for_current_device).
static __device__ __align__(256) uint8_t g_noalloc_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mtx;
uint8_t *g_noalloc_ptr[kMaxDevices] = {};

int noalloc_fail(int code, const std::string &msg) {
  gz_internal_set_error(msg);  // read back through gz_last_error()
  return code;
}

// Device address of the scratch array on the current device; looked up on the first call made
// on each device (that first call should therefore come before any stream capture).
int scratch_for_current_device(uint8_t **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(GZ_ERR_NO_DEVICE, cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(GZ_ERR_INVALID, "device index too large");
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
      return noalloc_fail(GZ_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    g_noalloc_ptr[dev] = static_cast<uint8_t *>(p);
  }
  *out = g_noalloc_ptr[dev];
  return GZ_OK;
}

// The reference sizing (include/sketch.h:62-76, :181, :188-190), same double expressions.
void noalloc_params(uint32_t V, double f, uint32_t &C, uint32_t &B) {
  const uint64_t vec_len = (uint64_t)std::ceil(double(V) * (uint32_t)(V - 1) / 2);
  B = (uint32_t)(std::ceil(std::log2((double)vec_len)) + 1);
  const double num_samples_div = 1 - std::log2(2 - 0.8);
  const size_t s = (size_t)std::ceil(f * std::log2((double)V) / num_samples_div);
  C = (uint32_t)std::max<size_t>(18, s);
}

#define NA_CUDA(call)                                                                     \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return noalloc_fail(GZ_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// Once a call has queued work on its stream, every return waits for that work: the scratch array
// must be idle before the lock is released, or the next call (on any stream) would overwrite the
// regions the queued kernels still use. Declared after the lock guard, so it runs first.
struct StreamDrain {
  cudaStream_t s;
  bool armed = false;
  ~StreamDrain() {
    if (armed) cudaStreamSynchronize(s);
  }
};

}  // namespace

extern "C" {

int gz_ingest_records_noalloc(void *d_sketches, uint32_t num_vertices, uint64_t seed,
                              double sketches_factor, const void *d_records, size_t n_records,
                              void *stream_ptr) {
  if (!d_sketches || (n_records && !d_records)) return noalloc_fail(GZ_ERR_INVALID, "null argument");
  if (num_vertices < 2 || num_vertices > kNoAllocMaxVertices)
    return noalloc_fail(GZ_ERR_INVALID, "num_vertices must be in [2, " +
                                            std::to_string(kNoAllocMaxVertices) + "] for this entry point");
  if (n_records > kNoAllocMaxRecords)
    return noalloc_fail(GZ_ERR_INVALID, "at most " + std::to_string(kNoAllocMaxRecords) +
                                            " records per call (the fixed scratch holds no more); "
                                            "split the stream");
  const double f = sketches_factor > 0 ? sketches_factor : 1;
  uint32_t C = 0, B = 0;
  noalloc_params(num_vertices, f, C, B);
  if (C > kNoAllocMaxColumns || B > 63)
    return noalloc_fail(GZ_ERR_INVALID, "sketch has too many columns for this entry point");
  if (n_records == 0) return GZ_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream_ptr);

  std::lock_guard<std::mutex> lk(g_noalloc_mtx);
  StreamDrain drain{s};
  uint8_t *scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc != GZ_OK) return rc;

  // tiles of 8 vertices with a gutter bin each; of 16 or 32 where that many more vertices still keep
  // the bins within the shared-memory sort, or within the scratch's bins, with several tiles of 32 a
  // bin past that
  const uint32_t nb = C * B + 1;
  int dev = 0, smem_optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem_optin <= 0) smem_optin = 227 * 1024;
  auto tiles_of = [&](uint32_t sh) { return (uint32_t)(((uint64_t)num_vertices + (1u << sh) - 1) >> sh); };
  uint32_t shift = 3;
  while (shift < 5 && (tiles_of(shift) > kNoAllocMaxBins ||
                       (tiles_of(shift) > gz::kSortBinsMax && tiles_of(5) <= gz::kSortBinsMax)))
    ++shift;
  uint32_t bshift = shift;
  while (tiles_of(bshift) > kNoAllocMaxBins) ++bshift;
  const uint32_t nbins = tiles_of(bshift);

  // scratch regions
  uint2 *entries = reinterpret_cast<uint2 *>(scratch + kOffEntries);
  uint64_t *counts = reinterpret_cast<uint64_t *>(scratch + kOffCounts);
  uint64_t *cursor = reinterpret_cast<uint64_t *>(scratch + kOffCursor);
  uint64_t *scan_tmp = reinterpret_cast<uint64_t *>(scratch + kOffScanTmp);
  uint64_t *total = reinterpret_cast<uint64_t *>(scratch + kOffTotal);
  uint32_t *bin_off = reinterpret_cast<uint32_t *>(scratch + kOffBinOff);
  uint32_t *fill = reinterpret_cast<uint32_t *>(scratch + kOffFill);
  uint32_t *status = reinterpret_cast<uint32_t *>(scratch + kOffStatus);  // [0] bits, [1] work

  // the array keeps the previous call's contents: reset what must start at zero
  drain.armed = true;
  NA_CUDA(cudaMemsetAsync(counts, 0, sizeof(uint64_t) * nbins, s));
  NA_CUDA(cudaMemsetAsync(fill, 0, sizeof(uint32_t) * nbins, s));
  NA_CUDA(cudaMemsetAsync(status, 0, 16, s));

  const gz::GutterGeom gg{num_vertices, bshift, nbins};
  const int G = (int)std::max<uint64_t>(
      1, std::min<uint64_t>(2ull * gz::num_sms(), (n_records + gz::kRecTile - 1) / gz::kRecTile));
  NA_CUDA(gz::gutter_count(gz::kInputRecords, d_records, n_records, gg, G, counts, status, s));
  NA_CUDA(gz::scan_exclusive_u64(counts, nbins, total, scan_tmp, s));
  NA_CUDA(gz::gutter_bin_offsets(counts, 1, nbins, total, bin_off, s));
  const uint32_t tile = gz::sort_scatter_tile(gz::kInputRecords, gg, (size_t)smem_optin - 1024);
  if (tile >= 1024) {
    NA_CUDA(gz::gutter_sort_scatter(gz::kInputRecords, d_records, n_records, gg, tile, counts, fill,
                                    entries, s));
  } else {
    NA_CUDA(gz::copy_u64(counts, cursor, nbins, s));
    NA_CUDA(gz::gutter_scatter_global(gz::kInputRecords, d_records, n_records, gg, G, cursor,
                                      entries, s));
  }
  gz::PlaneGeom g{};
  g.V = num_vertices;
  g.C = C;
  g.B = B;
  g.sketch_words = nb * 3;
  g.groups = (C + gz::kPlaneSlots) / gz::kPlaneSlots;
  g.tile_shift = shift;
  g.ntiles = tiles_of(shift);
  g.bin_shift = bshift;
  g.nbins = nbins;
  gz::ChunkTable chunks{};
  chunks.base[0] = 0;
  chunks.kind[0] = gz::kEntryPlain;
  NA_CUDA(gz::plane_update_plain(g, false, gz::plane_hash_wide(seed, C, B), static_cast<uint8_t *>(d_sketches),
                                 reinterpret_cast<const uint8_t *>(entries), chunks, bin_off, 1, status + 1, s));
  uint32_t st = 0;
  NA_CUDA(cudaMemcpyAsync(&st, status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  NA_CUDA(cudaStreamSynchronize(s));
  if (st & gz::kStatusTimeout) return noalloc_fail(GZ_ERR_TIMEOUT, "a bounded device wait timed out");
  if (st & gz::kStatusBadVertex)
    return noalloc_fail(GZ_ERR_BAD_VERTEX, "a record named a vertex id >= V; it was dropped");
  return GZ_OK;
}

}  // extern "C"
