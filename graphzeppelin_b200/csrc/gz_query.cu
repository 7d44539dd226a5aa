// gz_query.cu -- the whole connectivity query in one kernel launch.
//
// boruvka_emulation (src/cc_sketch_alg.cpp:464-513) with every round on the device: a fresh DSU,
// round 0, then per round two phases, each closed by a barrier of the whole launch --
//   A  accumulate: the root of every vertex; each vertex's sample of this round (and its
//      deterministic bucket) XORed into its root's accumulator (perform_boruvka_round,
//      src/cc_sketch_alg.cpp:246-380);
//   B  sample: every root's accumulator sampled (Sketch::sample, src/sketch.cpp:94-116), cleared
//      for the next round, and the sampled edges united (sample_supernode, :137-166).
//
// What bounds it, and why this form. A query reads 12 (B cps + 1) bytes per vertex and round, far
// less than the machine moves in the time a round takes: what counts is the number of dependent
// steps. Grouping the vertices by component first (count, scan, scatter, merge, fold, sample: six
// barriers a round) makes every merge a register XOR, but costs 28 of the 60 us of a round at
// 2^17 vertices. Here the members stay in vertex order and meet in L2: a warp XORs the words of
// its vertices into the roots' accumulators with 32-bit reductions on consecutive words (one
// 128-byte request per 32 words), so a round is two barriers. Three rules keep the traffic down:
//   - a warp orders its 32 vertices by root and reduces equal neighbours in registers;
//   - a component that samples ZERO and takes part in no union afterwards keeps its deterministic
//     bucket, so it samples ZERO in every later round: its vertices are skipped;
//   - a component holding most vertices (judged from 32 probe vertices) is accumulated from its
//     complement when every update reached both endpoints (the XOR of all sketches is zero): its
//     vertices are skipped, all others also go to its accumulator, and nothing else is skipped.
// Samples are checked flattened: the cps B + 1 buckets of a batch's members are dealt over the
// 32 lanes, so a batch of 8 members of 35 buckets takes 9 checks a lane instead of 24.
//
// Up to kClusterMaxV vertices the launch is one thread-block cluster, whose hardware barrier
// costs a fraction of a grid barrier through L2; above, a cooperative launch of one block per SM.
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

// Sketch::sample (src/sketch.cpp:94-116) of the n <= KB members of a landed batch: slot k holds
// member k's columns at byte offset (offs & 255) and its deterministic bucket at run_cap +
// (offs >> 8), offs being lane k's. The CPS B + 1 buckets of a member -- deterministic first, then the
// columns in order -- are checked SW at a time, 32 / SW members side by side and the batch's checks
// independent of each other; most members find their first good bucket among the first SW, so the
// next SW are looked at only while a member is undecided. Returns, on lane lane0 + k, member k's
// 0 GOOD / 1 ZERO / 2 FAIL and the sampled index.
template <int CPS, int KB>
__device__ __forceinline__ int sample_batch(const uint8_t *slots, uint32_t slot_bytes, uint32_t run_cap,
                                            uint32_t offs, uint32_t n, uint32_t lane0, uint32_t B,
                                            uint64_t flip_chk, uint64_t *idx) {
  constexpr uint32_t SW = KB == 1 ? 32 : 16, MPP = 32 / SW;  // members per pass
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nbk = CPS * B + 1;
  const uint32_t k = (lane - lane0) & (KB - 1);
  const uint32_t ok = __shfl_sync(kFull, offs, k);
  const bool mine = lane >= lane0 && lane - lane0 < n;
  const uint8_t *sl = slots + k * slot_bytes;
  const uint32_t *det = reinterpret_cast<const uint32_t *>(sl + run_cap + (ok >> 8));
  const bool zero = mine && (det[0] | det[1] | det[2]) == 0;
  int first = -1;
  auto check = [&](uint32_t q, auto passes) {
#pragma unroll
    for (uint32_t p = 0; p < decltype(passes)::value; ++p) {
      const uint32_t m = min(p * MPP + lane / SW, n - 1), pos = min(q + lane % SW, nbk - 1);
      const uint32_t o = __shfl_sync(kFull, offs, m);
      const uint32_t *w = reinterpret_cast<const uint32_t *>(
          slots + m * slot_bytes + (pos ? (o & 255u) + 12 * (pos - 1) : run_cap + (o >> 8)));
      const uint32_t bal = __ballot_sync(kFull, q + lane % SW < nbk && bucket_good(w[0], w[1], w[2], flip_chk));
      const uint32_t bits = SW == 32 ? bal : (bal >> (SW * (k % MPP))) & ((1u << (SW & 31)) - 1u);
      if (k / MPP == p && first < 0 && bits) first = (int)(q + __ffs(bits) - 1);
    }
  };
  constexpr int kPasses = KB / MPP > 0 ? KB / MPP : 1;
  for (uint32_t q = 0; q < nbk; q += SW) {
    if (!__any_sync(kFull, mine && !zero && first < 0)) break;
    if (kPasses > 1 && n <= MPP) check(q, std::integral_constant<int, 1>{});
    else check(q, std::integral_constant<int, kPasses>{});
  }
  *idx = 0;
  if (!mine || zero) return 1;
  if (first < 0) return 2;
  const uint32_t *w = first ? reinterpret_cast<const uint32_t *>(sl + (ok & 255u)) + 3 * (first - 1) : det;
  *idx = ((uint64_t)w[1] << 32) | w[0];
  return 0;
}

// Applies a sample result (sample_supernode, src/cc_sketch_alg.cpp:137-166): a GOOD one unites the
// sampled edge. A root is linked under another at most once in a query, so the spanning forest
// keeps each edge at the absorbed root's place. True when the round is modified (FAIL or a merge).
__device__ __forceinline__ bool apply_result(int res, uint64_t idx, uint32_t round, uint32_t key,
                                             const BoruvkaGeom &g, const BoruvkaBufs &b) {
  if (b.trace) {
    const uint32_t ti = atomicAdd(b.trace_n, 1u);
    if (ti < b.trace_cap) reinterpret_cast<TraceRec *>(b.trace)[ti] = TraceRec{round, key, (uint32_t)res, 0, idx};
  }
  if (res == 2) return true;
  if (res == 1) return false;
  uint32_t x = (uint32_t)(idx >> 32), y = (uint32_t)idx;
  if (x >= g.V || y >= g.V) {
    atomicOr(b.status, kStatusBadSample);
    return false;
  }
  if (!unite_two(b.parent, x, y, 0)) return false;
  b.rstate[2 * x + 1] = round + 1;
  b.forest[y] = idx;
  return true;
}

// Most threads of a block: 80 registers a thread for CameoSketch; CubeSketch keeps two samples of 7
// columns in registers.
template <int CPS>
constexpr int kBvqMaxThreads = CPS == 1 ? 768 : 384;
constexpr uint32_t kMinRingWords = 29;  // a warp's stage (3 words more) holds its 32 vertices

// State of a root (b.rstate): x = 1 + the last round it sampled ZERO in, y = 1 + the last round
// another root was linked under it in (0: never). The component is finished, with nothing but ZERO
// to come, while x > y.
template <int CPS, int NW, int KB, bool CL>
__global__ void __launch_bounds__(kBvqMaxThreads<CPS>, 1)
k_bv_query(BoruvkaGeom g, const uint32_t *__restrict__ sk_words, BoruvkaBufs b, uint32_t samples,
           uint32_t *labels_out, uint32_t *ncc) {
  extern __shared__ __align__(16) uint8_t bv_smem[];
  __shared__ uint32_t s_big;
  constexpr uint32_t BPG = 32 / KB;  // batches per 32 vertices
  const uint32_t V = g.V, tid = threadIdx.x, lane = tid & 31;
  const uint32_t W = 3 * CPS * g.B, SW = racc_words(CPS, g.B), detw = 3 * g.C * g.B;
  const uint32_t ring_words = max(W, kMinRingWords);
  BvRing ring;
  ring.init(bv_smem + (tid >> 5) * bv_warp_bytes(ring_words, KB), ring_words, KB);
  uint32_t *perm = ring.stage;  // 32 words: the warp's vertices in processing order
  uint32_t T = 0;               // batches through this warp's copy ring
  uint32_t nbar = 0;            // barriers passed
  bool failed = false;
  auto sync = [&]() { return launch_barrier<CL>(b.qbar, ++nbar, failed, b.status); };
  const uint32_t gw = (blockIdx.x * blockDim.x + tid) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t gt = blockIdx.x * blockDim.x + tid, nthreads = gridDim.x * blockDim.x;
  const uint32_t nbatch = (V + KB - 1) / KB;  // batches of KB consecutive vertices, dealt to the warps
  const bool trace = b.trace != nullptr;
  // When a warp's vertices fit one group, each lane keeps its vertex's root in a register between
  // the phases (kept; open: accumulated in this round); otherwise it goes through b.label.
  const bool once = nbatch <= BPG * nwarps;
  // lane's vertex of the group of BPG batches starting at batch it, or ~0
  auto my_vertex = [&](uint32_t it) {
    const uint32_t bt = it + (lane / KB) * nwarps, v = bt * KB + lane % KB;
    return bt < nbatch && v < V ? v : 0xffffffffu;
  };
  auto label_of = [&](uint32_t it) {
    const uint32_t v = my_vertex(it);
    return v != 0xffffffffu ? __ldcg(b.label + v) : 0u;
  };
  // a landed batch's slots, or the timeout status and failed = true
  auto landed = [&](uint32_t t, bool more) {
    if (ring.wait(T + t)) return true;
    if (lane == 0) atomicOr(b.status, kStatusTimeout);
    if (more) ring.wait(T + t + 1);  // its copies must land before the shared memory is freed
    failed = true;
    return false;
  };

  const bool dirty = __ldcg(b.racc_dirty) != 0;  // first use, or the last query did not finish
  for (uint32_t v = gt; v < V; v += nthreads) {
    b.parent[v] = v;
    b.label[v] = v;
    reinterpret_cast<uint2 *>(b.rstate)[v] = make_uint2(0, 0);
    b.forest[v] = kNoEdge;
    if (trace) b.minv[v] = 0xffffffffu;
  }
  if (dirty)
    for (uint64_t i = gt; i < (uint64_t)V * (SW / 4); i += nthreads)
      reinterpret_cast<uint4 *>(b.racc)[i] = make_uint4(0, 0, 0, 0);
  if (gt == 0) {
    *b.forest_n = V;
    if (trace) *b.trace_n = 0;
    b.flags[0] = b.flags[1] = b.flags[2] = 0;
    *ncc = 0;
  }
  if (!sync()) return;
  if (gt == 0) *b.racc_dirty = 1;

  // ---- round 0 (run_round_zero, src/cc_sketch_alg.cpp:223-244): every vertex samples its sample 0
  for (uint32_t it = gw; it < nbatch && !failed; it += BPG * nwarps) {
    auto issue = [&](uint32_t t) {
      const uint32_t v = (it + t * nwarps) * KB + lane;
      const bool mine = it + t * nwarps < nbatch && lane < (uint32_t)KB && v < V;
      const uint32_t *sk = sk_words + (uint64_t)(mine ? v : 0) * g.sketch_words;
      ring.issue(T + t, mine, sk, W, sk + detw, KB);
      return slot_offsets(sk, sk + detw);
    };
    const uint32_t nb = min(BPG, (nbatch - it + nwarps - 1) / nwarps);
    int my_res = 1;
    uint64_t my_idx = 0;
    uint32_t offs = issue(0);
    for (uint32_t t = 0; t < nb; ++t) {
      const uint32_t offs_next = t + 1 < nb ? issue(t + 1) : 0u;
      if (!landed(t, t + 1 < nb)) break;
      const uint32_t v0 = (it + t * nwarps) * KB;
      uint64_t idx;
      const int res = sample_batch<CPS, KB>(ring.slot(T + t, 0, KB), ring.slot_bytes, ring.run_cap, offs,
                                            min((uint32_t)KB, V - v0), t * KB, g.B, g.flip_chk, &idx);
      if (lane / KB == t) {
        my_res = res;
        my_idx = idx;
      }
      // the deterministic bucket is read in every round: kept in 16 bytes a vertex, side by side
      if (lane < (uint32_t)KB && v0 + lane < V) {
        const uint32_t *d = reinterpret_cast<const uint32_t *>(ring.slot(T + t, lane, KB) + ring.run_cap + (offs >> 8));
        reinterpret_cast<uint4 *>(b.det)[v0 + lane] = make_uint4(d[0], d[1], d[2], 0);
      }
      offs = offs_next;
      __syncwarp();
    }
    if (failed) break;
    T += nb;
    const uint32_t v = my_vertex(it);
    bool mod = false;
    if (v != 0xffffffffu) {
      if (my_res == 1) b.rstate[2 * v] = 1;
      mod = apply_result(my_res, my_idx, 0, v, g, b);
    }
    if (mod) atomicOr(b.flags, 1u);
    __syncwarp();
  }
  if (!sync()) return;

  uint32_t round = 0, kept = my_vertex(gw);
  bool open = false;
  for (;;) {
    const uint32_t modified = __ldcg(b.flags + round % 3);
    if (modified == 0 || round + 1 >= samples) {
      if (gt == 0) {
        b.ctl[0] = modified ? round + 1 : round;
        b.ctl[1] = modified ? 1u : 0u;
        b.ctl[2] = 0;
        *b.round = round;
        // every accumulator was cleared by the root that read it, unless a block gave up on the way
        if (!(__ldcg(b.status) & kStatusTimeout)) *b.racc_dirty = 0;
      }
      break;
    }
    ++round;
    uint32_t *flags = b.flags + round % 3;
    if (gt == 0) b.flags[(round + 1) % 3] = 0;  // last read before the previous round's barriers
    const uint32_t col = 3 * round * CPS * g.B;

    // ---- A
    if (round == 1) fence_proxy_async_all();  // b.det, written in round 0
    // the component merged from its complement, if one holds most of 32 probe vertices (every
    // block finds the same: no union runs in this phase); not worth its latency while a warp has
    // one batch at most
    uint32_t big = 0xffffffffu;
    if (g.complement && nbatch > nwarps) {
      if (tid < 32) {
        const uint32_t p = dsu_find(b.parent, (uint32_t)(((uint64_t)lane * V) >> 5));
        const uint32_t votes = __popc(__match_any_sync(kFull, p));
        const uint32_t m = __ballot_sync(kFull, votes >= 17);
        const uint32_t most = __shfl_sync(kFull, p, m ? __ffs(m) - 1 : 0);
        if (lane == 0) s_big = m ? most : 0xffffffffu;
      }
      __syncthreads();
      big = s_big;
    }
    const bool skip_done = big == 0xffffffffu && !trace;
    uint32_t cpl[NW], dcpl = 0;
#pragma unroll
    for (int k = 0; k < NW; ++k) cpl[k] = 0;
    auto reduce_into = [&](uint32_t root, const uint32_t (&x)[NW], uint32_t dx) {
      uint32_t *ac = b.racc + (uint64_t)root * SW;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t wi = k * 32 + lane;
        if (wi < W && x[k]) atomicXor(ac + wi, x[k]);
      }
      if (lane < 3 && dx) atomicXor(ac + W + lane, dx);
    };
    // labels are read one group ahead
    uint32_t ahead = once ? 0u : label_of(gw);
    for (uint32_t it = gw; it < nbatch && !failed; it += BPG * nwarps) {
      const uint32_t v = my_vertex(it);
      const bool in = v != 0xffffffffu;
      const uint32_t lab = ahead;
      if (!once) ahead = label_of(it + BPG * nwarps);
      // the vertex's root of the previous round, then its root now. Both are the same unless the
      // root was linked under another in the previous round, and then the root now was linked to
      // in it: only an unchanged root can be finished, so its state is read alongside its parent
      uint32_t r = 0;
      bool need = false;
      if (in) {
        const uint32_t r0 = once ? kept : lab;
        // (not for the complement's own vertices: they would all read one root's words)
        const uint32_t p = r0 == big ? r0 : __ldcg(b.parent + r0);
        const uint2 st = r0 == big ? make_uint2(0, 0) : __ldcg(reinterpret_cast<const uint2 *>(b.rstate) + r0);
        r = p;
        if (p != r0) {
          r = dsu_find(b.parent, p);
          if (!once) b.label[v] = r;
        }
        if (trace) atomicMin(b.minv + r, v);
        need = r != big && !(skip_done && p == r0 && st.x > st.y);
        kept = r;
      }
      open = need;
      const uint32_t needm = __ballot_sync(kFull, need);
      const uint32_t n = __popc(needm);
      if (!n) continue;
      // order the needed vertices by root (equal roots adjacent)
      uint32_t leader = 32;
      if (need) leader = __ffs(__match_any_sync(needm, r)) - 1;
      uint32_t rank = 0;
      for (uint32_t mm = needm; mm; mm &= mm - 1) {
        const uint32_t l = __ffs(mm) - 1, ll = __shfl_sync(kFull, leader, l);
        rank += ll < leader || (ll == leader && l < lane);
      }
      if (need) perm[rank] = lane;
      __syncwarp();
      const uint32_t src = lane < n ? perm[lane] : 0u;
      __syncwarp();
      const uint32_t vq = __shfl_sync(kFull, v, src), rq = __shfl_sync(kFull, r, src);
      auto issue = [&](uint32_t t) {  // lane k < KB copies member t KB + k
        const uint32_t m = t * KB + lane;
        const uint32_t vm = __shfl_sync(kFull, vq, m & 31);
        const bool mine = lane < (uint32_t)KB && m < n;
        const uint32_t *sk = sk_words + (uint64_t)(mine ? vm : 0) * g.sketch_words;
        ring.issue(T + t, mine, sk + col, W, b.det + 4 * (size_t)(mine ? vm : 0), KB);
      };
      const uint32_t nb = (n + KB - 1) / KB;
      issue(0);
      uint32_t acc[NW], dacc = 0, cur = 0xffffffffu;
#pragma unroll
      for (int k = 0; k < NW; ++k) acc[k] = 0;
      for (uint32_t t = 0; t < nb; ++t) {
        if (t + 1 < nb) issue(t + 1);
        if (!landed(t, t + 1 < nb)) break;
#pragma unroll 1
        for (uint32_t k = 0; k < (uint32_t)KB && t * KB + k < n; ++k) {
          const uint32_t m = t * KB + k;
          const uint32_t c = __shfl_sync(kFull, rq, m), vm = __shfl_sync(kFull, vq, m);
          const uint32_t *sk = sk_words + (uint64_t)vm * g.sketch_words;
          if (c != cur) {
            if (cur != 0xffffffffu) reduce_into(cur, acc, dacc);
            cur = c;
#pragma unroll
            for (int q = 0; q < NW; ++q) acc[q] = 0;
            dacc = 0;
          }
          const uint8_t *slt = ring.slot(T + t, k, KB);
          const uint32_t *sl = bulk_run_at(slt, sk + col);
          const uint32_t *sd = reinterpret_cast<const uint32_t *>(slt + ring.run_cap);
#pragma unroll
          for (int q = 0; q < NW; ++q) {
            const uint32_t wi = q * 32 + lane;
            if (wi < W) acc[q] ^= sl[wi];
          }
          if (lane < 3) dacc ^= sd[lane];
          if (big != 0xffffffffu) {
#pragma unroll
            for (int q = 0; q < NW; ++q) {
              const uint32_t wi = q * 32 + lane;
              if (wi < W) cpl[q] ^= sl[wi];
            }
            if (lane < 3) dcpl ^= sd[lane];
          }
        }
        __syncwarp();
      }
      if (failed) break;
      T += nb;
      reduce_into(cur, acc, dacc);
    }
    if (big != 0xffffffffu && !failed) reduce_into(big, cpl, dcpl);
    if (!sync()) return;

    // ---- B
    fence_proxy_async_all();
    ahead = once ? 0u : label_of(gw);
    for (uint32_t it = gw; it < nbatch && !failed; it += BPG * nwarps) {
      const uint32_t v = my_vertex(it);
      bool root = v != 0xffffffffu && (once ? kept : ahead) == v;
      if (!once) ahead = label_of(it + BPG * nwarps);
      if (once) {
        root = root && (open || v == big);
      } else if (root && skip_done) {
        // (a union of this phase may already have cleared a finished root's state: its accumulator
        // then reads as all zero, ZERO again)
        const uint2 st = __ldcg(reinterpret_cast<const uint2 *>(b.rstate) + v);
        root = st.x <= st.y;
      }
      const uint32_t rootm = __ballot_sync(kFull, root);
      const uint32_t n = __popc(rootm);
      if (!n) continue;
      if (root) perm[__popc(rootm & ((1u << lane) - 1u))] = v;
      __syncwarp();
      const uint32_t vq = lane < n ? perm[lane] : 0u;
      __syncwarp();
      auto issue = [&](uint32_t t) {
        const uint32_t m = t * KB + lane;
        const uint32_t vm = __shfl_sync(kFull, vq, m & 31);
        const bool mine = lane < (uint32_t)KB && m < n;
        const uint32_t *ac = b.racc + (uint64_t)(mine ? vm : 0) * SW;
        ring.issue(T + t, mine, ac, W, ac + W, KB);
        return slot_offsets(ac, ac + W);
      };
      const uint32_t nb = (n + KB - 1) / KB;
      int my_res = 1;
      uint64_t my_idx = 0;
      uint32_t offs = issue(0);
      for (uint32_t t = 0; t < nb; ++t) {
        const uint32_t offs_next = t + 1 < nb ? issue(t + 1) : 0u;
        if (!landed(t, t + 1 < nb)) break;
        const uint32_t nm = min((uint32_t)KB, n - t * KB);
        uint64_t idx;
        const int res = sample_batch<CPS, KB>(ring.slot(T + t, 0, KB), ring.slot_bytes, ring.run_cap, offs, nm,
                                              t * KB, g.B, g.flip_chk, &idx);
        if (lane / KB == t) {
          my_res = res;
          my_idx = idx;
        }
        for (uint32_t k = 0; k < nm; ++k) {  // cleared for the next round
          uint4 *ac = reinterpret_cast<uint4 *>(b.racc + (uint64_t)__shfl_sync(kFull, vq, t * KB + k) * SW);
          for (uint32_t i = lane; i < SW / 4; i += 32) ac[i] = make_uint4(0, 0, 0, 0);
        }
        offs = offs_next;
        __syncwarp();
      }
      if (failed) break;
      T += nb;
      bool mod = false;
      if (lane < n) {
        uint32_t key = vq;
        if (trace) {
          key = __ldcg(b.minv + vq);
          b.minv[vq] = 0xffffffffu;
        }
        if (my_res == 1) b.rstate[2 * vq] = round + 1;
        mod = apply_result(my_res, my_idx, round, key, g, b);
      }
      if (mod) atomicOr(flags, 1u);
      __syncwarp();
    }
    if (!sync()) return;
  }
  // labels and the number of roots (one add per block)
  uint32_t roots = 0;
  for (uint32_t v0 = 0; v0 < V; v0 += nthreads) {
    const uint32_t v = v0 + gt;
    uint32_t r = 0xffffffffu;
    if (v < V) labels_out[v] = r = dsu_find(b.parent, once ? v : __ldcg(b.label + v));
    roots += __syncthreads_count(v < V && r == v);
  }
  if (tid == 0 && roots) atomicAdd(ncc, roots);
}

// Largest vertex count queried by one cluster, and its shape: a query of 1,024 vertices (6 rounds)
// took 60 us as a cluster and 82 us as a cooperative launch; at 8,192 vertices 138 against 96 us.
// Batches of 4 members there: twice the warps, each with half the serial work.
constexpr uint32_t kClusterMaxV = 2048;
constexpr int kClusterBlocks = 16;
constexpr int kClusterThreads = 512;

}  // namespace

size_t query_racc_words(uint32_t V, uint32_t cps, uint32_t B) { return (size_t)V * racc_words(cps, B); }

cudaError_t boruvka_query_launch(const BoruvkaGeom &g, uint32_t samples, const uint8_t *sketches,
                                 const BoruvkaBufs &b, uint32_t *labels_out, uint32_t *ncc,
                                 cudaStream_t s) {
  const uint32_t *sk = reinterpret_cast<const uint32_t *>(sketches);
  auto warp_bytes = [&](uint32_t KB) {
    return (size_t)bv_warp_bytes(std::max(3 * g.cps * g.B, kMinRingWords), (int)KB);
  };
  const int most = g.cps == 1 ? kBvqMaxThreads<1> : kBvqMaxThreads<7>;
  auto launch = [&](auto kern, uint32_t KB, auto kern_cluster, uint32_t KBC) -> cudaError_t {
    if (g.V <= kClusterMaxV) {
      const uint32_t nbatch = (g.V + KBC - 1) / KBC;
      cudaError_t e = smem_optin(kern_cluster);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
      // a warp per batch while there are batches for it, at most the cluster's warps
      int threads = std::min(kClusterThreads, most), blocks = 1;
      while (blocks < kClusterBlocks && (uint32_t)(blocks * threads / 32) < nbatch) blocks *= 2;
      while (threads > 64 && (uint32_t)(blocks * threads / 64) >= nbatch) threads /= 2;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(blocks);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = (threads / 32) * warp_bytes(KBC);
      cfg.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = blocks;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      e = cudaLaunchKernelEx(&cfg, kern_cluster, g, sk, b, samples, labels_out, ncc);
      if (e == cudaSuccess) {
        add_launches(1);
        return e;
      }
      cudaGetLastError();  // a cluster of this shape does not fit this GPU: the cooperative launch below
    }
    const uint32_t nbatch = (g.V + KB - 1) / KB;
    const size_t warp_smem = warp_bytes(KB);
    cudaError_t e = smem_optin(kern);
    if (e != cudaSuccess) return e;
    // one block per SM (a barrier's cost grows with its arrivals), the most warps its shared
    // memory holds
    int optin = 0, dev = 0;
    cudaFuncAttributes fa{};
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncGetAttributes(&fa, kern)) != cudaSuccess) return e;
    const int max_warps = (int)((optin - (int)fa.sharedSizeBytes) / warp_smem);
    // a warp per batch while there are batches for it
    const int want = (int)((nbatch + num_sms() - 1) / num_sms());
    const int threads = 32 * std::min(std::max(want, 2), std::min(most / 32, max_warps));
    const int blocks = std::min<int>(num_sms(), (int)((nbatch + threads / 32 - 1) / (threads / 32)));
    if ((e = cudaMemsetAsync(b.qbar, 0, sizeof(uint32_t), s)) != cudaSuccess) return e;
    BoruvkaGeom a_g = g;
    const uint32_t *a_sk = sk;
    BoruvkaBufs a_b = b;
    uint32_t a_samples = samples;
    uint32_t *a_labels = labels_out, *a_ncc = ncc;
    void *args[] = {&a_g, &a_sk, &a_b, &a_samples, &a_labels, &a_ncc};
    // every block resident at once (the launch fails otherwise): a barrier never waits for a block
    // that has not started
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kern), dim3(blocks), dim3(threads), args,
                                    (threads / 32) * warp_smem, s);
    add_launches(1);
    return e;
  };
  if (g.cps == 1 && g.B <= 42) return launch(k_bv_query<1, 4, 8, false>, 8, k_bv_query<1, 4, 4, true>, 4);
  if (g.cps == 1) return launch(k_bv_query<1, 6, 8, false>, 8, k_bv_query<1, 6, 4, true>, 4);
  if (g.cps == 7)
    return launch(k_bv_query<7, Region<7>::kNW, 1, false>, 1, k_bv_query<7, Region<7>::kNW, 1, true>, 1);
  return cudaErrorInvalidValue;
}

}  // namespace gz
