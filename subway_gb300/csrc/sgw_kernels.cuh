// Device kernels of the engine (sm_103a).
//
// Hot path per global iteration (reference: shared/subgraph_generator.cu:
// 128-204 and subway/*-{sync,async}.cu):
//   k_generate_count / k_generate_write (_pr: PageRank) activeness,
//                scan and compaction into the active queue (replaces
//                prePrefix, thrust::reduce, two thrust::exclusive_scan,
//                makeQueue, makeActiveNodesPointer), and the greedy partition
//                boundaries (Partitioner); k_plan: the boundaries on their own
//   k_gather_v   active-edge gather from the engine's mapped pinned transfer
//                copy of the edges into an HBM edge buffer, 16-byte reads
//                (replaces the host std::thread copy dynamic<E>); k_gather
//                is the one-record-per-thread form
//   k_relax_all  a first pass over a queue whose every source is active, cut by
//                edges; sync passes read the host copy themselves
//                (bfs/sssp/sswp/cc kernels, sync and async forms)
//   k_relax_warp label-driven expansion of 32 sources at a time by a warp
//                (later async inner iterations); k_relax_tile
//                the CTA-tile form staged in shared memory
//   k_relax_chunks warp-per-chunk expansion of high-degree sources
//   k_pr_all, k_pr_claim, k_pr_warp the same for PageRank
// Learned policy only (no reference counterpart):
//   k_select_*   value range, degree histogram and cut of the frontier when
//                far vertices are deferred
//   k_range_stats per-range features and the scheduler network's forward pass
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "sgw_internal.h"
#include "sgw_mlp.cuh"
#include "sgw_warp.cuh"

namespace sgw {

constexpr uint32_t kInf = 4294967294u;  // DIST_INFINITY (shared/globals.hpp:27)

// ---- device control block -------------------------------------------------
struct Part {                // one partition of the active queue
  uint32_t from;             // first queue index
  uint32_t size;             // queue entries
  uint32_t edge_from;        // ptr[from]
  uint32_t first_vertex;     // queue[from]
  unsigned long long edge_count;
};
constexpr uint32_t kCtlParts = 16;  // partitions reported with the control block

struct Ctl {
  uint32_t tile_done;        // finished tiles of the running generate
  uint32_t degree_max;       // largest degree queued so far by the running generate
  uint32_t error;            // nonzero: a device-side check failed
  uint32_t num_active;       // queued vertices (degree > 0) of the last generate
  unsigned long long num_active_edges;
  uint32_t num_parts;        // partitions of the last plan
  uint32_t max_degree;       // largest degree queued by the last generate
  uint32_t upd[4];           // async inner iteration k: relaxations that improved
  uint32_t wl_count[4];      // chunk-list items of inner iteration k
  uint32_t hub_active;       // single-vertex partition: the source was dirty
  uint32_t hub_value;        // single-vertex partition: its value
  uint32_t sel_bin;          // deferral: the last value bin selected this iteration
  uint32_t iters_total;      // inner iterations that did work, whole run
  unsigned long long reached_edges;
  unsigned long long relaxed_edges;
  unsigned long long relaxed_sources;
  unsigned long long host_edges;  // records that caching passes read from the host copy
  double hub_push;           // single-vertex PR partition: its push value
  Part first[kCtlParts];     // the partition table's first entries
};

struct WorkItem {            // a chunk of one high-degree source's edges
  uint32_t boff;             // first edge in the device edge buffer
  uint32_t count;            // edges in this chunk
  uint32_t value;            // source value snapshot
  uint32_t vertex;
};

// ---- small PTX helpers ----------------------------------------------------
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// First index in a[0, n) whose value is >= x (a sorted ascending), found by a
// warp in 32-way steps; every lane returns it.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t *a, uint32_t n, uint32_t x, int lane) {
  uint32_t lo = 0, hi = n;  // the answer is in [lo, hi]
  while (hi - lo > 32u) {
    const uint32_t step = (hi - lo + 31u) / 32u, i = lo + (uint32_t)lane * step;
    const uint32_t below = __ballot_sync(0xffffffffu, i < hi && a[i] < x);  // a prefix of lanes
    if (below == 0) return lo;
    const uint32_t k = 31u - (uint32_t)__clz((int)below);
    hi = min(hi, lo + (k + 1) * step);
    lo += k * step + 1;
  }
  const uint32_t i = lo + (uint32_t)lane;
  return lo + (uint32_t)__popc(__ballot_sync(0xffffffffu, i < hi && a[i] < x));
}

// ---- generate: activeness -> scan -> compaction --------------------------
constexpr int kGenThreads = 256;
constexpr int kGenRounds = 16;
constexpr uint32_t kGenTile = kGenThreads * kGenRounds;  // 4096 vertices

struct GenTotals {
  unsigned long long cnt, edges;
};

struct GenArgs {
  uint32_t n;
  uint8_t *l1;
  uint8_t *l2;
  const uint32_t *off;       // n + 1 node pointers (device copy)
  uint32_t *queue;           // activeNodes
  uint32_t *ptr;             // activeNodesPointer (count + 1)
  unsigned long long *tagg;  // per tile: queued vertices << 32 | edges (under an edge limit)
  GenTotals *runs;           // per CTA: the totals of its run of tiles
  uint32_t run_tiles;        // tiles per CTA
  Ctl *ctl;
  uint32_t *gmask;           // per 16-vertex group, keep bits | clear bits << 16 (null: recomputed)
  uint32_t *have;            // edge cache, per group: rows held | rows stored since << 16 (null: no cache)
  uint32_t num_tiles;
  int aligned;               // the label, pointer and value arrays start on 16-byte boundaries
  int consume;               // sync: labels of queued vertices are cleared
  // Most edges one generate queues (0: no limit).  Only
  // whole tiles are queued, in order, up to the limit (the first tile with
  // edges always); the later tiles keep their labels, and the count pass
  // leaves label clearing to the write pass of the tiles that are queued.
  uint32_t edge_limit = 0;
  // PageRank form (activeness delta > acc instead of labels)
  double *delta;             // pending residual per vertex
  double *pval;              // accumulated rank per vertex
  double *qpush;             // per queued vertex: damping * delta / outdeg
  double acc;
  double damping;
  // Value-aware selection (integer algorithms, learned policy), bit flags:
  // 1: active vertices that cannot push (BFS/SSSP value INF, SSWP value 0)
  //    are dropped like degree-0 ones, since relaxing them changes nothing;
  // 2: active vertices whose value lies beyond the bin chosen by
  //    k_select_pick are deferred (labels kept, not queued).
  int sel_mode = 0;
  int algo = 0;
  const uint32_t *value = nullptr;
  // Partition plan, made by the write pass's last CTA (null: none)
  Part *parts = nullptr;
  uint32_t max_parts = 0;
  unsigned long long cap = 0;
};

// Whether a vertex with this value produces candidates when relaxed.
__device__ __forceinline__ bool pushable(int algo, uint32_t v) {
  if (algo == SGW_BFS || algo == SGW_SSSP) return v != kInf;
  if (algo == SGW_SSWP) return v != 0;
  return true;
}

// Deferral bins: fixed and monotone in the value, so one pass builds the
// histogram: values below 64 get a bin each, larger ones 32 bins per power of
// two (bin < 896 of kSelBins).  Min-algorithms take the lowest bins first,
// SSWP (max) the highest.
constexpr uint32_t kSelBins = 1024;
__device__ __forceinline__ uint32_t sel_bin_of(uint32_t v) {
  if (v < 64u) return v;
  const uint32_t e = 31u - (uint32_t)__clz((int)v);
  return 64u + (e - 6u) * 32u + ((v >> (e - 5u)) & 31u);
}
__device__ __forceinline__ bool selected(int algo, uint32_t v, uint32_t bin) {
  const uint32_t b = sel_bin_of(v);
  return algo == SGW_SSWP ? b >= bin : b <= bin;
}

// Generate in two launches, with no chain between CTAs: k_generate_count and
// k_generate_write, each CTA a run of neighbouring 4096-vertex tiles (as many
// CTAs as fit on the GPU at once), 16 consecutive vertices per lane.  A lane
// reads its vertices' labels as two 16-byte words, the next tile's while it
// works on this one's,
// and, only if one of them is active, their 17 node pointers (and values, for
// the learned policy's selection) as 16-byte words.  The count pass stores
// each run's (queued vertices, edges) total; a CTA of the write pass sums the
// totals before its own, scans within its tiles, writes
// the queue and pointers in order and clears the consumed labels.  Labels
// and values do not change between the passes (nothing else runs on the
// stream in between), so both passes select the same vertices.
// Active vertices of degree 0 have nothing to relax: their labels are
// cleared here and they are not queued.
//
// Where the caller gives no room for the keep bits (the allocation-free entry
// point) the write pass selects again, from labels and pointers that are
// mostly still in L2.
//
// Bound by memory traffic on large graphs and by the launches on small ones.
// A single pass with a decoupled look-back was slower: with hundreds of tiles
// in flight the prefixes travel 32 tiles per round trip to L2 (a whole call of
// the allocation-free entry point on 16.8 M vertices, a quarter active: 181 us,
// two passes 78-87); so was a scan kernel of one CTA
// between the two (3.5 us per generate, 11 at 2^25 vertices), and giving each
// tile a CTA of its own, which sums the prefix once per tile (94 us).
constexpr uint32_t kGenVPerLane = 16;
constexpr int kGenCtas = 4;  // per SM; the grid is one wave of them (3: 87 us for the call above, 5: 87)

struct GenLabels {
  uint32_t l1w[4] = {0, 0, 0, 0}, l2w[4] = {0, 0, 0, 0};
};
struct GenLane : GenLabels {
  uint32_t keepmask = 0, clearmask = 0, cnt = 0, edges = 0, maxd = 0;
  uint32_t o[kGenVPerLane + 1];  // node pointers; a queued vertex's degree is o[k + 1] - o[k]
};

// The labels of the lane's 16 vertices starting at v0.
__device__ __forceinline__ void gen_labels(const GenArgs &a, uint32_t v0, bool full, GenLabels &L) {
  if (full) {
    const uint4 x = *reinterpret_cast<const uint4 *>(a.l1 + v0);
    const uint4 y = *reinterpret_cast<const uint4 *>(a.l2 + v0);
    L.l1w[0] = x.x; L.l1w[1] = x.y; L.l1w[2] = x.z; L.l1w[3] = x.w;
    L.l2w[0] = y.x; L.l2w[1] = y.y; L.l2w[2] = y.z; L.l2w[3] = y.w;
  } else {
    for (uint32_t k = 0; k < kGenVPerLane; ++k)
      if (v0 < a.n && v0 + k < a.n) {
        L.l1w[k / 4] |= (uint32_t)a.l1[v0 + k] << (8 * (k % 4));
        L.l2w[k / 4] |= (uint32_t)a.l2[v0 + k] << (8 * (k % 4));
      }
  }
}

// Selection for the lane's 16 vertices, whose labels L holds.  SEL: by value
// too (a.sel_mode).
template <bool SEL>
__device__ __forceinline__ void gen_select(const GenArgs &a, uint32_t v0, bool full, GenLane &L) {
  uint32_t sel_bin = 0;
  if (SEL && (a.sel_mode & 2)) sel_bin = a.ctl->sel_bin;
  uint32_t actmask = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t lw = L.l1w[q] | L.l2w[q];
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if ((lw >> (8 * b)) & 0xffu) actmask |= 1u << (4 * q + b);
  }
  if (!actmask) return;
  uint32_t val[kGenVPerLane];
  if (full) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 p = __ldg(reinterpret_cast<const uint4 *>(a.off + v0) + q);
      L.o[4 * q] = p.x; L.o[4 * q + 1] = p.y; L.o[4 * q + 2] = p.z; L.o[4 * q + 3] = p.w;
    }
    L.o[kGenVPerLane] = __ldg(&a.off[v0 + kGenVPerLane]);
    if (SEL) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 p = reinterpret_cast<const uint4 *>(a.value + v0)[q];
        val[4 * q] = p.x; val[4 * q + 1] = p.y; val[4 * q + 2] = p.z; val[4 * q + 3] = p.w;
      }
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k <= kGenVPerLane; ++k) L.o[k] = (v0 + k <= a.n) ? __ldg(&a.off[v0 + k]) : 0u;
#pragma unroll
    for (uint32_t k = 0; k < kGenVPerLane; ++k) val[k] = (SEL && v0 + k < a.n) ? a.value[v0 + k] : 0u;
  }
#pragma unroll
  for (uint32_t k = 0; k < kGenVPerLane; ++k) {
    if (!((actmask >> k) & 1u)) continue;
    uint32_t d = L.o[k + 1] - L.o[k];
    bool drop = d == 0, defer = false;
    if (SEL && !drop) {
      if (!pushable(a.algo, val[k])) drop = (a.sel_mode & 1) != 0;
      else if ((a.sel_mode & 2) && !selected(a.algo, val[k], sel_bin)) defer = true;
    }
    if (!defer && (a.consume || drop)) L.clearmask |= 1u << k;
    if (!drop && !defer) {
      L.keepmask |= 1u << k;
      ++L.cnt;
      L.edges += d;
      L.maxd = max(L.maxd, d);
    }
  }
}

// Clears the labels of the lane's vertices in L.clearmask (16-byte stores of
// the words that gen_labels read when the group is whole).
__device__ __forceinline__ void gen_clear(const GenArgs &a, uint32_t v0, bool full, const GenLane &L) {
  if (!L.clearmask) return;
  uint32_t cw[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    cw[q] = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if ((L.clearmask >> (4 * q + b)) & 1u) cw[q] |= 0xffu << (8 * b);
  }
  if (full) {
    *reinterpret_cast<uint4 *>(a.l1 + v0) =
        make_uint4(L.l1w[0] & ~cw[0], L.l1w[1] & ~cw[1], L.l1w[2] & ~cw[2], L.l1w[3] & ~cw[3]);
    *reinterpret_cast<uint4 *>(a.l2 + v0) =
        make_uint4(L.l2w[0] & ~cw[0], L.l2w[1] & ~cw[1], L.l2w[2] & ~cw[2], L.l2w[3] & ~cw[3]);
  } else {
    for (uint32_t k = 0; k < kGenVPerLane; ++k)
      if ((L.clearmask >> k) & 1u) { a.l1[v0 + k] = 0; a.l2[v0 + k] = 0; }
  }
}

// Sums of two words over the CTA, on every thread.
template <int THREADS>
__device__ __forceinline__ GenTotals gen_block_sum(GenTotals x, GenTotals *s_warp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    x.cnt += __shfl_xor_sync(0xffffffffu, x.cnt, d);
    x.edges += __shfl_xor_sync(0xffffffffu, x.edges, d);
  }
  if (lane == 0) s_warp[warp] = x;
  __syncthreads();
  GenTotals y{0, 0};
  if (lane < THREADS / 32) y = s_warp[lane];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    y.cnt += __shfl_xor_sync(0xffffffffu, y.cnt, d);
    y.edges += __shfl_xor_sync(0xffffffffu, y.edges, d);
  }
  return y;
}

// What the runs before this CTA's queue.
template <int THREADS>
__device__ __forceinline__ GenTotals gen_prefix(const GenArgs &a, GenTotals *s_warp) {
  GenTotals x{0, 0};
  for (uint32_t i = threadIdx.x; i < blockIdx.x; i += THREADS) {
    const GenTotals y = a.runs[i];
    x.cnt += y.cnt;
    x.edges += y.edges;
  }
  return gen_block_sum<THREADS>(x, s_warp);
}

// Whether a tile whose predecessors queue `before` is queued.  Under an edge
// limit the queued tiles are a prefix: those whose edges end within the limit,
// and the first with edges in any case.
__device__ __forceinline__ bool gen_queued(const GenArgs &a, unsigned long long before, unsigned long long own) {
  return !a.edge_limit || before + own <= a.edge_limit || before == 0;
}

// The totals and the pointer sentinel (subgraph_generator.cu:160), by one
// thread of the write pass: what the tiles before `tile` queue, called for the
// first tile that is not queued or past the last one.
__device__ __forceinline__ void gen_report(const GenArgs &a, const GenTotals &total) {
  a.ctl->num_active = (uint32_t)total.cnt;
  a.ctl->num_active_edges = total.edges;
  a.ptr[total.cnt] = (uint32_t)total.edges;
}

// One tile's turn in a write pass under an edge limit, on every thread: whether
// it is queued; the first that is not reports the totals.
__device__ __forceinline__ bool gen_limit(const GenArgs &a, uint32_t tile, const GenTotals &before) {
  if (gen_queued(a, before.edges, a.tagg[tile] & 0xffffffffull)) return true;
  // tile 0 is always queued, so there is a predecessor
  const unsigned long long prev = a.tagg[tile - 1] & 0xffffffffull;
  if (threadIdx.x == 0 && gen_queued(a, before.edges - prev, prev)) gen_report(a, before);
  return false;
}

__device__ void plan_cta(const uint32_t *ptr, const uint32_t *queue, Ctl *ctl, Part *parts, uint32_t max_parts,
                          unsigned long long cap);

// End of a CTA's write pass: the last one to finish makes the partition plan
// and readies the counters for the next generate.
__device__ __forceinline__ void gen_finish(const GenArgs &a, uint32_t *s_last) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *s_last = atomicAdd(&a.ctl->tile_done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!*s_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    a.ctl->tile_done = 0;
    a.ctl->max_degree = __ldcg(&a.ctl->degree_max);
    a.ctl->degree_max = 0;
  }
  if (a.parts) plan_cta(a.ptr, a.queue, a.ctl, a.parts, a.max_parts, a.cap);
}

// Rows that the passes since the last generate have stored in the edge cache are
// held from now on.
__device__ __forceinline__ void gen_have(const GenArgs &a, uint32_t v0) {
  const uint32_t h = a.have[v0 / kGenVPerLane];
  if (h >> 16) a.have[v0 / kGenVPerLane] = (h | h >> 16) & 0xffffu;
}

__device__ __forceinline__ uint32_t gen_v0(uint32_t tile) {
  return tile * kGenTile + (threadIdx.x >> 5) * (32 * kGenRounds) + (threadIdx.x & 31) * kGenVPerLane;
}
__device__ __forceinline__ bool gen_full(const GenArgs &a, uint32_t v0) {
  return a.aligned && v0 + kGenVPerLane <= a.n;
}

// Count pass: the selection of every lane's 16 vertices, whose keep and
// clear bits it records per group (so the write pass reads 4 bytes per 16
// vertices instead of the labels and values again), the label clearing, and
// the run's (count, edges) total.
template <bool SEL>
__global__ void __launch_bounds__(kGenThreads, kGenCtas) k_generate_count(GenArgs a) {
  chain_wait();
  chain_open();
  __shared__ GenTotals s_sum[kGenThreads / 32];
  const int lane = threadIdx.x & 31;
  const uint32_t t0 = blockIdx.x * a.run_tiles, t1 = min(a.num_tiles, t0 + a.run_tiles);
  GenTotals sum{0, 0};
  uint32_t maxd = 0;
  GenLabels next;
  gen_labels(a, gen_v0(t0), gen_full(a, gen_v0(t0)), next);
  for (uint32_t tile = t0; tile < t1; ++tile) {
    const uint32_t v0 = gen_v0(tile);
    const bool full = gen_full(a, v0);
    GenLane L;
    static_cast<GenLabels &>(L) = next;
    next = GenLabels();
    if (tile + 1 < t1) gen_labels(a, gen_v0(tile + 1), gen_full(a, gen_v0(tile + 1)), next);
    if (v0 < a.n) {
      if (a.have) gen_have(a, v0);
      gen_select<SEL>(a, v0, full, L);
      if (a.gmask) {
        if (!a.edge_limit) gen_clear(a, v0, full, L);
        a.gmask[v0 / kGenVPerLane] = L.keepmask | (L.clearmask << 16);
      }
    }
    sum.cnt += L.cnt;
    sum.edges += L.edges;
    maxd = max(maxd, L.maxd);
    if (a.edge_limit) {
      const GenTotals t = gen_block_sum<kGenThreads>(GenTotals{L.cnt, L.edges}, s_sum);
      if (threadIdx.x == 0) a.tagg[tile] = t.cnt << 32 | t.edges;
      __syncthreads();
    }
  }
  maxd = __reduce_max_sync(0xffffffffu, maxd);
  if (lane == 0 && maxd && a.gmask) atomicMax(&a.ctl->degree_max, maxd);
  sum = gen_block_sum<kGenThreads>(sum, s_sum);
  if (threadIdx.x == 0) a.runs[blockIdx.x] = sum;
}

// Write pass: the group's keep bits from the count pass (MASKS: the engine's
// generate) or selected again (a caller's arrays, where there is no room for the
// bits, no plan to make and no counter to ready: 77 us for 16.8 M vertices, 86
// with a memset of the control block and the last CTA's turn), the node pointers
// of groups that queue a vertex, and the queue / pointer entries.
template <bool MASKS>
__global__ void __launch_bounds__(kGenThreads, kGenCtas) k_generate_write(GenArgs a) {
  chain_wait();
  chain_open();
  __shared__ GenTotals s_sum[kGenThreads / 32];
  __shared__ unsigned long long s_warp[2][kGenThreads / 32];
  __shared__ uint32_t s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t t0 = blockIdx.x * a.run_tiles, t1 = min(a.num_tiles, t0 + a.run_tiles);
  GenLabels next;
  uint32_t next_gm = 0;
  auto fetch = [&](uint32_t tile) {
    const uint32_t v0 = gen_v0(tile);
    next = GenLabels();
    next_gm = 0;
    if (MASKS) {
      if (v0 < a.n) next_gm = a.gmask[v0 / kGenVPerLane];
    } else {
      gen_labels(a, v0, gen_full(a, v0), next);
    }
  };
  fetch(t0);  // goes out before the prefix's loads
  GenTotals before = gen_prefix<kGenThreads>(a, s_sum);
  bool cut = false;
  for (uint32_t tile = t0; tile < t1; ++tile) {
    const uint32_t v0 = gen_v0(tile);
    const bool full = gen_full(a, v0);
    GenLane L;
    static_cast<GenLabels &>(L) = next;
    const uint32_t gm = next_gm;
    if (tile + 1 < t1) fetch(tile + 1);
    if (a.edge_limit && !gen_limit(a, tile, before)) {  // beyond the limit, as all later tiles: labels kept
      cut = true;
      break;
    }
    if (!MASKS) {
      if (v0 < a.n) {
        gen_select<false>(a, v0, full, L);
        gen_clear(a, v0, full, L);
      }
    } else {
      L.keepmask = gm & 0xffffu;
      if (a.edge_limit && (gm >> 16)) {  // the clearing the count pass left to this tile
        gen_labels(a, v0, full, L);
        L.clearmask = gm >> 16;
        gen_clear(a, v0, full, L);
      }
      if (L.keepmask) {
        if (full) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 p = __ldg(reinterpret_cast<const uint4 *>(a.off + v0) + q);
            L.o[4 * q] = p.x; L.o[4 * q + 1] = p.y; L.o[4 * q + 2] = p.z; L.o[4 * q + 3] = p.w;
          }
          L.o[kGenVPerLane] = __ldg(&a.off[v0 + kGenVPerLane]);
        } else {
#pragma unroll
          for (uint32_t k = 0; k <= kGenVPerLane; ++k) L.o[k] = (v0 + k <= a.n) ? __ldg(&a.off[v0 + k]) : 0u;
        }
        L.cnt = (uint32_t)__popc(L.keepmask);
#pragma unroll
        for (uint32_t k = 0; k < kGenVPerLane; ++k)
          if ((L.keepmask >> k) & 1u) L.edges += L.o[k + 1] - L.o[k];
      }
    }
    if (!__syncthreads_or(L.keepmask != 0)) continue;  // a tile that queues nothing
    const uint32_t incl_c = warp_incl_scan(L.cnt, lane);
    const uint32_t incl_e = warp_incl_scan(L.edges, lane);
    unsigned long long *const sums = s_warp[tile & 1u];  // the other half may still be read
    if (lane == 31) sums[warp] = ((unsigned long long)incl_c << 32) | incl_e;
    __syncthreads();
    // positions stay below 2^32: so do the edges of a queue
    uint32_t pos = (uint32_t)before.cnt + incl_c - L.cnt, ep = (uint32_t)before.edges + incl_e - L.edges;
#pragma unroll
    for (int w = 0; w < kGenThreads / 32; ++w) {
      const unsigned long long x = sums[w];
      before.cnt += x >> 32;
      before.edges += x & 0xffffffffull;
      if (w < warp) {
        pos += (uint32_t)(x >> 32);
        ep += (uint32_t)x;
      }
    }
    if (L.keepmask) {
#pragma unroll
      for (uint32_t k = 0; k < kGenVPerLane; ++k) {
        if ((L.keepmask >> k) & 1u) {
          const uint32_t d = L.o[k + 1] - L.o[k];
          a.queue[pos] = v0 + k;
          a.ptr[pos] = ep;
          ++pos;
          ep += d;
        }
      }
    }
  }
  // past the last tile: the totals, unless a tile was beyond the limit
  if (t1 == a.num_tiles && !cut && tid == 0) gen_report(a, before);
  if (MASKS) gen_finish(a, &s_last);
}

// PageRank's two passes (prePrefix PR overload, shared/subgraph_generator.cu:
// 24-41): active = delta > acc; the queue takes the active vertices with
// out-edges.  A tile of 4096 vertices by 1024 threads, four neighbouring-lane
// rounds each, so the 8-byte residuals and ranks are read and written
// coalesced, two CTAs per SM.  PageRank's generate at 2^20 vertices, plan included:
// 34 us and four launches before, 28 us and two now.  The write pass moves every active vertex's residual into
// its rank (value += delta, delta = 0, the first half of pr_kernel,
// shared/gpu_kernels.cu:234-250); its queue entry carries the push
// damping * delta / outdeg, so each round is a bulk-synchronous snapshot.
constexpr int kGenPrThreads = 1024;
constexpr int kGenPrRounds = kGenTile / kGenPrThreads;

// x > acc for acc > 0, as integers (a 64-bit floating-point compare holds a warp
// for about 15 cycles): non-negative doubles order as their bits, negative
// ones have the sign bit, and NaN is not above anything.
__device__ __forceinline__ bool pr_above(double x, double acc) {
  const long long b = __double_as_longlong(x);
  return b > __double_as_longlong(acc) && b <= 0x7ff0000000000000ll;
}

__device__ __forceinline__ void gen_pr_select(const GenArgs &a, uint32_t tile, double (&dl)[kGenPrRounds],
                                              uint32_t (&deg)[kGenPrRounds]) {
#pragma unroll
  for (int r = 0; r < kGenPrRounds; ++r) {
    const uint32_t v = tile * kGenTile + r * kGenPrThreads + threadIdx.x;
    dl[r] = v < a.n ? a.delta[v] : 0.0;
  }
#pragma unroll
  for (int r = 0; r < kGenPrRounds; ++r) {
    const uint32_t v = tile * kGenTile + r * kGenPrThreads + threadIdx.x;
    deg[r] = v < a.n && pr_above(dl[r], a.acc) ? __ldg(&a.off[v + 1]) - __ldg(&a.off[v]) : 0u;
  }
}

__global__ void __launch_bounds__(kGenPrThreads, 2) k_generate_count_pr(GenArgs a) {
  chain_wait();
  chain_open();
  __shared__ GenTotals s_sum[kGenPrThreads / 32];
  const uint32_t t0 = blockIdx.x * a.run_tiles, t1 = min(a.num_tiles, t0 + a.run_tiles);
  GenTotals sum{0, 0};
  uint32_t maxd = 0;
  for (uint32_t tile = t0; tile < t1; ++tile) {
    double dl[kGenPrRounds];
    uint32_t deg[kGenPrRounds];
    if (a.have && threadIdx.x % kGenVPerLane == 0)
#pragma unroll
      for (int r = 0; r < kGenPrRounds; ++r) {
        const uint32_t v = tile * kGenTile + r * kGenPrThreads + threadIdx.x;
        if (v < a.n) gen_have(a, v);
      }
    gen_pr_select(a, tile, dl, deg);
    GenTotals x{0, 0};
#pragma unroll
    for (int r = 0; r < kGenPrRounds; ++r) {
      x.cnt += deg[r] > 0;
      x.edges += deg[r];
      maxd = max(maxd, deg[r]);
    }
    sum.cnt += x.cnt;
    sum.edges += x.edges;
    if (a.edge_limit) {
      x = gen_block_sum<kGenPrThreads>(x, s_sum);
      if (threadIdx.x == 0) a.tagg[tile] = x.cnt << 32 | x.edges;
      __syncthreads();
    }
  }
  maxd = __reduce_max_sync(0xffffffffu, maxd);
  if ((threadIdx.x & 31) == 0 && maxd) atomicMax(&a.ctl->degree_max, maxd);
  sum = gen_block_sum<kGenPrThreads>(sum, s_sum);
  if (threadIdx.x == 0) a.runs[blockIdx.x] = sum;
}

__global__ void __launch_bounds__(kGenPrThreads, 2) k_generate_write_pr(GenArgs a) {
  chain_wait();
  chain_open();
  constexpr int kWarps = kGenPrThreads / 32, kParts = kGenPrRounds * kWarps;
  __shared__ GenTotals s_sum[kWarps];
  __shared__ unsigned long long s_part[kParts + 1];  // (round, warp): count << 32 | edges, then the tile's total
  __shared__ uint32_t s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t t0 = blockIdx.x * a.run_tiles, t1 = min(a.num_tiles, t0 + a.run_tiles);
  GenTotals before = gen_prefix<kGenPrThreads>(a, s_sum);
  bool cut = false;
  for (uint32_t tile = t0; tile < t1; ++tile) {
    if (a.edge_limit && !gen_limit(a, tile, before)) {  // beyond the limit: residuals kept
      cut = true;
      break;
    }
    double dl[kGenPrRounds];
    uint32_t deg[kGenPrRounds], incl[kGenPrRounds];
    gen_pr_select(a, tile, dl, deg);
#pragma unroll
    for (int r = 0; r < kGenPrRounds; ++r) {
      incl[r] = warp_incl_scan(deg[r], lane);
      const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, deg[r] > 0));
      if (lane == 31) s_part[r * kWarps + warp] = ((unsigned long long)c << 32) | incl[r];
    }
    __syncthreads();
    if (warp == 0) {  // exclusive prefixes in (round, warp) order, kGenPrRounds entries per lane
      unsigned long long x[kGenPrRounds], sum = 0;
#pragma unroll
      for (int k = 0; k < kGenPrRounds; ++k) {
        x[k] = s_part[lane * kGenPrRounds + k];
        sum += x[k];
      }
      unsigned long long run = sum;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, run, d);
        if (lane >= d) run += y;
      }
      if (lane == 31) s_part[kParts] = run;
      run -= sum;
#pragma unroll
      for (int k = 0; k < kGenPrRounds; ++k) {
        s_part[lane * kGenPrRounds + k] = run;
        run += x[k];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kGenPrRounds; ++r) {
      const uint32_t v = tile * kGenTile + r * kGenPrThreads + tid;
      const uint32_t keep = __ballot_sync(0xffffffffu, deg[r] > 0);
      if (v < a.n && pr_above(dl[r], a.acc)) {  // every active vertex, queued or of degree 0
        a.pval[v] += dl[r];
        a.delta[v] = 0.0;
      }
      if (deg[r]) {
        const unsigned long long p = s_part[r * kWarps + warp];
        const uint32_t pos = (uint32_t)before.cnt + (uint32_t)(p >> 32) + __popc(keep & lanemask_lt());
        a.queue[pos] = v;
        a.ptr[pos] = (uint32_t)before.edges + (uint32_t)p + incl[r] - deg[r];
        a.qpush[pos] = a.damping * dl[r];
      }
    }
    // the divisions, over the tile's queue entries instead of its vertices: a
    // 64-bit division holds a warp for a few hundred cycles whether one of its
    // lanes needs it or all
    const unsigned long long total = s_part[kParts];
    const uint32_t cnt = (uint32_t)(total >> 32), end = (uint32_t)before.edges + (uint32_t)total;
    __syncthreads();
    for (uint32_t i = tid; i < cnt; i += kGenPrThreads) {
      const uint32_t pos = (uint32_t)before.cnt + i;
      const uint32_t d = (i + 1 < cnt ? a.ptr[pos + 1] : end) - a.ptr[pos];
      a.qpush[pos] = a.qpush[pos] / (double)d;
    }
    before.cnt += cnt;
    before.edges += total & 0xffffffffull;
  }
  if (t1 == a.num_tiles && !cut && tid == 0) gen_report(a, before);
  gen_finish(a, &s_last);
}

// ---- frontier deferral (learned policy) --------------------------------------
// Before a generate, two small passes pick how much of the frontier to take:
// a histogram of the pushable active vertices' out-degrees over the fixed
// value bins, and the bin at which the cumulative degree reaches the target
// (lowest values first; highest for SSWP).  The
// generate then queues only the selected vertices; the rest keep their labels
// for a later iteration.  Relaxing far vertices first wastes their edges'
// transfer when they improve again later; this is the delta-stepping idea
// applied to out-of-memory partitions.
// Visits the pushable active vertices of degree > 0: each thread reads the
// two label arrays 16 bytes at a time (label arrays are 256-byte aligned),
// so a pass over n vertices keeps enough loads in flight to run at memory
// speed; only active vertices read their pointers and value.
template <class F>
__device__ __forceinline__ void for_sel_candidates(uint32_t n, int algo, const uint8_t *l1, const uint8_t *l2,
                                                   const uint32_t *off, const uint32_t *value, F f) {
  const uint32_t nvec = n / 16u;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  auto visit = [&](uint32_t v) {
    const uint32_t deg = __ldg(&off[v + 1]) - __ldg(&off[v]);
    if (deg == 0) return;
    const uint32_t val = value[v];
    if (pushable(algo, val)) f(val, deg);
  };
  for (uint32_t i = tid; i < nvec; i += nth) {
    const uint4 a = reinterpret_cast<const uint4 *>(l1)[i];
    const uint4 b = reinterpret_cast<const uint4 *>(l2)[i];
    const uint32_t w[4] = {a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (w[q] == 0) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if ((w[q] >> (8 * k)) & 0xffu) visit(16u * i + 4u * q + k);
    }
  }
  for (uint32_t v = 16u * nvec + tid; v < n; v += nth)
    if ((l1[v] | l2[v]) != 0) visit(v);
}

// Per-CTA bins in shared memory (per-CTA sums stay below m < 2^32), added
// into 64-bit global bins at the end.
__global__ void __launch_bounds__(256) k_select_hist(uint32_t n, int algo, const uint8_t *l1, const uint8_t *l2,
                                                     const uint32_t *off, const uint32_t *value, const Ctl *ctl,
                                                     unsigned long long *hist) {
  __shared__ uint32_t s_hist[kSelBins];
  for (uint32_t i = threadIdx.x; i < kSelBins; i += blockDim.x) s_hist[i] = 0u;
  __syncthreads();
  for_sel_candidates(n, algo, l1, l2, off, value,
                     [&](uint32_t val, uint32_t deg) { atomicAdd(&s_hist[sel_bin_of(val)], deg); });
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < kSelBins; i += blockDim.x)
    if (s_hist[i]) atomicAdd(&hist[i], (unsigned long long)s_hist[i]);
}

// One CTA of kSelBins / 4 threads: cumulative degree over the bins in
// selection order; sel_bin = first bin at which it reaches `target`.
__global__ void __launch_bounds__(kSelBins / 4) k_select_pick(int algo, const unsigned long long *hist,
                                                              unsigned long long target, Ctl *ctl) {
  chain_wait();
  chain_open();
  __shared__ unsigned long long s_part[kSelBins / 4 / 32];
  __shared__ uint32_t s_k;  // first position (selection order) reaching the target
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool rev = algo == SGW_SSWP;
  if (tid == 0) s_k = kSelBins - 1u;  // target never reached: take everything
  // thread t owns 4 consecutive bins in selection order
  unsigned long long h[4], mine = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t k = 4u * tid + q;
    h[q] = hist[rev ? kSelBins - 1u - k : k];
    mine += h[q];
  }
  unsigned long long incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) s_part[warp] = incl;
  __syncthreads();
  if (tid == 0) {
    unsigned long long acc = 0;
    for (int w = 0; w < (int)(kSelBins / 4 / 32); ++w) {
      const unsigned long long x = s_part[w];
      s_part[w] = acc;
      acc += x;
    }
  }
  __syncthreads();
  unsigned long long run = s_part[warp] + incl - mine;
  uint32_t first = 0xffffffffu;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    run += h[q];
    if (first == 0xffffffffu && h[q] && run >= target) first = 4u * tid + q;
  }
  if (first != 0xffffffffu) atomicMin(&s_k, first);
  __syncthreads();
  if (tid == 0) ctl->sel_bin = rev ? kSelBins - 1u - s_k : s_k;
}

// ---- partition planner ------------------------------------------------------
// One CTA.  For each partition: the largest run of queue entries starting at
// `from` whose edges fit `cap`, found by a search as many ways as the CTA has
// threads (each step probes evenly spaced entries and keeps the bracket of the
// last one that fits: two round trips to L2 for 64 K entries and 256 threads,
// where one warp takes four).
// Loads go through L2: the CTAs of the generate that runs it wrote the queue.
__device__ void plan_cta(const uint32_t *ptr, const uint32_t *queue, Ctl *ctl, Part *parts, uint32_t max_parts,
                         unsigned long long cap) {
  const uint32_t tid = threadIdx.x, nth = blockDim.x;
  const uint32_t count = __ldcg(&ctl->num_active);
  const unsigned long long edges = __ldcg(&ctl->num_active_edges);
  uint32_t from = 0, p = 0;
  if (count && edges <= cap) {  // everything in one partition: nothing to search
    if (tid == 0) {
      const Part q{0, count, 0, __ldcg(&queue[0]), edges};
      if (max_parts) parts[0] = q;
      ctl->first[0] = q;
    }
    from = count;
    p = 1;
  }
  while (from < count) {
    const uint32_t start = __ldcg(&ptr[from]);
    const unsigned long long limit = (unsigned long long)start + cap;
    // answer t in [from, count]: largest index with ptr[t] <= limit
    uint32_t lo = from + 1, hi = count;  // candidates above `from`
    uint32_t best = from;
    while (lo <= hi) {
      const uint32_t span = hi - lo + 1;
      const uint32_t step = (span + nth - 1) / nth;
      const unsigned long long idx = lo + (unsigned long long)tid * step;
      const bool ok = idx <= hi && (unsigned long long)__ldcg(&ptr[idx]) <= limit;
      const uint32_t k = (uint32_t)__syncthreads_count(ok);  // ok is a prefix of the threads
      if (k == 0) break;
      const uint32_t last_ok = lo + (k - 1) * step;
      best = last_ok;
      if (step == 1) break;
      lo = last_ok + 1;
      const unsigned long long next_bad = (unsigned long long)last_ok + step;  // first probe that failed
      if (k < nth && next_bad - 1 < hi) hi = (uint32_t)next_bad - 1;
    }
    const uint32_t to = best > from ? best : from + 1;  // a vertex beyond cap runs alone
    if (tid == 0 && p < max_parts) {
      Part q;
      q.from = from;
      q.size = to - from;
      q.edge_from = start;
      q.first_vertex = __ldcg(&queue[from]);
      q.edge_count = (unsigned long long)__ldcg(&ptr[to]) - start;
      parts[p] = q;
      if (p < kCtlParts) ctl->first[p] = q;
    }
    ++p;
    from = to;
  }
  if (tid == 0) {
    ctl->num_parts = p;
    if (p > max_parts) atomicExch(&ctl->error, 2u);
  }
}

// The plan on its own (the step API's sgw_partition).
__global__ void k_plan(const uint32_t *ptr, const uint32_t *queue, Ctl *ctl, Part *parts, uint32_t max_parts,
                       unsigned long long cap) {
  plan_cta(ptr, queue, ctl, parts, max_parts, cap);
}

// ---- gather: host CSR -> device edge buffer -------------------------------
// The engine's host transfer copy is a series of pinned chunks of 2^shift
// bytes (allocated by two host threads at once, which halves the set-up of
// a 21 GB copy); base is a device table of their device addresses.  A
// 16-byte word or a record never straddles two chunks.
struct HostChunks {
  const unsigned long long *base;
  uint32_t shift;
};

__device__ __forceinline__ const char *hc_at(const HostChunks &h, size_t byte) {
  const char *c = reinterpret_cast<const char *>(__ldg(h.base + (byte >> h.shift)));
  return c + (byte & ((size_t(1) << h.shift) - 1));
}

// Copies bytes [off, off + bytes) of a host stream to dst, for streams in
// pageable memory (read through the host page tables), where a DMA copy would
// be staged by the host thread.  Each thread reads one aligned 16-byte word of
// the stream (words never straddle chunks) and stores the part in range as
// one 16-byte word, four 4-byte words or single bytes, whichever the two
// addresses' alignment allows.  Chunks are padded to 16 bytes, so the words at
// either end stay inside their chunk.
__global__ void __launch_bounds__(256) k_copy_host(HostChunks src, unsigned long long off,
                                                   unsigned long long bytes, uint8_t *__restrict__ dst) {
  const unsigned long long w0 = off >> 4, w1 = (off + bytes + 15) >> 4, end = off + bytes;
  const unsigned long long skew = (reinterpret_cast<uintptr_t>(dst) - off) & 15;
  for (unsigned long long w = w0 + blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; w < w1;
       w += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long s = w << 4;
    const uint4 v = *reinterpret_cast<const uint4 *>(hc_at(src, s));
    if (skew == 0 && s >= off && s + 16 <= end) {
      *reinterpret_cast<uint4 *>(dst + (s - off)) = v;
      continue;
    }
    const uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned long long a = s + 4 * k;
      if ((skew & 3) == 0 && a >= off && a + 4 <= end) {
        *reinterpret_cast<uint32_t *>(dst + (a - off)) = q[k];
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (a + i >= off && a + i < end) dst[a + i - off] = (uint8_t)(q[k] >> (8 * i));
      }
    }
  }
}

constexpr int kGatherThreads = 256;
// Output edges per CTA tile of the vectorised gather (its shared memory is
// dynamic: 16 bytes per tile edge plus the weight bytes); the scalar gather
// keeps 2048.
#ifndef SGW_GATHER_TILE
#define SGW_GATHER_TILE 2048
#endif
constexpr uint32_t kGatherTile = SGW_GATHER_TILE;
constexpr uint32_t kScalarGatherTile = 2048;

// Index of the last element <= x in a[0..len) (a non-decreasing, a[0] <= x).
__device__ __forceinline__ uint32_t last_le(const uint32_t *a, uint32_t len, uint32_t x) {
  uint32_t lo = 0, hi = len;  // first index with a[i] > x in [lo, hi)
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (a[mid] <= x) lo = mid + 1; else hi = mid;
  }
  return lo - 1;
}

// Last queue index i in [lo, hi) with ptr[i] - edge_from <= target, found by
// one warp in 32-way steps (about five dependent loads for 2^24 entries
// instead of one per halving).  ptr is non-decreasing and
// ptr[lo] - edge_from <= target.  Every lane returns the answer.
__device__ __forceinline__ uint32_t warp_last_le(const uint32_t *__restrict__ ptr, uint32_t lo, uint32_t hi,
                                                 uint32_t edge_from, uint32_t target, int lane) {
  while (hi - lo > 32u) {
    const uint32_t step = (hi - lo + 31u) / 32u;
    const uint32_t idx = lo + (uint32_t)lane * step;
    const bool le = idx < hi && ptr[idx] - edge_from <= target;
    const uint32_t m = __ballot_sync(0xffffffffu, le);  // a prefix of lanes; lane 0 always
    const uint32_t k = 31u - (uint32_t)__clz((int)m);
    lo += k * step;
    hi = min(hi, lo + step);
  }
  const uint32_t idx = lo + (uint32_t)lane;
  const bool le = idx < hi && ptr[idx] - edge_from <= target;
  const uint32_t m = __ballot_sync(0xffffffffu, le);
  return lo + 31u - (uint32_t)__clz((int)m);
}

// Copies the edges of queue entries [from, from+size) from the mapped host
// CSR to buf[0 .. edge_count).  Output positions are balanced per CTA; each
// CTA stages the (buffer offset, host offset) of the sources its tile covers
// in shared memory and every thread copies edges by binary search in it.
// Consecutive threads read consecutive host edges of one source, so host
// reads are coalesced; E is the edge record (one or two u32 words).
template <int W, bool WIDE>
__global__ void __launch_bounds__(kGatherThreads) k_gather(
    const uint32_t *__restrict__ queue, const uint32_t *__restrict__ ptr,
    const uint32_t *__restrict__ off, const unsigned long long *__restrict__ obase, HostChunks host_edges,
    uint32_t *__restrict__ buf, uint32_t from, uint32_t size, uint32_t edge_from,
    uint32_t edge_count) {
  using HP = typename std::conditional<WIDE, unsigned long long, uint32_t>::type;
  __shared__ uint32_t s_bpos[kScalarGatherTile + 1];
  __shared__ HP s_hpos[kScalarGatherTile + 1];
  __shared__ uint32_t s_first, s_last;
  const uint32_t ntiles = (edge_count + kScalarGatherTile - 1) / kScalarGatherTile;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint32_t j0 = t * kScalarGatherTile;
    const uint32_t j1 = min(edge_count, j0 + kScalarGatherTile);
    // sources covering [j0, j1): warp 0 finds the first, warp 1 the last
    if (threadIdx.x < 64) {
      const int lane = threadIdx.x & 31;
      const uint32_t r = warp_last_le(ptr, from, from + size, edge_from, threadIdx.x < 32 ? j0 : j1 - 1, lane);
      if (lane == 0) (threadIdx.x < 32 ? s_first : s_last) = r;
    }
    __syncthreads();
    const uint32_t first = s_first, nsrc = s_last - s_first + 1;
    for (uint32_t k = threadIdx.x; k < nsrc; k += blockDim.x) {
      const uint32_t i = first + k;
      s_bpos[k] = ptr[i] - edge_from;
      s_hpos[k] = WIDE ? (HP)off_at(off, obase, queue[i]) : (HP)off[queue[i]];
    }
    __syncthreads();
    // four independent host loads in flight per thread before any store
    constexpr int U = 4;
    for (uint32_t jb = j0 + threadIdx.x; jb < j1; jb += U * blockDim.x) {
      uint2 e[U];
      uint32_t jj[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t j = jb + u * blockDim.x;
        jj[u] = j;
        if (j < j1) {
          const uint32_t k = last_le(s_bpos, nsrc, j);
          const size_t h = (size_t)s_hpos[k] + (j - s_bpos[k]);
          if (W == 1) e[u].x = *reinterpret_cast<const uint32_t *>(hc_at(host_edges, h * 4));
          else e[u] = *reinterpret_cast<const uint2 *>(hc_at(host_edges, h * 8));
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (jj[u] < j1) {
          if (W == 1) buf[jj[u]] = e[u].x;
          else reinterpret_cast<uint2 *>(buf)[jj[u]] = e[u];
        }
      }
    }
    __syncthreads();
  }
}

// Same tiling as k_gather, but host memory is read as aligned 16-byte words:
// each source's clipped host range is covered by ceil-aligned chunks of
// R = 16 / RB records of RB bytes, the CTA scans the chunk counts of its
// tile's sources, and every thread loads whole chunks (4 in flight) and
// scatters the records that belong to the source into the device buffer.
// RB = 4 (one word per edge) or 8 (the reference's {end, w8}).  With WS the
// split form's weight bytes of the same edges follow in the same tile (same
// source ranges, chunks of 16 weights), put together in shared memory and
// stored as 16-byte words.  Needs 16-byte aligned host arrays (the engine's
// own allocations are 64 KiB aligned).
constexpr uint32_t kGatherPer = (kGatherTile + kGatherThreads - 1) / kGatherThreads;

// Exclusive scan of the tile's per-source chunk counts (R records per
// chunk) into s_cs; returns the tile's chunk total.
template <uint32_t R>
__device__ __forceinline__ uint32_t gather_scan(uint32_t nsrc, const uint32_t *s_hlo, const uint32_t *s_len,
                                                uint32_t *s_cs, uint32_t *s_part) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto chunks = [&](uint32_t k) {  // depends on the source's record mod R only
    return (s_hlo[k] % R + s_len[k] + R - 1) / R;
  };
  uint32_t part = 0;
  for (uint32_t q = 0; q < kGatherPer; ++q) {
    const uint32_t k = tid * kGatherPer + q;
    if (k < nsrc) part += chunks(k);
  }
  const uint32_t incl = warp_incl_scan(part, lane);
  if (lane == 31) s_part[warp] = incl;
  __syncthreads();
  if (tid == 0) {
    uint32_t acc = 0;
    for (int w = 0; w < kGatherThreads / 32; ++w) { uint32_t x = s_part[w]; s_part[w] = acc; acc += x; }
    s_part[kGatherThreads] = acc;
  }
  __syncthreads();
  uint32_t run = s_part[warp] + incl - part;
  for (uint32_t q = 0; q < kGatherPer; ++q) {
    const uint32_t k = tid * kGatherPer + q;
    if (k < nsrc) { s_cs[k] = run; run += chunks(k); }
  }
  __syncthreads();
  return s_part[kGatherThreads];
}

// Copies the tile's chunks of RB-byte records: RB 4 / 8 straight into buf,
// RB 1 into the shared byte tile at position - j0.  A source's first record
// is (s_hhi:s_hlo), s_hhi only with WIDE; a chunk's records are matched to
// the source by their distance from it, which fits 32 bits.
template <int RB, bool WIDE>
__device__ __forceinline__ void gather_copy(uint32_t total, uint32_t nsrc, uint32_t j0, const uint32_t *s_cs,
                                            const uint32_t *s_hlo, const uint32_t *s_hhi, const uint32_t *s_len,
                                            const uint32_t *s_bpos, const HostChunks &host16,
                                            void *__restrict__ buf, uint8_t *s_bytes) {
  using CT = typename std::conditional<WIDE, unsigned long long, uint32_t>::type;
  constexpr uint32_t R = 16 / RB;
  constexpr int U = 4;
  for (uint32_t jb = threadIdx.x; jb < total; jb += U * blockDim.x) {
    uint4 v[U];
    uint32_t kk[U];
    CT cc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t j = jb + u * blockDim.x;
      kk[u] = 0xffffffffu;
      if (j < total) {
        const uint32_t k = last_le(s_cs, nsrc, j);
        CT h = s_hlo[k];
        if (WIDE) h |= (CT)s_hhi[k] << (WIDE ? 32 : 0);
        const CT c = h / R + (j - s_cs[k]);
        kk[u] = k;
        cc[u] = c;
        v[u] = *reinterpret_cast<const uint4 *>(hc_at(host16, (size_t)c << 4));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (kk[u] == 0xffffffffu) continue;
      const uint32_t k = kk[u];
      const uint32_t len = s_len[k], bpos = s_bpos[k];
      // distance of the chunk's first record from the source's first (mod 2^32)
      const uint32_t d0 = (uint32_t)cc[u] * R - s_hlo[k];
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (uint32_t r = 0; r < R; ++r) {
        const uint32_t d = d0 + r;
        if (d < len) {
          const uint32_t o = bpos + d;
          if (RB == 4) reinterpret_cast<uint32_t *>(buf)[o] = w[r];
          else if (RB == 8) reinterpret_cast<uint2 *>(buf)[o] = make_uint2(w[2 * r], w[2 * r + 1]);
          else s_bytes[o - j0] = (uint8_t)(w[r / 4] >> (8 * (r % 4)));
        }
      }
    }
  }
}

// Dynamic shared memory of k_gather_v: four u32 arrays of kGatherTile + 1
// entries, the scan partials, then (16-byte aligned) the tile's weight bytes;
// the WIDE form adds the high words of the sources' host positions.
constexpr size_t kGatherBytesOff = ((4 * (kGatherTile + 1) + kGatherThreads + 1) * 4 + 15) / 16 * 16;
constexpr size_t kGatherSmemBytes = kGatherBytesOff + kGatherTile;
constexpr size_t kGatherSmemBytesWide = kGatherSmemBytes + ((kGatherTile + 1) * 4 + 15) / 16 * 16;

template <int RB, bool WS, bool WIDE>
__global__ void __launch_bounds__(kGatherThreads) k_gather_v(
    const uint32_t *__restrict__ queue, const uint32_t *__restrict__ ptr,
    const uint32_t *__restrict__ off, const unsigned long long *__restrict__ obase, HostChunks host16,
    void *__restrict__ buf, HostChunks host_w16, uint8_t *__restrict__ wbuf,
    uint32_t from, uint32_t size, uint32_t edge_from, uint32_t edge_count) {
  extern __shared__ __align__(16) unsigned char g_gather_smem[];
  uint32_t *const s_bpos = reinterpret_cast<uint32_t *>(g_gather_smem);
  uint32_t *const s_hlo = s_bpos + (kGatherTile + 1);
  uint32_t *const s_len = s_hlo + (kGatherTile + 1);
  uint32_t *const s_cs = s_len + (kGatherTile + 1);
  uint32_t *const s_part = s_cs + (kGatherTile + 1);
  uint8_t *const s_bytes = g_gather_smem + kGatherBytesOff;
  uint32_t *const s_hhi = WIDE ? reinterpret_cast<uint32_t *>(g_gather_smem + kGatherSmemBytes) : nullptr;
  __shared__ uint32_t s_first, s_last;
  const uint32_t ntiles = (edge_count + kGatherTile - 1) / kGatherTile;
  const int tid = threadIdx.x;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint32_t j0 = t * kGatherTile;
    const uint32_t j1 = min(edge_count, j0 + kGatherTile);
    // sources covering [j0, j1): warp 0 finds the first, warp 1 the last
    if (tid < 64) {
      const int lane = tid & 31;
      const uint32_t r = warp_last_le(ptr, from, from + size, edge_from, tid < 32 ? j0 : j1 - 1, lane);
      if (lane == 0) (tid < 32 ? s_first : s_last) = r;
    }
    __syncthreads();
    const uint32_t first = s_first, nsrc = s_last - s_first + 1;
    // per-source clipped ranges (buffer position, host record, length)
#pragma unroll
    for (uint32_t q = 0; q < kGatherPer; ++q) {
      const uint32_t k = tid * kGatherPer + q;
      if (k < nsrc) {
        const uint32_t i = first + k;
        const uint32_t bp = ptr[i] - edge_from, be = ptr[i + 1] - edge_from;
        const uint32_t lo = max(bp, j0), hi = min(be, j1);
        s_bpos[k] = lo;
        if (WIDE) {
          const unsigned long long h = off_at(off, obase, queue[i]) + (lo - bp);
          s_hlo[k] = (uint32_t)h;
          s_hhi[k] = (uint32_t)(h >> 32);
        } else {
          s_hlo[k] = off[queue[i]] + (lo - bp);
        }
        s_len[k] = hi - lo;
      }
    }
    __syncthreads();
    uint32_t total = gather_scan<16 / RB>(nsrc, s_hlo, s_len, s_cs, s_part);
    gather_copy<RB, WIDE>(total, nsrc, j0, s_cs, s_hlo, s_hhi, s_len, s_bpos, host16, buf, s_bytes);
    if (WS) {
      __syncthreads();  // s_cs is reused
      total = gather_scan<16>(nsrc, s_hlo, s_len, s_cs, s_part);
      gather_copy<1, WIDE>(total, nsrc, j0, s_cs, s_hlo, s_hhi, s_len, s_bpos, host_w16, nullptr, s_bytes);
      __syncthreads();
      uint8_t *dst = wbuf + j0;
      const uint32_t len = j1 - j0;
      if (((uintptr_t)dst & 15u) == 0) {  // j0 is a multiple of the tile; wbuf is 16-byte aligned
        for (uint32_t i = tid; i < len / 16u; i += blockDim.x)
          reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(s_bytes)[i];
        for (uint32_t i = (len & ~15u) + tid; i < len; i += blockDim.x) dst[i] = s_bytes[i];
      } else {
        for (uint32_t i = tid; i < len; i += blockDim.x) dst[i] = s_bytes[i];
      }
    }
    __syncthreads();
  }
}

// ---- relaxation ----------------------------------------------------------------
// Per-algorithm semiring (shared/gpu_kernels.cu): candidate value from the
// source value and the edge, and whether it improves the destination.
template <int ALGO> struct Op;
template <> struct Op<SGW_BFS> {   // bfs_kernel: value+1, atomicMin (:45-46)
  static constexpr bool kMax = false;
  __device__ static uint32_t cand(uint32_t v, uint32_t) { return v + 1; }
};
template <> struct Op<SGW_SSSP> {  // sssp_kernel: value+w8, atomicMin (:146-149)
  static constexpr bool kMax = false;
  __device__ static uint32_t cand(uint32_t v, uint32_t w) { return v + w; }
};
template <> struct Op<SGW_SSWP> {  // sswp_kernel: min(value,w8), atomicMax (:196-199)
  static constexpr bool kMax = true;
  __device__ static uint32_t cand(uint32_t v, uint32_t w) { return min(v, w); }
};
template <> struct Op<SGW_CC> {    // cc_kernel: value, atomicMin (:96-98)
  static constexpr bool kMax = false;
  __device__ static uint32_t cand(uint32_t v, uint32_t) { return v; }
};

// Relaxes one edge given the destination's value as read beforehand: when
// the candidate beats it, a non-returning atomicMin/atomicMax (a reduction,
// no round trip for the thread) lowers the value and the destination's label
// is set.  The label is right even when another thread's candidate won: the
// read value is at most as good as the value when this kernel started (values
// move one way), so the candidate beat that value and the destination did
// improve in this kernel, by this thread or by the winner.  Returns whether
// the candidate beat the read value.
template <int ALGO>
__device__ __forceinline__ bool relax_edge_seen(uint32_t sval, uint32_t dst, uint32_t w, uint32_t cur,
                                                uint32_t *value, uint8_t *nxt) {
  const uint32_t c = Op<ALGO>::cand(sval, w);
  if (Op<ALGO>::kMax ? (c > cur) : (c < cur)) {
    if (Op<ALGO>::kMax) atomicMax(&value[dst], c);
    else atomicMin(&value[dst], c);
    nxt[dst] = 1;
    return true;
  }
  return false;
}

template <int ALGO>
__device__ __forceinline__ bool relax_edge(uint32_t sval, uint32_t dst, uint32_t w,
                                           uint32_t *value, uint8_t *nxt) {
  return relax_edge_seen<ALGO>(sval, dst, w, value[dst], value, nxt);
}

// Whether a source with this value may push (guards u32 overflow of INF+w;
// the reference relies on INF vertices never carrying a label).
template <int ALGO>
__device__ __forceinline__ bool can_push(uint32_t v) {
  if (ALGO == SGW_BFS || ALGO == SGW_SSSP) return v != kInf;
  if (ALGO == SGW_SSWP) return v != 0;
  return true;
}

// Reads edge record e of a device edge buffer: W = 2 words {end, w8};
// W = 1 either {end} (pbits = 0; its weight, if any, in the byte stream wbuf
// of the split form) or the packed transfer form (w8 << pbits) | end.
template <int W>
__device__ __forceinline__ void load_edge(const uint32_t *buf, uint32_t e, uint32_t pbits,
                                          uint32_t &dst, uint32_t &w, const uint8_t *wbuf = nullptr) {
  if (W == 1) {
    const uint32_t r = buf[e];
    if (pbits) { dst = r & ((1u << pbits) - 1u); w = r >> pbits; }
    else { dst = r; w = wbuf ? (uint32_t)wbuf[e] : 0u; }
  } else {
    const uint2 ed = reinterpret_cast<const uint2 *>(buf)[e];
    dst = ed.x;
    w = ed.y;
  }
}

// Reads edge record e of the host transfer copy (or of the graph's records
// where they are read in place): the same forms, streams of chunks.
struct HostEdges {
  HostChunks ends, w;        // edge words, weight bytes (split form)
  uint32_t split;            // this run reads the weight bytes
};
template <int W>
__device__ __forceinline__ void load_edge_host(const HostEdges &h, uint32_t e, uint32_t pbits, uint32_t &dst,
                                               uint32_t &w) {
  if (W == 1) {
    const uint32_t r = *reinterpret_cast<const uint32_t *>(hc_at(h.ends, (size_t)e * 4));
    if (pbits) { dst = r & ((1u << pbits) - 1u); w = r >> pbits; }
    else { dst = r; w = h.split ? (uint32_t)*reinterpret_cast<const uint8_t *>(hc_at(h.w, e)) : 0u; }
  } else {
    const uint2 ed = *reinterpret_cast<const uint2 *>(hc_at(h.ends, (size_t)e * 8));
    dst = ed.x;
    w = ed.y;
  }
}

// Edge cache of a sync run: the edge buffers, which passes that read the host
// copy leave unused, hold the first `edges` records of the graph at their own
// positions.  A row that lies among them is stored as its first pass reads it
// and read from there afterwards; `have` says which rows those are.  Sync runs
// are bound by the host link: PageRank-sync on an Erdos-Renyi graph of 16 M
// edges in memory 15.2 -> 8.4 ms, on R-MAT 2^20 with half the edges' room 14.1 ->
// 11.7 ms, CC-sync on 32 M arcs (half) 1.66 -> 1.45 ms, SSSP-sync on 2^25
// vertices (half) 18.0 -> 14.3 ms.
struct EdgeCache {
  uint32_t *buf;
  uint8_t *wbuf;             // split form: the weight bytes
  uint32_t *have;            // per 16 vertices: rows held | rows stored since the last generate << 16
  uint32_t edges;
};
// Where a first pass finds a partition's records.
constexpr int kSrcBuffer = 0;  // gathered (or streamed) into an edge buffer
constexpr int kSrcHost = 1;    // in the host copy
constexpr int kSrcCache = 2;   // in the edge cache or the host copy

enum : uint32_t { kRowHost = 0, kRowStore = 1, kRowHeld = 2 };
__device__ __forceinline__ uint32_t cache_row(const EdgeCache &c, uint32_t u, uint32_t off, uint32_t deg) {
  if ((unsigned long long)off + deg > c.edges) return kRowHost;
  return (c.have[u >> 4] >> (u & 15u)) & 1u ? kRowHeld : kRowStore;
}
// The row's first pass (one lane of it): held from the next generate on.
__device__ __forceinline__ void cache_stored(const EdgeCache &c, uint32_t u) {
  atomicOr(&c.have[u >> 4], 0x10000u << (u & 15u));
}

template <int W>
__device__ __forceinline__ void load_edge_cached(const HostEdges &h, const EdgeCache &c, uint32_t how, uint32_t e,
                                                 uint32_t pbits, uint32_t &dst, uint32_t &w) {
  if (W == 1) {
    uint32_t r, x = 0;
    if (how == kRowHeld) {
      r = c.buf[e];
      if (h.split) x = c.wbuf[e];
    } else {
      r = *reinterpret_cast<const uint32_t *>(hc_at(h.ends, (size_t)e * 4));
      if (h.split) x = *reinterpret_cast<const uint8_t *>(hc_at(h.w, e));
      if (how == kRowStore) {
        c.buf[e] = r;
        if (h.split) c.wbuf[e] = (uint8_t)x;
      }
    }
    if (pbits) { dst = r & ((1u << pbits) - 1u); w = r >> pbits; }
    else { dst = r; w = x; }
  } else {
    uint2 ed;
    if (how == kRowHeld) ed = reinterpret_cast<const uint2 *>(c.buf)[e];
    else {
      ed = *reinterpret_cast<const uint2 *>(hc_at(h.ends, (size_t)e * 8));
      if (how == kRowStore) reinterpret_cast<uint2 *>(c.buf)[e] = ed;
    }
    dst = ed.x;
    w = ed.y;
  }
}

// What an edge needs of its source in a first pass: its value and, with the
// cache, where its row is.
template <class T>
struct CachedRow { T val; uint32_t how; };
template <class T, int SRC> struct RowOf { using V = T; };
template <class T> struct RowOf<T, kSrcCache> { using V = CachedRow<T>; };

struct RelaxArgs {
  const uint32_t *queue;
  const uint32_t *ptr;
  const uint32_t *buf;       // device edge buffer (W words per edge)
  uint32_t *value;
  uint8_t *cur;              // async: label of this inner iteration (cleared)
  uint8_t *nxt;              // label set on improvement
  Ctl *ctl;
  WorkItem *wl;
  uint32_t wl_cap;
  uint32_t from, size, edge_from;
  uint32_t iter;             // inner iteration of the partition (1-based)
  uint32_t base;             // inner iterations launched before this partition's
  unsigned long long *poll;  // host word that async iterations > 1 report to (null: none)
  uint32_t poll_tag;
  uint32_t tile_degree_max;  // sources above this go to the chunk list
  uint32_t chunk_edges;
  uint32_t pbits;            // packed records: bits of the destination
  // streamed partition: the buffer holds a whole vertex range starting at
  // edge stream_base, so a source's edges sit at off[u] - stream_base
  uint32_t streamed;
  uint32_t stream_base;
  const uint32_t *off;
  const uint8_t *wbuf;       // split form: the buffer's weight bytes (else null)
  HostEdges host;            // first passes that read the host copy themselves
  EdgeCache cache;
};

constexpr int kRelaxThreads = 256;

// Tells the host that inner iteration `iter` has begun (the one before it is
// complete) and whether it has nothing to do: one 64-bit word of mapped host
// memory that the host polls instead of waiting for a copy of the control block.
__device__ __forceinline__ void poll_report(unsigned long long *poll, uint32_t tag, uint32_t iter, int skip) {
  if (poll && iter > 1) {
    const unsigned long long x = (unsigned long long)tag << 48 | (unsigned long long)iter << 1 | (unsigned)skip;
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(poll), "l"(x) : "memory");
  }
}
// The same for the iteration after a capped partition's last.
__global__ void k_poll_end(unsigned long long *poll, uint32_t tag, uint32_t iter) {
  chain_wait();
  chain_open();
  poll_report(poll, tag, iter, 1);
}

// Tile of kRelaxThreads partition sources per CTA (grid-stride).  Each thread
// claims one source (async: only if its label is set, clearing it), the CTA
// scans the degrees in shared memory and all threads expand the tile's edges
// together: edge j of the tile belongs to the source found by binary search
// in the scanned degrees.  Sources above tile_degree_max are cut into chunks
// and appended to the chunk list instead.
struct TileSmem {
  uint32_t scan[kRelaxThreads + 1];
  uint32_t boff[kRelaxThreads];
  uint32_t val[kRelaxThreads];
  uint32_t hub[kRelaxThreads];
  uint32_t wsum[kRelaxThreads / 32];
  uint32_t nhub, wbase;
  int skip;
};

template <int ALGO, bool ASYNC, int W>
__device__ __forceinline__ void relax_tile_phase(const RelaxArgs &a, TileSmem &sm) {
  uint32_t *const s_scan = sm.scan;
  uint32_t *const s_boff = sm.boff;
  uint32_t *const s_val = sm.val;
  uint32_t *const s_hub = sm.hub;
  uint32_t &s_nhub = sm.nhub;
  uint32_t &s_wbase = sm.wbase;
  int &s_skip = sm.skip;
  const int tid = threadIdx.x;
  const uint32_t slot = (a.base + a.iter) & 3u;
  if (tid == 0) {
    int skip = 0;
    if (ASYNC && a.iter > 1 && ld_acquire_u32(&a.ctl->upd[(a.base + a.iter - 1) & 3u]) == 0) skip = 1;
    s_skip = skip;
    if (blockIdx.x == 0) {
      a.ctl->upd[(a.base + a.iter + 1) & 3u] = 0;
      a.ctl->wl_count[(a.base + a.iter + 1) & 3u] = 0;
      if (!skip) atomicAdd(&a.ctl->iters_total, 1u);
      if (ASYNC) poll_report(a.poll, a.poll_tag, a.iter, skip);
    }
  }
  __syncthreads();
  if (s_skip) return;
  bool any_update = false;
  const uint32_t ntiles = (a.size + kRelaxThreads - 1) / kRelaxThreads;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    if (tid == 0) s_nhub = 0;
    __syncthreads();
    const uint32_t idx = t * kRelaxThreads + tid;
    uint32_t d = 0, boff = 0, val = 0, u = 0;
    if (idx < a.size) {
      const uint32_t i = a.from + idx;
      u = a.queue[i];
      bool act = true;
      if (ASYNC) {
        act = a.cur[u] != 0;
        if (act) a.cur[u] = 0;
      }
      if (act) {
        val = a.value[u];
        if (can_push<ALGO>(val)) {
          const uint32_t p0 = a.ptr[i];
          d = a.ptr[i + 1] - p0;
          boff = a.streamed ? a.off[u] - a.stream_base : p0 - a.edge_from;
          if (d > a.tile_degree_max) {
            s_hub[atomicAdd(&s_nhub, 1u)] = tid;
            atomicAdd(&a.ctl->relaxed_edges, (unsigned long long)d);
          }
        }
      }
    }
    s_boff[tid] = boff;
    s_val[tid] = val;
    {
      const int nsrc = __syncthreads_count(d > 0);
      if (tid == 0 && nsrc) atomicAdd(&a.ctl->relaxed_sources, (unsigned long long)nsrc);
    }
    // chunk out high-degree sources (whole CTA writes the items)
    const uint32_t nhub = s_nhub;
    for (uint32_t h = 0; h < nhub; ++h) {
      const uint32_t ht = s_hub[h];
      if (tid == ht) {
        const uint32_t nch = (d + a.chunk_edges - 1) / a.chunk_edges;
        s_wbase = atomicAdd(&a.ctl->wl_count[slot], nch);
        s_scan[kRelaxThreads] = d;  // temporary: degree of this hub
      }
      __syncthreads();
      const uint32_t hd = s_scan[kRelaxThreads];
      const uint32_t nch = (hd + a.chunk_edges - 1) / a.chunk_edges;
      const uint32_t wb = s_wbase;
      for (uint32_t c = tid; c < nch; c += blockDim.x) {
        if (wb + c < a.wl_cap) {
          WorkItem it;
          it.boff = s_boff[ht] + c * a.chunk_edges;
          it.count = min(a.chunk_edges, hd - c * a.chunk_edges);
          it.value = s_val[ht];
          it.vertex = 0;
          a.wl[wb + c] = it;
        } else {
          atomicExch(&a.ctl->error, 3u);
        }
      }
      __syncthreads();
    }
    if (d > a.tile_degree_max) d = 0;
    // block exclusive scan of d
    {
      const int lane = tid & 31, warp = tid >> 5;
      const uint32_t incl = warp_incl_scan(d, lane);
      uint32_t *const s_wsum = sm.wsum;
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      if (tid == 0) {
        uint32_t acc = 0;
        for (int w = 0; w < kRelaxThreads / 32; ++w) { uint32_t x = s_wsum[w]; s_wsum[w] = acc; acc += x; }
        s_scan[kRelaxThreads] = acc;
      }
      __syncthreads();
      s_scan[tid] = s_wsum[warp] + incl - d;
      __syncthreads();
    }
    const uint32_t total = s_scan[kRelaxThreads];
    if (tid == 0 && total) atomicAdd(&a.ctl->relaxed_edges, (unsigned long long)total);
    for (uint32_t j0 = tid; j0 < total; j0 += kRelaxUnroll * kRelaxThreads) {
      uint32_t dst[kRelaxUnroll], w[kRelaxUnroll], sv[kRelaxUnroll], cur[kRelaxUnroll];
      bool ok[kRelaxUnroll];
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q) {
        const uint32_t j = j0 + q * kRelaxThreads;
        ok[q] = j < total;
        if (ok[q]) {
          // last source k with s_scan[k] <= j (sources with d == 0 share
          // offsets; the last one with that offset is the one that owns edge j)
          uint32_t lo = 0, hi = kRelaxThreads;
          while (lo < hi) {
            uint32_t mid = (lo + hi) >> 1;
            if (s_scan[mid] <= j) lo = mid + 1; else hi = mid;
          }
          const uint32_t k = lo - 1;
          load_edge<W>(a.buf, s_boff[k] + (j - s_scan[k]), a.pbits, dst[q], w[q], a.wbuf);
          sv[q] = s_val[k];
        }
      }
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q)
        if (ok[q]) cur[q] = a.value[dst[q]];
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q)
        if (ok[q]) any_update |= relax_edge_seen<ALGO>(sv[q], dst[q], w[q], cur[q], a.value, a.nxt);
    }
    __syncthreads();
  }
  if (__syncthreads_or(any_update) && tid == 0) atomicAdd(&a.ctl->upd[slot], 1u);
}

template <int ALGO, bool ASYNC, int W>
__global__ void __launch_bounds__(kRelaxThreads) k_relax_tile(RelaxArgs a) {
  __shared__ TileSmem sm;
  relax_tile_phase<ALGO, ASYNC, W>(a, sm);
}

// Relaxes the kRelaxUnroll edges of a lane: all record loads, then all
// destination values, then the compares and reductions.
template <int ALGO, int W, int SRC = kSrcBuffer>
__device__ __forceinline__ bool relax_lane(const RelaxArgs &a, const uint32_t (&pos)[kRelaxUnroll],
                                           const uint32_t (&sv)[kRelaxUnroll], const bool (&ok)[kRelaxUnroll]) {
  uint32_t dst[kRelaxUnroll], w[kRelaxUnroll], cur[kRelaxUnroll];
  bool any = false;
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) {
      if (SRC == kSrcHost) load_edge_host<W>(a.host, pos[q], a.pbits, dst[q], w[q]);
      else load_edge<W>(a.buf, pos[q], a.pbits, dst[q], w[q], a.wbuf);
    }
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) cur[q] = a.value[dst[q]];
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) any |= relax_edge_seen<ALGO>(sv[q], dst[q], w[q], cur[q], a.value, a.nxt);
  return any;
}

// The same with the edge cache.
template <int ALGO, int W, int SRC>
__device__ __forceinline__ bool relax_lane(const RelaxArgs &a, const uint32_t (&pos)[kRelaxUnroll],
                                           const CachedRow<uint32_t> (&sv)[kRelaxUnroll],
                                           const bool (&ok)[kRelaxUnroll]) {
  uint32_t dst[kRelaxUnroll], w[kRelaxUnroll], cur[kRelaxUnroll];
  bool go[kRelaxUnroll];
  bool any = false;
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) load_edge_cached<W>(a.host, a.cache, sv[q].how, pos[q], a.pbits, dst[q], w[q]);
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q) {
    go[q] = ok[q] && can_push<ALGO>(sv[q].val);  // a row is stored whole whether or not it pushes
    if (go[q]) cur[q] = a.value[dst[q]];
  }
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (go[q]) any |= relax_edge_seen<ALGO>(sv[q].val, dst[q], w[q], cur[q], a.value, a.nxt);
  return any;
}

// Warp-tile form of k_relax_tile for async inner iterations (sync passes take
// k_relax_all): each warp takes 32 partition sources at a
// time and expands their edges on its own (warp_expand), so
// warps never wait on each other: a warp that runs out of tiles adds its counters
// to the CTA's in shared memory and leaves, and the last warp of the CTA to
// leave publishes them.  Sources above tile_degree_max go to the chunk list
// as in the CTA form.
constexpr int kWarpsPerCta = kRelaxThreads / 32;
// Resident CTAs per SM the warp relaxation is compiled for (registers are
// capped to fit them); 4 keeps it free of spills.
#ifndef SGW_RELAX_MIN_BLOCKS
#define SGW_RELAX_MIN_BLOCKS 4
#endif

// Counters of a CTA whose warps finish independently.
struct CtaTally {
  unsigned long long edges, srcs, host;
  uint32_t any, done;
  int skip;
};

// Start of inner iteration a.iter: whether it runs at all, the next
// iteration's counters cleared, the run counted.
template <bool ASYNC, class Args>
__device__ __forceinline__ bool iter_begin(const Args &a, CtaTally &t) {
  if (threadIdx.x == 0) {
    int skip = 0;
    if (ASYNC && a.iter > 1 && ld_acquire_u32(&a.ctl->upd[(a.base + a.iter - 1) & 3u]) == 0) skip = 1;
    t.skip = skip;
    t.edges = 0;
    t.srcs = 0;
    t.host = 0;
    t.any = 0;
    t.done = 0;
    if (blockIdx.x == 0) {
      a.ctl->upd[(a.base + a.iter + 1) & 3u] = 0;
      a.ctl->wl_count[(a.base + a.iter + 1) & 3u] = 0;
      if (!skip) atomicAdd(&a.ctl->iters_total, 1u);
      if (ASYNC) poll_report(a.poll, a.poll_tag, a.iter, skip);
    }
  }
  __syncthreads();
  return !t.skip;
}

// End of a warp's share; the CTA's last warp publishes.
__device__ __forceinline__ void warp_publish(CtaTally &t, Ctl *ctl, uint32_t slot, int lane, bool any,
                                             unsigned long long edges, unsigned long long srcs,
                                             unsigned long long host = 0) {
  const bool warp_any = __any_sync(0xffffffffu, any);
  if (lane == 0) {
    if (edges) atomicAdd(&t.edges, edges);
    if (srcs) atomicAdd(&t.srcs, srcs);
    if (host) atomicAdd(&t.host, host);
    if (warp_any) atomicOr(&t.any, 1u);
    __threadfence_block();
    if (atomicAdd(&t.done, 1u) == kWarpsPerCta - 1) {
      __threadfence_block();
      if (t.any) atomicAdd(&ctl->upd[slot], 1u);
      if (t.edges) atomicAdd(&ctl->relaxed_edges, t.edges);
      if (t.srcs) atomicAdd(&ctl->relaxed_sources, t.srcs);
      if (t.host) atomicAdd(&ctl->host_edges, t.host);
    }
  }
}

template <int ALGO, int W>
__global__ void __launch_bounds__(kRelaxThreads, SGW_RELAX_MIN_BLOCKS) k_relax_warp(RelaxArgs a) {
  chain_wait();
  __shared__ CtaTally s_tally;
  __shared__ WarpExpand<uint32_t> s_exp[kWarpsPerCta];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t slot = (a.base + a.iter) & 3u;
  if (!iter_begin<true>(a, s_tally)) return;
  bool any_update = false;
  unsigned long long my_edges = 0, my_srcs = 0;
  const uint32_t ntiles = (a.size + 31u) / 32u;
  const uint32_t gw = blockIdx.x * kWarpsPerCta + wid, nw = gridDim.x * kWarpsPerCta;
  for (uint32_t t = gw; t < ntiles; t += nw) {
    const uint32_t idx = t * 32u + lane;
    uint32_t d = 0, boff = 0, val = 0;
    if (idx < a.size) {
      const uint32_t i = a.from + idx;
      const uint32_t u = a.queue[i];
      if (a.cur[u]) {
        a.cur[u] = 0;
        val = a.value[u];
        if (can_push<ALGO>(val)) {
          const uint32_t p0 = a.ptr[i];
          d = a.ptr[i + 1] - p0;
          boff = a.streamed ? a.off[u] - a.stream_base : p0 - a.edge_from;
        }
      }
    }
    my_srcs += __popc(__ballot_sync(0xffffffffu, d > 0));
    // high-degree sources: the warp writes their chunk items together
    unsigned hubs = __ballot_sync(0xffffffffu, d > a.tile_degree_max);
    while (hubs) {
      const int h = __ffs(hubs) - 1;
      hubs &= hubs - 1;
      const uint32_t hd = __shfl_sync(0xffffffffu, d, h);
      const uint32_t hb = __shfl_sync(0xffffffffu, boff, h);
      const uint32_t hv = __shfl_sync(0xffffffffu, val, h);
      const uint32_t nch = (hd + a.chunk_edges - 1) / a.chunk_edges;
      uint32_t wb = 0;
      if (lane == 0) wb = atomicAdd(&a.ctl->wl_count[slot], nch);
      wb = __shfl_sync(0xffffffffu, wb, 0);
      for (uint32_t c = lane; c < nch; c += 32) {
        if (wb + c < a.wl_cap) {
          WorkItem it;
          it.boff = hb + c * a.chunk_edges;
          it.count = min(a.chunk_edges, hd - c * a.chunk_edges);
          it.value = hv;
          it.vertex = 0;
          a.wl[wb + c] = it;
        } else {
          atomicExch(&a.ctl->error, 3u);
        }
      }
      my_edges += hd;
    }
    if (d > a.tile_degree_max) d = 0;
    my_edges += warp_expand(s_exp[wid], lane, d, boff, val,
                            [&](const uint32_t (&pos)[kRelaxUnroll], const uint32_t (&sv)[kRelaxUnroll],
                                const bool (&ok)[kRelaxUnroll]) { any_update |= relax_lane<ALGO, W>(a, pos, sv, ok); });
  }
  warp_publish(s_tally, a.ctl, slot, lane, any_update, my_edges, my_srcs);
}

// First pass over a queue whose every source is active (every sync pass; an
// async partition's first inner iteration, whose labels the generate step or
// k_claim has taken).  The work is cut by edges, not by sources: source i of
// the partition stands for kRelaxHeader + degree units, each warp takes an
// equal run of units, finds its first source with a 32-way search and clips
// the rows at both ends, so hubs are shared by many warps (no chunk list and
// no second launch) and a partition of few, long rows still fills the chip.
// kRelaxHeader is about what a source costs beside its edges: it keeps a warp
// that holds thousands of one-edge rows from being the last.  Against source
// tiles plus a chunk list, relaxation per run: BFS-sync on R-MAT 2^16 0.145
// and 0.058 ms, CC-sync on 32 M symmetric arcs 1.10 and 0.78 ms, SSSP-async on
// an Erdos-Renyi graph of 36 M edges 10.6 and 8.0 ms (there mostly the chunk
// launches, which queues without a long row no longer make).
constexpr uint32_t kRelaxHeader = 8;
constexpr uint32_t kRelaxMinUnits = 256;  // per warp: about one tile

// Last source i in [0, size) that starts at or before unit t; every lane
// returns it.  Source i starts at unit ptr[from + i] - edge_from + H * i.
template <uint32_t H>
__device__ __forceinline__ uint32_t warp_find_unit(const uint32_t *ptr, uint32_t from, uint32_t size,
                                                   uint32_t edge_from, unsigned long long t, int lane) {
  uint32_t lo = 0, hi = size;
  auto le = [&](uint32_t i) {
    return i < hi && (unsigned long long)(ptr[from + i] - edge_from) + (unsigned long long)H * i <= t;
  };
  while (hi - lo > 32u) {
    const uint32_t step = (hi - lo + 31u) / 32u;
    const uint32_t m = __ballot_sync(0xffffffffu, le(lo + (uint32_t)lane * step));  // a prefix of lanes; lane 0 always
    lo += (31u - (uint32_t)__clz((int)m)) * step;
    hi = min(hi, lo + step);
  }
  const uint32_t m = __ballot_sync(0xffffffffu, le(lo + (uint32_t)lane));
  return lo + 31u - (uint32_t)__clz((int)m);
}

// The part of source idx's row that units [t0, t1) hold: first edge *lo and
// count (0: none); *head: whether the source's first unit is among them.
template <uint32_t H>
__device__ __forceinline__ uint32_t unit_clip(unsigned long long start, uint32_t deg, unsigned long long t0,
                                              unsigned long long t1, uint32_t *lo, bool *head) {
  *head = start >= t0 && start < t1;
  const unsigned long long e0 = start + H;  // the row's edges are units [e0, e0 + deg)
  const unsigned long long a = t0 > e0 ? t0 - e0 : 0, b = t1 > e0 ? t1 - e0 : 0;
  const unsigned long long hi = b < deg ? b : deg;
  *lo = (uint32_t)a;
  return a < hi ? (uint32_t)(hi - a) : 0u;
}

// With kSrcHost the records are read over the host link by the pass itself (a
// partition that is relaxed once: every sync pass), at edge off[u] + j of the
// host copy, so nothing is written to an edge buffer and read back, and the
// relaxation hides behind the link.  Bound by the link (211 GB/s by DMA):
// CC-sync over 32 M arcs out of memory reads at 193 GB/s (gather and relaxation
// before: 1.45 + 0.78 ms partly overlapped, now 1.43), PageRank-sync's query on
// R-MAT 2^20 went from 21.1 to 16.1 ms.  The windows of a tile start on
// multiples of 32 edges there (warp_expand's align): without it each one
// touches two 128-byte lines and CC's passes take 1.65 ms.  kSrcCache: see
// EdgeCache.
template <int ALGO, int W, int SRC>
__global__ void __launch_bounds__(kRelaxThreads, SGW_RELAX_MIN_BLOCKS) k_relax_all(RelaxArgs a,
                                                                                  unsigned long long units,
                                                                                  unsigned long long per_warp) {
  chain_wait();
  __shared__ CtaTally s_tally;
  constexpr bool kHost = SRC != kSrcBuffer, kCache = SRC == kSrcCache;
  using V = typename RowOf<uint32_t, SRC>::V;
  __shared__ WarpExpand<V> s_exp[kWarpsPerCta];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  iter_begin<false>(a, s_tally);
  bool any_update = false;
  unsigned long long my_edges = 0, my_srcs = 0, my_host = 0;
  const unsigned long long t0 = per_warp * (blockIdx.x * kWarpsPerCta + wid);
  const unsigned long long t1 = min(units, t0 + per_warp);
  if (t0 < t1) {
    const uint32_t first = warp_find_unit<kRelaxHeader>(a.ptr, a.from, a.size, a.edge_from, t0, lane);
    for (uint32_t i0 = first; i0 < a.size; i0 += 32) {
      const uint32_t idx = i0 + lane;
      uint32_t d = 0, boff = 0, val = 0, how = kRowHost;
      bool past = true, head = false;
      if (idx < a.size) {
        const uint32_t p0 = a.ptr[a.from + idx], p1 = a.ptr[a.from + idx + 1];
        const uint32_t u = a.queue[a.from + idx];
        const unsigned long long start = (unsigned long long)(p0 - a.edge_from) + (unsigned long long)kRelaxHeader * idx;
        past = start >= t1;
        uint32_t lo;
        d = unit_clip<kRelaxHeader>(start, p1 - p0, t0, t1, &lo, &head);
        if (d || head) {
          val = a.value[u];
          boff = (kHost ? a.off[u] : a.streamed ? a.off[u] - a.stream_base : p0 - a.edge_from) + lo;
          if (kCache) {
            how = cache_row(a.cache, u, boff - lo, p1 - p0);
            if (head && how == kRowStore) cache_stored(a.cache, u);
          }
          if (!can_push<ALGO>(val)) {
            head = false;
            if (!kCache) d = 0;
          }
        }
      }
      my_srcs += __popc(__ballot_sync(0xffffffffu, head));
      V row;
      if constexpr (kCache) {
        row.val = val;
        row.how = how;
        my_host += __reduce_add_sync(0xffffffffu, how != kRowHeld ? d : 0u);
      } else {
        row = val;
      }
      my_edges += warp_expand(s_exp[wid], lane, d, boff, row,
                              [&](const uint32_t (&pos)[kRelaxUnroll], const V (&sv)[kRelaxUnroll],
                                  const bool (&ok)[kRelaxUnroll]) { any_update |= relax_lane<ALGO, W, SRC>(a, pos, sv, ok); },
                              kHost);
      if (__any_sync(0xffffffffu, past)) break;
    }
  }
  warp_publish(s_tally, a.ctl, (a.base + a.iter) & 3u, lane, any_update, my_edges, my_srcs, my_host);
}

// Chunk list of inner iteration `iter`: one warp per item.
template <int ALGO, bool ASYNC, int W>
__device__ __forceinline__ void relax_chunks_phase(const RelaxArgs &a) {
  const uint32_t slot = (a.base + a.iter) & 3u;
  if (ASYNC && a.iter > 1 && ld_acquire_u32(&a.ctl->upd[(a.base + a.iter - 1) & 3u]) == 0) return;
  const uint32_t items = min(ld_acquire_u32(&a.ctl->wl_count[slot]), a.wl_cap);
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  bool any_update = false;
  for (uint32_t it = gw; it < items; it += nw) {
    const WorkItem wi = a.wl[it];
    for (uint32_t j0 = lane; j0 < wi.count; j0 += 32 * kRelaxUnroll) {
      uint32_t dst[kRelaxUnroll], w[kRelaxUnroll], cur[kRelaxUnroll];
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q)
        if (j0 + 32 * q < wi.count) load_edge<W>(a.buf, wi.boff + j0 + 32 * q, a.pbits, dst[q], w[q], a.wbuf);
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q)
        if (j0 + 32 * q < wi.count) cur[q] = a.value[dst[q]];
#pragma unroll
      for (int q = 0; q < kRelaxUnroll; ++q)
        if (j0 + 32 * q < wi.count)
          any_update |= relax_edge_seen<ALGO>(wi.value, dst[q], w[q], cur[q], a.value, a.nxt);
    }
  }
  if (__syncthreads_or(any_update) && threadIdx.x == 0) atomicAdd(&a.ctl->upd[slot], 1u);
}

template <int ALGO, bool ASYNC, int W>
__global__ void __launch_bounds__(kRelaxThreads) k_relax_chunks(RelaxArgs a) {
  chain_wait();
  relax_chunks_phase<ALGO, ASYNC, W>(a);
}

// Single-vertex partition (degree above the edge buffer): claim the source
// once, then relax its edges piece by piece.  how: 0 the source is active and
// its labels are as they should be (sync), 1 active if labelled, labels
// cleared, 2 active, labels cleared.
__global__ void k_hub_claim(uint32_t u, const uint32_t *value, uint8_t *l1, uint8_t *l2, Ctl *ctl, int how) {
  uint32_t act = 1;
  if (how == 1) act = (l1[u] | l2[u]) != 0;
  if (how) {
    l1[u] = 0;
    l2[u] = 0;
  }
  ctl->hub_active = act;
  ctl->hub_value = value[u];
}

template <int ALGO, int W>
__global__ void k_relax_flat(const uint32_t *buf, const uint8_t *wbuf, uint32_t count, uint32_t pbits,
                             uint32_t *value, uint8_t *nxt, Ctl *ctl) {
  if (!ctl->hub_active) return;
  const uint32_t sval = ctl->hub_value;
  if (!can_push<ALGO>(sval)) return;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
    uint32_t dst, w;
    load_edge<W>(buf, j, pbits, dst, w, wbuf);
    relax_edge<ALGO>(sval, dst, w, value, nxt);
  }
}

// ---- label hand-off (shared/gpu_kernels.cu:515-534) ------------------------
// mixLabels: label1 |= label2; label2 = 0 for the partition's sources.
__global__ void k_mix(const uint32_t *queue, uint32_t from, uint32_t size, uint8_t *l1, uint8_t *l2) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
    const uint32_t u = queue[from + i];
    if (l2[u]) { l1[u] = 1; l2[u] = 0; }
  }
}

// Every source of the partition is relaxed by its first pass: its labels are
// taken now, so that what is set from here on marks improvements.
__global__ void k_claim(const uint32_t *queue, uint32_t from, uint32_t size, uint8_t *l1, uint8_t *l2) {
  chain_wait();
  chain_open();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < size; i += gridDim.x * blockDim.x) {
    const uint32_t u = queue[from + i];
    l1[u] = 0;
    l2[u] = 0;
  }
}

// ---- state init and summaries ------------------------------------------------
// Initial values and labels of subway/<algo>-<mode>.cu.
__global__ void k_init(uint32_t n, int algo, int mode, uint32_t source, uint32_t *value,
                       uint8_t *l1, uint8_t *l2) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    uint32_t val;
    switch (algo) {
      case SGW_BFS:
      case SGW_SSSP: val = (v == source) ? 0u : kInf; break;
      case SGW_SSWP: val = (v == source) ? kInf : 0u; break;
      default: val = v; break;  // CC
    }
    value[v] = val;
    uint8_t a1, a2;
    if (mode == SGW_ASYNC) { a1 = 1; a2 = 0; }            // all active for the first generate
    else if (algo == SGW_CC) { a1 = 0; a2 = 1; }           // cc-sync.cu:31-33
    else { a1 = 0; a2 = (v == source) ? 1 : 0; }           // bfs-sync.cu:30-36
    l1[v] = a1;
    l2[v] = a2;
  }
}

// After the first async generate, label1 = {source} (subway/sssp-async.cu:59-63);
// cc-async keeps every vertex active.
__global__ void k_async_reset(uint32_t n, uint32_t source, uint8_t *l1) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    l1[v] = (v == source) ? 1 : 0;
}

// Graph500 m_reached: edges whose source left its initial value.
__global__ void k_reached(uint32_t n, int algo, uint32_t source, const uint32_t *value,
                          const uint32_t *off, Ctl *ctl) {
  unsigned long long acc = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t x = value[v];
    bool reached;
    switch (algo) {
      case SGW_BFS:
      case SGW_SSSP: reached = x != kInf; break;
      case SGW_SSWP: reached = x != 0 || v == source; break;
      default: reached = true; break;
    }
    if (reached) acc += off[v + 1] - off[v];
  }
  acc = __reduce_add_sync(0xffffffffu, (uint32_t)acc) ; // per-warp (degree sums fit u32 per warp)
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(&ctl->reached_edges, acc);
}

// ---- PageRank (pr_kernel / pr_async, shared/gpu_kernels.cu:211-254, :459-502) --
// Ranks and residuals are kept in double precision on the device; the
// reference's float results are the final cast.
struct PrArgs {
  const uint32_t *queue;
  const uint32_t *ptr;
  const uint32_t *buf;       // device edge buffer (W words per edge)
  double *pval;
  double *delta;
  double *qpush;             // push of each queued source (0: none this iteration)
  Ctl *ctl;
  uint32_t from, size, edge_from;
  uint32_t iter, base;
  unsigned long long *poll;
  uint32_t poll_tag;
  uint32_t pbits;
  uint32_t streamed;
  uint32_t stream_base;
  const uint32_t *off;
  double acc;
  double damping;
  HostEdges host;
  EdgeCache cache;
};

__device__ __forceinline__ double ld_relaxed_f64(const double *p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

// Adds each edge's push to its destination's residual: the records of
// kRelaxUnroll edges of a lane are loaded before their (non-returning) adds.
template <int W, int SRC>
__device__ __forceinline__ void pr_lane(const PrArgs &a, const uint32_t (&pos)[kRelaxUnroll],
                                        const double (&push)[kRelaxUnroll], const bool (&ok)[kRelaxUnroll]) {
  uint32_t dst[kRelaxUnroll], w;
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) {
      if (SRC == kSrcHost) load_edge_host<W>(a.host, pos[q], a.pbits, dst[q], w);
      else load_edge<W>(a.buf, pos[q], a.pbits, dst[q], w);
    }
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) atomicAdd(&a.delta[dst[q]], push[q]);
}
template <int W, int SRC>
__device__ __forceinline__ void pr_lane(const PrArgs &a, const uint32_t (&pos)[kRelaxUnroll],
                                        const CachedRow<double> (&row)[kRelaxUnroll],
                                        const bool (&ok)[kRelaxUnroll]) {
  uint32_t dst[kRelaxUnroll], w;
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) load_edge_cached<W>(a.host, a.cache, row[q].how, pos[q], a.pbits, dst[q], w);
#pragma unroll
  for (int q = 0; q < kRelaxUnroll; ++q)
    if (ok[q]) atomicAdd(&a.delta[dst[q]], row[q].val);
}

// Pushes of one inner iteration, the work cut by edges as in k_relax_all:
// source i pushes qpush[i], which the generate step (first iteration, every
// queued source) or k_pr_claim (later async ones; 0 for the sources that are
// not active again) has written.  PageRank's later rounds queue a few tens of
// thousands of long rows, which left most of the chip idle when each CTA took
// 256 of them and found its edges' owners by binary search.
template <int W, int SRC>
__global__ void __launch_bounds__(kRelaxThreads, SGW_RELAX_MIN_BLOCKS) k_pr_all(PrArgs a, unsigned long long units,
                                                                               unsigned long long per_warp) {
  chain_wait();
  __shared__ CtaTally s_tally;
  constexpr bool kHost = SRC != kSrcBuffer, kCache = SRC == kSrcCache;
  using V = typename RowOf<double, SRC>::V;
  __shared__ WarpExpand<V> s_exp[kWarpsPerCta];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint32_t slot = (a.base + a.iter) & 3u;
  if (a.iter > 1) {  // k_pr_claim began the iteration and counted its sources
    if (ld_acquire_u32(&a.ctl->upd[slot]) == 0) return;
    if (threadIdx.x == 0) s_tally = CtaTally{};
    __syncthreads();
  } else {
    iter_begin<false>(a, s_tally);
  }
  unsigned long long my_edges = 0, my_srcs = 0, my_host = 0;
  const unsigned long long t0 = per_warp * (blockIdx.x * kWarpsPerCta + wid);
  const unsigned long long t1 = min(units, t0 + per_warp);
  if (t0 < t1) {
    const uint32_t first = warp_find_unit<kRelaxHeader>(a.ptr, a.from, a.size, a.edge_from, t0, lane);
    for (uint32_t i0 = first; i0 < a.size; i0 += 32) {
      const uint32_t idx = i0 + lane;
      uint32_t d = 0, boff = 0, how = kRowHost;
      double push = 0.0;
      bool past = true, head = false;
      if (idx < a.size) {
        const uint32_t i = a.from + idx;
        const uint32_t p0 = a.ptr[i], p1 = a.ptr[i + 1];
        push = a.qpush[i];
        const unsigned long long start = (unsigned long long)(p0 - a.edge_from) + (unsigned long long)kRelaxHeader * idx;
        past = start >= t1;
        uint32_t lo;
        d = unit_clip<kRelaxHeader>(start, p1 - p0, t0, t1, &lo, &head);
        if (a.iter > 1 && push == 0.0) d = 0;  // not claimed
        if (d || (kCache && head)) {
          boff = (kHost ? a.off[a.queue[i]] : a.streamed ? a.off[a.queue[i]] - a.stream_base : p0 - a.edge_from) + lo;
          if (kCache) {
            const uint32_t u = a.queue[i];
            how = cache_row(a.cache, u, boff - lo, p1 - p0);
            if (head && how == kRowStore) cache_stored(a.cache, u);
          }
        }
      }
      if (a.iter == 1) my_srcs += __popc(__ballot_sync(0xffffffffu, head));
      V row;
      if constexpr (kCache) {
        row.val = push;
        row.how = how;
        my_host += __reduce_add_sync(0xffffffffu, how != kRowHeld ? d : 0u);
      } else {
        row = push;
      }
      my_edges += warp_expand(s_exp[wid], lane, d, boff, row,
                              [&](const uint32_t (&pos)[kRelaxUnroll], const V (&rv)[kRelaxUnroll],
                                  const bool (&ok)[kRelaxUnroll]) { pr_lane<W, SRC>(a, pos, rv, ok); },
                              kHost);
      if (__any_sync(0xffffffffu, past)) break;
    }
  }
  warp_publish(s_tally, a.ctl, slot, lane, my_srcs != 0, my_edges, my_srcs, my_host);
}

// Async inner iterations > 1 of a partition without long rows: one launch in
// which each warp takes 32 sources, moves the residuals above acc into the
// ranks (value += delta; delta -= delta, atomically against concurrent
// pushes) and pushes its tile's edges.  PageRank-async to 1e-6 on an
// Erdos-Renyi graph of 4.2 M edges, 1643 passes: 23.3 ms of relaxation, 38.4
// with the claim and the cut, which pays where rows are long.
template <int W>
__global__ void __launch_bounds__(kRelaxThreads, SGW_RELAX_MIN_BLOCKS) k_pr_warp(PrArgs a) {
  chain_wait();
  chain_open();
  __shared__ CtaTally s_tally;
  __shared__ WarpExpand<double> s_exp[kWarpsPerCta];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (!iter_begin<true>(a, s_tally)) return;
  unsigned long long my_edges = 0, my_srcs = 0;
  for (uint32_t i0 = (blockIdx.x * kWarpsPerCta + wid) * 32u; i0 < a.size; i0 += gridDim.x * kRelaxThreads) {
    const uint32_t i = a.from + i0 + lane;
    uint32_t d = 0, boff = 0;
    double push = 0.0;
    if (i0 + lane < a.size) {
      const uint32_t u = a.queue[i];
      const uint32_t p0 = a.ptr[i], p1 = a.ptr[i + 1];
      const double res = ld_relaxed_f64(&a.delta[u]);
      if (res > a.acc) {
        a.pval[u] += res;
        atomicAdd(&a.delta[u], -res);
        d = p1 - p0;
        push = a.damping * res / (double)d;
        boff = a.streamed ? a.off[u] - a.stream_base : p0 - a.edge_from;
      }
    }
    my_srcs += __popc(__ballot_sync(0xffffffffu, d > 0));
    my_edges += warp_expand(s_exp[wid], lane, d, boff, push,
                            [&](const uint32_t (&pos)[kRelaxUnroll], const double (&pv)[kRelaxUnroll],
                                const bool (&ok)[kRelaxUnroll]) { pr_lane<W, kSrcBuffer>(a, pos, pv, ok); });
  }
  warp_publish(s_tally, a.ctl, (a.base + a.iter) & 3u, lane, my_srcs != 0, my_edges, my_srcs);
}

// Async inner iterations > 1 where some row is long: the partition's sources
// whose residual grew above acc are active again (value += delta; delta -= delta, atomically
// against pushes still to come); their pushes go to qpush.
__global__ void __launch_bounds__(kRelaxThreads) k_pr_claim(PrArgs a) {
  chain_wait();
  chain_open();
  __shared__ CtaTally s_tally;
  const int lane = threadIdx.x & 31;
  if (!iter_begin<true>(a, s_tally)) return;
  uint32_t srcs = 0;
  for (uint32_t i0 = (blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5)) * 32u; i0 < a.size;
       i0 += gridDim.x * kRelaxThreads) {
    const uint32_t i = a.from + i0 + lane;
    bool act = false;
    if (i0 + lane < a.size) {
      const uint32_t u = a.queue[i];
      const double res = ld_relaxed_f64(&a.delta[u]);
      double push = 0.0;
      act = res > a.acc;
      if (act) {
        a.pval[u] += res;
        atomicAdd(&a.delta[u], -res);
        push = a.damping * res / (double)(a.ptr[i + 1] - a.ptr[i]);
      }
      a.qpush[i] = push;
    }
    srcs += __popc(__ballot_sync(0xffffffffu, act));
  }
  warp_publish(s_tally, a.ctl, (a.base + a.iter) & 3u, lane, srcs != 0, 0, srcs);
}

// Single-vertex PR partition: the generate snapshot of its push.
__global__ void k_pr_hub_claim(uint32_t from, const double *qpush, Ctl *ctl) {
  ctl->hub_push = qpush[from];
}

template <int W>
__global__ void k_pr_flat(const uint32_t *buf, uint32_t count, uint32_t pbits, double *delta,
                          const Ctl *ctl) {
  const double push = ctl->hub_push;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
    uint32_t dst, w;
    load_edge<W>(buf, j, pbits, dst, w);
    atomicAdd(&delta[dst], push);
  }
}

// delta = init, value = 0 (subway/pr-sync.cu:36-40).
__global__ void k_pr_init(uint32_t n, double init, double *pval, double *delta) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    pval[v] = 0.0;
    delta[v] = init;
  }
}

// ---- learned scheduler: per-range statistics and prediction -------------------
struct RangeInfo {           // a static vertex range [v0, v1) with edges [e0, e1)
  uint32_t v0, v1;
  unsigned long long e0, e1;
};

struct RangeStat {           // one global iteration of one range
  uint32_t qa, qb;           // its segment of the active queue
  uint32_t edge_from;        // ptr[qa]
  uint32_t act_edges;        // ptr[qb] - ptr[qa]
  uint32_t prev_edges;       // act_edges of the previous global iteration
  uint32_t first_vertex;     // queue[qa]
  float pred;                // predicted active edge fraction next iteration
  float feat[kMlpIn];
  uint32_t pad;
};

// One warp per range: locate the range's queue segment, form the five
// features, evaluate the network (or, with no weights, predict that the
// current active edge fraction persists).
__global__ void k_range_stats(const RangeInfo *ranges, uint32_t num_ranges, const uint32_t *queue,
                              const uint32_t *ptr, const Ctl *ctl, RangeStat *st, const __nv_bfloat16 *w,
                              uint32_t iter, uint32_t cap) {
  chain_wait();
  chain_open();
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (s >= num_ranges) return;
  const RangeInfo r = ranges[s];
  const uint32_t count = ctl->num_active;
  // 32-way searches: five round trips to memory for 2^24 entries, where one lane
  // bisecting takes 24 (the kernel, network included: 25-28 us per global
  // iteration before, 8 with these and its weights read in 16-byte words)
  const uint32_t qa = warp_lower_bound(queue, count, r.v0, lane);
  const uint32_t qb = qa + warp_lower_bound(queue + qa, count - qa, r.v1, lane);
  const uint32_t efrom = ptr[qa];
  const uint32_t act = ptr[qb] - efrom;
  const uint32_t prev = st[s].prev_edges;
  const float redges = (float)(r.e1 - r.e0);
  float x[kMlpIn];
  x[0] = (r.v1 > r.v0) ? (float)(qb - qa) / (float)(r.v1 - r.v0) : 0.0f;
  x[1] = redges > 0.0f ? (float)act / redges : 0.0f;
  x[2] = fminf(fmaxf(__log2f(((float)act + 1.0f) / ((float)prev + 1.0f)) / 16.0f, -1.0f), 1.0f);
  x[3] = fminf((float)iter, 64.0f) / 64.0f;
  x[4] = cap ? fminf(redges / (float)cap, 1.0f) : 0.0f;
  const float pred = w ? mlp_forward_warp(w, x, lane) : x[1];
  if (lane == 0) {
    RangeStat o;
    o.qa = qa;
    o.qb = qb;
    o.edge_from = efrom;
    o.act_edges = act;
    o.prev_edges = act;  // becomes "previous" for the next iteration
    o.first_vertex = qb > qa ? queue[qa] : r.v0;
    o.pred = pred;
#pragma unroll
    for (int k = 0; k < kMlpIn; ++k) o.feat[k] = x[k];
    o.pad = prev;        // the previous count, reported with this iteration
    st[s] = o;
  }
}

__global__ void k_pr_to_f32(uint32_t n, const double *pval, float *out) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
    out[v] = (float)pval[v];
}

}  // namespace sgw
