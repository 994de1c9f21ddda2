// Batched multi-source BFS / SSSP over a graph resident in HBM: up to 64
// queries share one traversal, one lane (bit / distance column) per query.
// No counterpart in the reference, which answers one source per process.
//
// Device state: the CSR (packed 4-byte records when weights fit, as in the
// engine), per-vertex 64-bit lane masks, and for SSSP dist[v][lane]
// (vertex-major: an edge touches one 128-byte line per 32 queries), for BFS the
// bits of the levels as planes in the same space.  One iteration:
//   k_b_frontier  vertices with a next mask move it to the current mask and
//                 become rows of a compacted frontier with a prefix of work units
//   k_b_relax     the rows' edges, cut into equal shares for the warps: BFS one
//                 edge per lane for all queries at once, SSSP one edge per eight
//                 lanes and 32 queries
//   k_b_cond      sets the conditional handle: loop while the frontier was
//                 non-empty (bounded by an iteration limit)
// The iteration is the body of a CUDA-graph conditional WHILE node, so a
// whole batch is one graph launch with no host round trip per iteration.

#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <vector>

#include "sgw_internal.h"
#include "sgw_warp.cuh"

#define CK(call)                                                                       \
  do {                                                                                 \
    cudaError_t _e = (call);                                                           \
    if (_e != cudaSuccess)                                                             \
      return sgw::fail(SGW_ECUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), \
                       __FILE__, __LINE__);                                            \
  } while (0)

namespace {

using namespace sgw;

constexpr uint32_t kBInf = 4294967294u;
constexpr int kBThreads = 256;
constexpr int kBWarps = kBThreads / 32;

// Per-vertex lane masks.  BFS keeps the queries that have reached a vertex
// beside those that reach it next, so an edge tests both with one 16-byte
// load; SSSP uses `next` alone.
struct __align__(16) BMask {
  unsigned long long seen, next;
};

// Counter words (ctr).  Graph loop: [0..1] one 64-bit counter, the frontier's
// rows (high word) and work units (low word), [2] iterations run, [3] error
// (2 = iteration limit, 4 = a grid barrier gave up), [12] frontier vertices.
// Persistent form: [4..5] / [6..7] and [12] / [13] the counters of even / odd
// iterations, [8] barrier arrivals, [9] barrier generation.  [10] 16-bit
// overflow.
template <int L, bool SSSP>
__global__ void k_b_fill(uint32_t *dist, BMask *mask, uint32_t n) {
  const size_t stride = (size_t)gridDim.x * blockDim.x, t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (SSSP) {  // BFS answers are built from level planes that need no fill
    const uint4 inf = make_uint4(kBInf, kBInf, kBInf, kBInf);
    for (size_t i = t; i < (size_t)n * (L / 4); i += stride) reinterpret_cast<uint4 *>(dist)[i] = inf;
  }
  for (size_t v = t; v < n; v += stride) *reinterpret_cast<uint4 *>(&mask[v]) = make_uint4(0, 0, 0, 0);
}

template <int L, bool SSSP>
__global__ void k_b_seed(const uint32_t *src, uint32_t nsrc, uint32_t *dist, BMask *mask, uint32_t *ctr) {
  const uint32_t l = threadIdx.x;
  if (l < nsrc) {
    const uint32_t s = src[l];
    if (SSSP) dist[(size_t)s * L + l] = 0;
    atomicOr(&mask[s].next, 1ull << l);
  }
  if (l < 16) ctr[l] = 0;
}

// ---- frontier phase ----------------------------------------------------------------
// Every vertex whose `next` mask holds a query that is new to it joins the
// frontier: its mask moves to cur, and it gets a row in (rows, unit).  A row is
// 1 + ceil(degree / unit edges) work units; `unit` is its first one.  A CTA takes
// kBVerts vertices at a time and reserves their rows and units with one
// 64-bit add, so both counts are prefixes in the same order and the relax
// phase can cut the units into equal shares.  The units of a frontier that
// holds every vertex have to stay below 2^32: see b_unit_log2.
//
// Loads that follow writes made earlier in the same launch (the persistent
// form runs every phase in one kernel) go through L2 (__ldcg): L1 and the
// read-only path are not kept coherent within a kernel.
constexpr uint32_t kBUnitLog2 = 3, kBWideUnitLog2 = 6;  // edges of a work unit: 8, or 64
constexpr int kBPer = 4;          // vertices per thread
constexpr uint32_t kBVerts = kBThreads * kBPer;

struct BState {
  uint32_t n, pbits;
  const uint32_t *off, *edges;
  const unsigned long long *obase;
  uint32_t *dist;                // SSSP distances / BFS level planes
  unsigned long long *cur;
  BMask *mask;
  uint32_t *rows, *unit;         // frontier rows: vertex, first work unit
  uint32_t min_units;            // fewest units in a warp's share
  uint32_t unit_log2;            // edges of a work unit
};

struct BFrontierSmem {
  unsigned long long warp[kBWarps];
  unsigned long long base;
  uint32_t act;
};

// Level planes (BFS): bit l of plane k of vertex v is bit k of query l's
// level.  Plane k is first written, for every vertex, at level 2^k, so planes
// need no fill, a frontier vertex costs a few coalesced words per level instead
// of a scattered store per query, and the planes that a traversal of D levels
// writes take log2(D) words of the space that 32-bit levels would.
template <int L> struct BPlane { using T = unsigned long long; };
template <> struct BPlane<32> { using T = uint32_t; };

template <int L>
__device__ __forceinline__ void b_set_level(const BState &s, uint32_t v, unsigned long long fresh, uint32_t level) {
  using T = typename BPlane<L>::T;
  T *const plane = reinterpret_cast<T *>(s.dist);
  if (level == 0) return;
  if ((level & (level - 1)) == 0) {  // this level is the first with its highest bit
    plane[(size_t)(31 - __clz((int)level)) * s.n + v] = (T)fresh;
    return;
  }
  if (!fresh) return;
  for (uint32_t m = level; m; m &= m - 1) {
    T *const p = plane + (size_t)(__ffs((int)m) - 1) * s.n + v;
    *p = __ldcg(p) | (T)fresh;
  }
}

template <bool SSSP, int L>
__device__ __forceinline__ void b_frontier(const BState &s, BFrontierSmem &sm, unsigned long long *ctr,
                                           uint32_t *active, uint32_t level) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint32_t base = blockIdx.x * kBVerts; base < s.n; base += gridDim.x * kBVerts) {
    uint32_t units[kBPer], mine = 0, rows = 0, act = 0;
#pragma unroll
    for (int k = 0; k < kBPer; ++k) {
      const uint32_t v = base + k * kBThreads + tid;
      units[k] = 0;
      if (v >= s.n) continue;
      unsigned long long fresh;
      if (SSSP) {
        fresh = __ldcg(&s.mask[v].next);
        if (fresh) s.mask[v].next = 0ull;
      } else {
        const ulonglong2 m = __ldcg(reinterpret_cast<const ulonglong2 *>(&s.mask[v]));
        fresh = m.y & ~m.x;
        if (m.y) *reinterpret_cast<ulonglong2 *>(&s.mask[v]) = make_ulonglong2(m.x | fresh, 0ull);
        b_set_level<L>(s, v, fresh, level);
      }
      if (fresh) {
        s.cur[v] = fresh;
        ++act;
        const uint32_t deg = s.off[v + 1] - s.off[v];
        if (deg) {
          units[k] = 2 + ((deg - 1) >> s.unit_log2);
          mine += units[k];
          ++rows;
        }
      }
    }
    // exclusive prefix of (rows, units) over the CTA's threads
    unsigned long long incl = ((unsigned long long)rows << 32) | mine;
    const unsigned long long own = incl;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += y;
    }
    const uint32_t wact = __reduce_add_sync(0xffffffffu, act);
    if (tid == 0) sm.act = 0;
    if (lane == 31) sm.warp[warp] = incl;
    __syncthreads();
    if (lane == 0 && wact) atomicAdd(&sm.act, wact);
    if (tid == 0) {
      unsigned long long acc = 0;
#pragma unroll
      for (int w = 0; w < kBWarps; ++w) {
        const unsigned long long x = sm.warp[w];
        sm.warp[w] = acc;
        acc += x;
      }
      sm.base = acc ? atomicAdd(ctr, acc) : 0ull;
    }
    __syncthreads();
    if (tid == 0 && sm.act) atomicAdd(active, sm.act);
    unsigned long long at = sm.base + sm.warp[warp] + incl - own;
#pragma unroll
    for (int k = 0; k < kBPer; ++k)
      if (units[k]) {
        s.rows[at >> 32] = base + k * kBThreads + tid;
        s.unit[at >> 32] = (uint32_t)at;
        at += (1ull << 32) | units[k];
      }
    __syncthreads();  // the tables are rewritten by the next tile
  }
}

template <bool SSSP, int L>
__global__ void __launch_bounds__(kBThreads) k_b_frontier(BState s, uint32_t *ctr) {
  __shared__ BFrontierSmem sm;
  b_frontier<SSSP, L>(s, sm, reinterpret_cast<unsigned long long *>(ctr), ctr + 12, ctr[2]);
}

// ---- relax phase -------------------------------------------------------------------
// The frontier's work units are cut into equal shares of at most `share` (at
// least min_units, if the caller sets more than that); a warp
// finds a share's first row with a 32-way search and goes through its rows 32
// at a time, the first and the last clipped to the share.  (One warp per row or
// per piece of 256 edges left most warps waiting at the end of an iteration for
// the few that had drawn the long rows: 60% of the SSSP kernel's stalls.)
// SSSP shares are short, since a warp takes several microseconds per edge group
// and the rows, hubs first, should see each other's improvements (64 queries on
// R-MAT 2^20: 5.4 ms with 16 units, 5.9 with 64, 6.6 with 4); BFS shares are long
// enough to hide the search (0.50 ms with 256, 0.57 with 32, 0.73 with 16).
// f(u, e0, d, mask) gets a lane's row part.
constexpr uint32_t kBSsspShare = 16, kBBfsShare = 256;
// CTAs per SM each form is compiled for: SSSP gains from more warps than its
// registers would leave (1.39 ms unbounded, 1.01 at 5, 1.28 at 8 for 32 queries
// on R-MAT 2^18), BFS loses (0.49 ms at 3, 0.52 at 4, 0.86 at 6).
constexpr int kBSsspCtas = 5, kBBfsCtas = 3;
template <class F>
__device__ __forceinline__ void b_rows(const BState &s, unsigned long long total, uint32_t share, F f) {
  const uint32_t count = (uint32_t)(total >> 32), units = (uint32_t)total;
  const int lane = threadIdx.x & 31;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t per = max(s.min_units, min(share, (units + nw - 1) / nw));
  for (unsigned long long t0 = (unsigned long long)per * gw; t0 < units; t0 += (unsigned long long)per * nw) {
    const unsigned long long t1 = min((unsigned long long)units, t0 + per);
    uint32_t lo = 0, hi = count;  // last row whose first unit is <= t0
    while (hi - lo > 32u) {
      const uint32_t step = (hi - lo + 31u) / 32u, i = lo + (uint32_t)lane * step;
      const uint32_t m = __ballot_sync(0xffffffffu, i < hi && __ldcg(&s.unit[i]) <= t0);
      lo += (31u - (uint32_t)__clz((int)m)) * step;
      hi = min(hi, lo + step);
    }
    {
      const uint32_t i = lo + (uint32_t)lane;
      const uint32_t m = __ballot_sync(0xffffffffu, i < hi && __ldcg(&s.unit[i]) <= t0);
      lo += 31u - (uint32_t)__clz((int)m);
    }
    for (uint32_t i0 = lo; i0 < count; i0 += 32) {
      const uint32_t i = i0 + lane;
      uint32_t u = 0, d = 0;
      unsigned long long e0 = 0, mask = 0;
      bool past = true;
      if (i < count) {
        const unsigned long long first = (unsigned long long)__ldcg(&s.unit[i]) + 1;  // the row's first edge unit
        past = first > t1;
        if (!past) {
          u = __ldcg(&s.rows[i]);
          const uint32_t deg = s.off[u + 1] - s.off[u];
          const unsigned long long x = t0 > first ? (t0 - first) << s.unit_log2 : 0,
                                   y = t1 > first ? (t1 - first) << s.unit_log2 : 0;
          const unsigned long long end = min(y, (unsigned long long)deg);
          if (x < end) {
            d = (uint32_t)(end - x);
            e0 = off_at(s.off, s.obase, u) + x;
            mask = __ldcg(&s.cur[u]);
          }
        }
      }
      f(u, e0, d, mask);
      if (__any_sync(0xffffffffu, past)) break;
    }
  }
}

// What an edge needs of its row.
struct BRow {
  uint32_t lane;            // the row's lane
  uint32_t lo32;            // low word of the row's first edge
  unsigned long long e0;    // the row's first edge
  unsigned long long mask;
};
__device__ __forceinline__ size_t b_edge(const BRow &r, uint32_t pos) { return (size_t)r.e0 + (uint32_t)(pos - r.lo32); }

// BFS, bit-parallel over the lanes (multi-source BFS): lane i of a window takes
// edge i and adds the row's queries that have not reached the destination to
// its next mask.  The adds are non-returning, and only the frontier phase
// writes `seen`, so an edge whose queries are all there already costs one
// 16-byte load.
template <int W>
__device__ __forceinline__ void b_bfs_relax(const BState &s, WarpExpand<BRow> *exp, unsigned long long total) {
  const int lane = threadIdx.x & 31;
  const uint32_t dmask = s.pbits ? ((1u << s.pbits) - 1u) : 0xffffffffu;
  b_rows(s, total, kBBfsShare, [&](uint32_t, unsigned long long e0, uint32_t d, unsigned long long mask) {
    BRow r;
    r.lane = (uint32_t)lane;
    r.lo32 = (uint32_t)e0;
    r.e0 = e0;
    r.mask = mask;
    warp_expand(*exp, lane, d, (uint32_t)e0, r,
                [&](const uint32_t (&pos)[kRelaxUnroll], const BRow (&row)[kRelaxUnroll],
                    const bool (&ok)[kRelaxUnroll]) {
                  uint32_t dst[kRelaxUnroll];
                  ulonglong2 m[kRelaxUnroll];
#pragma unroll
                  for (int q = 0; q < kRelaxUnroll; ++q)
                    if (ok[q]) {
                      const size_t e = b_edge(row[q], pos[q]);
                      dst[q] = W == 1 ? (s.edges[e] & dmask) : s.edges[2 * e];
                    }
#pragma unroll
                  for (int q = 0; q < kRelaxUnroll; ++q)
                    if (ok[q]) m[q] = __ldcg(reinterpret_cast<const ulonglong2 *>(&s.mask[dst[q]]));
#pragma unroll
                  for (int q = 0; q < kRelaxUnroll; ++q)
                    if (ok[q]) {
                      const unsigned long long add = row[q].mask & ~(m[q].x | m[q].y);
                      if (add) atomicOr(&s.mask[dst[q]].next, add);
                    }
                });
  });
}

// SSSP: a lane relaxes one edge for four queries (16 bytes of distances), so
// eight lanes cover the 32 queries of one half and a warp four edges at once;
// kBGroup such groups of loads are in flight.  Lane i first loads edge i of a
// window (destination, weight, its row's lane), then each eight lanes take
// every fourth edge, reading the source's distances where the row changes and
// the destination's.  What bounds a batch is issuing instructions, not the L2:
// with one query per lane an edge cost a warp about 35 of them (32 queries on
// R-MAT 2^18: 2.6 ms, now 1.0; 64 on 2^20: 10.9 and 5.3).  A candidate below the
// value read improves the destination in this iteration (by this lane or by
// whichever wins), so non-returning reductions suffice and the lane bits are
// right.  In a small frontier, bound by latency, a query whose distance has
// improved again since the frontier phase is left to the next iteration, which
// it is in anyway: next bits are set before distances are lowered and read
// after them, so no distance travels two edges in one iteration and the number
// of iterations does not hang on timing.  In a large one a fresh distance is
// used at once, which saves a fifth of the time.
constexpr int kBGroup = 2;
constexpr uint32_t kBLarge = 32768;  // work units

template <int W, int L>
__device__ __forceinline__ void b_sssp_relax(const BState &s, WarpExpand<BRow> *exp, unsigned long long total) {
  const int lane = threadIdx.x & 31, g = lane >> 3, c = lane & 7;
  const uint32_t dmask = s.pbits ? ((1u << s.pbits) - 1u) : 0xffffffffu;
  const bool large = (uint32_t)total > kBLarge;
  b_rows(s, total, kBSsspShare, [&](uint32_t u, unsigned long long e0, uint32_t d0, unsigned long long mask) {
#pragma unroll 1
    for (int h = 0; h < L / 32; ++h) {
      uint32_t *const dist = s.dist + 32 * h + 4 * c;
      const uint32_t bits = d0 ? (uint32_t)(mask >> (32 * h)) : 0u;
      BRow r;
      r.lane = (uint32_t)lane;
      r.lo32 = (uint32_t)e0;
      r.e0 = e0;
      r.mask = 0;
      uint32_t held = 32;  // the row whose distances du holds
      uint4 du = make_uint4(kBInf, kBInf, kBInf, kBInf);
      warp_expand<1>(
          *exp, lane, bits ? d0 : 0u, (uint32_t)e0, r,
          [&](const uint32_t (&pos)[1], const BRow (&row)[1], const bool (&ok)[1]) {
            uint32_t rd = 0, rw = 0;
            if (ok[0]) {
              const size_t e = b_edge(row[0], pos[0]);
              if (W == 1) {
                const uint32_t x = s.edges[e];
                rd = x & dmask;
                rw = s.pbits ? (x >> s.pbits) : 0u;
              } else {
                rd = s.edges[2 * e];
                rw = s.edges[2 * e + 1];
              }
            }
            const uint32_t rl = row[0].lane;
            const uint32_t cnt = (uint32_t)__popc(__ballot_sync(0xffffffffu, ok[0]));  // a prefix of lanes
            for (uint32_t k0 = 0; k0 < cnt; k0 += 4 * kBGroup) {
              uint32_t dst[kBGroup], w[kBGroup];
              uint4 src[kBGroup], seen[kBGroup];
#pragma unroll
              for (int q = 0; q < kBGroup; ++q) {
                const uint32_t k = k0 + 4 * q + g, kk = min(k, cnt - 1);
                const uint32_t row_lane = __shfl_sync(0xffffffffu, rl, kk);
                dst[q] = __shfl_sync(0xffffffffu, rd, kk);
                w[q] = __shfl_sync(0xffffffffu, rw, kk);
                const uint32_t ru = __shfl_sync(0xffffffffu, u, row_lane);
                uint32_t on = __shfl_sync(0xffffffffu, bits, row_lane) >> (4 * c);
                if (row_lane != held) {
                  held = row_lane;
                  du = make_uint4(kBInf, kBInf, kBInf, kBInf);
                  if (on & 15u) {
                    du = __ldcg(reinterpret_cast<const uint4 *>(dist + (size_t)ru * L));
                    if (!large) {
                      __threadfence();  // a distance improved in this iteration comes after its next bit
                      on &= ~(__ldcg(reinterpret_cast<const uint32_t *>(&s.mask[ru].next) + h) >> (4 * c));
                    }
                    if (!(on & 1u)) du.x = kBInf;
                    if (!(on & 2u)) du.y = kBInf;
                    if (!(on & 4u)) du.z = kBInf;
                    if (!(on & 8u)) du.w = kBInf;
                  }
                }
                src[q] = du;
                seen[q] = make_uint4(0, 0, 0, 0);
                if (k < cnt && (on & 15u)) seen[q] = __ldcg(reinterpret_cast<const uint4 *>(dist + (size_t)dst[q] * L));
              }
#pragma unroll
              for (int q = 0; q < kBGroup; ++q) {
                const uint32_t cand[4] = {src[q].x + w[q], src[q].y + w[q], src[q].z + w[q], src[q].w + w[q]};
                uint32_t imp = 0;
                if (src[q].x != kBInf && cand[0] < seen[q].x) imp |= 1u;
                if (src[q].y != kBInf && cand[1] < seen[q].y) imp |= 2u;
                if (src[q].z != kBInf && cand[2] < seen[q].z) imp |= 4u;
                if (src[q].w != kBInf && cand[3] < seen[q].w) imp |= 8u;
                if (!__any_sync(0xffffffffu, imp)) continue;
                uint32_t m = imp << (4 * c);  // the edge's improved queries, from its eight lanes
                m |= __shfl_xor_sync(0xffffffffu, m, 1);
                m |= __shfl_xor_sync(0xffffffffu, m, 2);
                m |= __shfl_xor_sync(0xffffffffu, m, 4);
                if (c == 0 && m) atomicOr(&s.mask[dst[q]].next, (unsigned long long)m << (32 * h));
                if (!large) {  // uniform: the bits before the distances
                  __threadfence();
                  __syncwarp();
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if ((imp >> i) & 1u) atomicMin(dist + (size_t)dst[q] * L + i, cand[i]);
              }
            }
          });
    }
  });
}

template <bool SSSP, int W, int L>
__global__ void __launch_bounds__(kBThreads, SSSP ? kBSsspCtas : kBBfsCtas) k_b_relax(BState s, const uint32_t *ctr) {
  __shared__ WarpExpand<BRow> s_exp[kBWarps];
  const unsigned long long total = *reinterpret_cast<const unsigned long long *>(ctr);
  if (SSSP) b_sssp_relax<W, L>(s, &s_exp[threadIdx.x >> 5], total);
  else b_bfs_relax<W>(s, &s_exp[threadIdx.x >> 5], total);
}

// ---- persistent form -----------------------------------------------------------
// One cooperative launch runs every iteration of a batch: frontier phase,
// grid barrier, relaxation phase, grid barrier, and the loop test, all on the
// device.  The counters of even and odd iterations alternate (the next
// iteration's are cleared during the relaxation phase).  A barrier waits at
// most wait_ns (GPU global timer); a block that gives up records error 4 and
// returns, and every other block then gives up at its next barrier, so a lost
// block ends the kernel with an error instead of a hang.
struct BPersist {
  BState s;
  uint32_t max_iters, expect_blocks;
  unsigned long long wait_ns;
  uint32_t *ctr;
};

__device__ __forceinline__ unsigned long long b_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier with a bounded wait; false once any block has given up.
__device__ bool b_grid_sync(const BPersist &a) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile uint32_t *gen = a.ctr + 9;
    const uint32_t g = *gen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(a.ctr + 8, 1u) == a.expect_blocks - 1) {
      a.ctr[8] = 0;
      __threadfence();
      atomicAdd(a.ctr + 9, 1u);
    } else {
      const unsigned long long t0 = b_now();
      while (*gen == g) {
        if (b_now() - t0 > a.wait_ns) {
          atomicExch(a.ctr + 3, 4u);
          ok = 0;
          break;
        }
        __nanosleep(200);
      }
    }
    __threadfence();
    if (*(volatile uint32_t *)(a.ctr + 3) == 4u) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <bool SSSP, int W, int L>
__global__ void __launch_bounds__(kBThreads, SSSP ? kBSsspCtas : kBBfsCtas) k_b_persist(BPersist a) {
  __shared__ union {
    BFrontierSmem frontier;
    WarpExpand<BRow> exp[kBWarps];
  } sm;
  for (uint32_t it = 0;; ++it) {
    unsigned long long *c = reinterpret_cast<unsigned long long *>(a.ctr + 4 + 2 * (it & 1u));
    uint32_t *const act = a.ctr + 12 + (it & 1u);
    b_frontier<SSSP, L>(a.s, sm.frontier, c, act, it);
    if (!b_grid_sync(a)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *reinterpret_cast<unsigned long long *>(a.ctr + 4 + 2 * ((it + 1) & 1u)) = 0ull;
      a.ctr[12 + ((it + 1) & 1u)] = 0;
    }
    const unsigned long long total = *(volatile unsigned long long *)c;
    if (SSSP) b_sssp_relax<W, L>(a.s, &sm.exp[threadIdx.x >> 5], total);
    else b_bfs_relax<W>(a.s, &sm.exp[threadIdx.x >> 5], total);
    if (!b_grid_sync(a)) return;
    const bool more = *(volatile uint32_t *)act > 0;
    if (!more || it + 1 >= a.max_iters) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.ctr[2] = it + 1;
        if (more) a.ctr[3] = 2;  // iteration limit
      }
      return;
    }
  }
}

__global__ void k_b_cond(cudaGraphConditionalHandle handle, uint32_t *ctr, uint32_t max_iters) {
  const uint32_t it = ++ctr[2];
  uint32_t go = ctr[12] > 0 ? 1u : 0u;
  if (ctr[3]) go = 0;
  if (go && it >= max_iters) { ctr[3] = 2; go = 0; }
  ctr[0] = ctr[1] = 0;  // the next iteration's counters
  ctr[12] = 0;
  cudaGraphSetConditional(handle, go);
}

// BFS answers of vertices [v0, v0 + len): out[l * len + v - v0] = query l's
// level, put together from the level planes (lane i of a warp holds vertex i's
// words, so planes are read and answers written coalesced).  The traversal's
// last iteration found no fresh query: levels are below ctr[2].
template <int L, class OUT>
__global__ void k_b_levels(BState s, uint32_t v0, uint32_t len, uint32_t nsrc, OUT *out, uint32_t *ctr) {
  using T = typename BPlane<L>::T;
  const T *const plane = reinterpret_cast<const T *>(s.dist);
  const uint32_t planes = 32u - (uint32_t)__clz((int)(ctr[2] > 0 ? ctr[2] - 1 : 0));
  constexpr uint32_t kInf = sizeof(OUT) == 2 ? 0xffffu : kBInf;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= len) return;
  const uint32_t v = v0 + i;
  const T seen = (T)s.mask[v].seen;
  bool over = false;
  if (planes <= 4) {
    T p[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) p[k] = k < planes ? plane[(size_t)k * s.n + v] : (T)0;
    for (uint32_t l = 0; l < nsrc; ++l) {
      const uint32_t x = (uint32_t)((p[0] >> l) & 1) | (uint32_t)((p[1] >> l) & 1) << 1 |
                         (uint32_t)((p[2] >> l) & 1) << 2 | (uint32_t)((p[3] >> l) & 1) << 3;
      out[(size_t)l * len + i] = (OUT)((seen >> l) & 1 ? x : kInf);
    }
    return;
  }
  for (uint32_t l = 0; l < nsrc; ++l) {
    uint32_t x = 0;
    for (uint32_t k = 0; k < planes; ++k) x |= (uint32_t)((plane[(size_t)k * s.n + v] >> l) & 1) << k;
    if (!((seen >> l) & 1)) x = kInf;
    else if (sizeof(OUT) == 2 && x >= 0xffffu) { over = true; x = 0xfffeu; }
    out[(size_t)l * len + i] = (OUT)x;
  }
  if (over) atomicExch(&ctr[10], 1u);
}

// out[l * n + v - v0] = dist[v * L + l] for v in [v0, v0 + len), l < nsrc.
template <int L>
__global__ void k_b_transpose(const uint32_t *dist, uint32_t v0, uint32_t len, uint32_t nsrc, uint32_t *out,
                              uint32_t *) {
  __shared__ uint32_t tile[32][L + 1];
  const uint32_t vb = blockIdx.x * 32;
  for (uint32_t i = threadIdx.x; i < 32 * L; i += blockDim.x) {
    const uint32_t r = i / L, l = i % L;
    tile[r][l] = (vb + r < len) ? dist[(size_t)(v0 + vb + r) * L + l] : 0;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 32 * L; i += blockDim.x) {
    const uint32_t l = i / 32, r = i % 32;
    if (l < nsrc && vb + r < len) out[(size_t)l * len + vb + r] = tile[r][l];
  }
}

// 16-bit answers: unreached (kBInf) becomes 0xffff; a reached distance that
// does not fit below 0xffff sets *overflow (the run then reports SGW_ERANGE).
template <int L>
__global__ void k_b_transpose16(const uint32_t *dist, uint32_t v0, uint32_t len, uint32_t nsrc, uint16_t *out,
                                uint32_t *overflow) {
  __shared__ uint32_t tile[32][L + 1];
  const uint32_t vb = blockIdx.x * 32;
  for (uint32_t i = threadIdx.x; i < 32 * L; i += blockDim.x) {
    const uint32_t r = i / L, l = i % L;
    tile[r][l] = (vb + r < len) ? dist[(size_t)(v0 + vb + r) * L + l] : 0;
  }
  __syncthreads();
  bool over = false;
  for (uint32_t i = threadIdx.x; i < 32 * L; i += blockDim.x) {
    const uint32_t l = i / 32, r = i % 32;
    if (l < nsrc && vb + r < len) {
      uint32_t v = tile[r][l];
      if (v == kBInf) v = 0xffffu;
      else if (v >= 0xffffu) { over = true; v = 0xfffeu; }
      out[(size_t)l * len + vb + r] = (uint16_t)v;
    }
  }
  if (over) atomicExch(overflow, 1u);
}

}  // namespace

struct sgw_batch {
  const sgw_graph *g = nullptr;
  int device = 0;
  int num_sms = 0;
  uint32_t n = 0, W = 1, pbits = 0;
  uint64_t m = 0;
  uint32_t lanes = 64;            // 32 or 64 distance columns
  uint32_t min_units = 0;         // option: fewest work units of a warp's share (0: by algorithm)
  uint32_t unit_log2 = kBUnitLog2;
  char *d_arena = nullptr;
  size_t arena_bytes = 0;
  uint32_t *d_off = nullptr, *d_edges = nullptr, *d_dist = nullptr, *d_stage = nullptr;
  unsigned long long *d_obase = nullptr;  // u64 node pointers: full pointer of every 1024th vertex
  unsigned long long *d_cur = nullptr;
  BMask *d_mask = nullptr;
  uint32_t *d_rows = nullptr, *d_unit = nullptr;
  uint32_t *d_ctr = nullptr, *d_src = nullptr;
  uint32_t stage_vertices = 0;
  uint32_t *h_ctr = nullptr;      // pinned
  uint32_t *h_out = nullptr;      // pinned results, lanes x n (lane-major)
  cudaStream_t s = nullptr;
  cudaEvent_t t0 = nullptr, t1 = nullptr;
  cudaGraph_t graph[2] = {nullptr, nullptr};        // BFS, SSSP
  cudaGraphExec_t exec[2] = {nullptr, nullptr};
  uint32_t max_iters = 0;
  int form = 0;                   // 0: by algorithm, 1: persistent, 2: graph loop
};

namespace {

size_t al(size_t x) { return (x + 255) / 256 * 256; }

// Edges of a work unit, as a power of two.  A frontier's units are counted in
// the low 32 bits of a counter whose high word counts its rows, and a row of d
// edges has 1 + ceil(d / unit) of them, so a frontier of n vertices and m edges
// has at most 2 n + m / unit: 8 edges where that is below 2^32, 64 on larger
// graphs (156 n bytes of state and 4 m of edges fit 288 GB only with fewer than
// 2^32 of those).
uint32_t b_unit_log2(uint64_t n, uint64_t m) {
  return 2 * n + (m >> kBUnitLog2) < (uint64_t(1) << 32) ? kBUnitLog2 : kBWideUnitLog2;
}

BState state_of(const sgw_batch *b, bool sssp) {
  BState s;
  s.n = b->n;
  s.pbits = b->pbits;
  s.off = b->d_off;
  s.edges = b->d_edges;
  s.obase = b->d_obase;
  s.dist = b->d_dist;
  s.cur = b->d_cur;
  s.mask = b->d_mask;
  s.rows = b->d_rows;
  s.unit = b->d_unit;
  // a warp's share is at least 128 edges of BFS (one round of its loads) and 16 of
  // SSSP (two of its groups): a small frontier is spread over as many warps
  s.min_units = b->min_units ? b->min_units : sssp ? 2u : 16u;
  s.unit_log2 = b->unit_log2;
  return s;
}

template <bool SSSP, int W, int L>
int capture_body(sgw_batch *b, cudaGraph_t body, cudaGraphConditionalHandle h) {
  CK(cudaStreamBeginCaptureToGraph(b->s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
  const BState s = state_of(b, SSSP);
  const uint32_t tiles = (b->n + kBVerts - 1) / kBVerts;
  const uint32_t grid = (uint32_t)b->num_sms * 8;
  k_b_frontier<SSSP, L><<<std::min(tiles, grid), kBThreads, 0, b->s>>>(s, b->d_ctr);
  k_b_relax<SSSP, W, L><<<grid, kBThreads, 0, b->s>>>(s, b->d_ctr);
  k_b_cond<<<1, 1, 0, b->s>>>(h, b->d_ctr, b->max_iters);
  cudaGraph_t out = nullptr;
  CK(cudaStreamEndCapture(b->s, &out));
  return SGW_OK;
}

template <bool SSSP>
int build_graph(sgw_batch *b) {
  const int k = SSSP ? 1 : 0;
  CK(cudaGraphCreate(&b->graph[k], 0));
  cudaGraphConditionalHandle h;
  CK(cudaGraphConditionalHandleCreate(&h, b->graph[k], 1, cudaGraphCondAssignDefault));
  // the parameter union has no default constructor: build it in zeroed storage
  alignas(cudaGraphNodeParams) unsigned char raw[sizeof(cudaGraphNodeParams)];
  memset(raw, 0, sizeof(raw));
  cudaGraphNodeParams &cp = *reinterpret_cast<cudaGraphNodeParams *>(raw);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  CK(cudaGraphAddNode(&node, b->graph[k], nullptr, nullptr, 0, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  int st;
  if (b->lanes == 64)
    st = b->W == 1 ? capture_body<SSSP, 1, 64>(b, body, h) : capture_body<SSSP, 2, 64>(b, body, h);
  else
    st = b->W == 1 ? capture_body<SSSP, 1, 32>(b, body, h) : capture_body<SSSP, 2, 32>(b, body, h);
  if (st != SGW_OK) return st;
  CK(cudaGraphInstantiate(&b->exec[k], b->graph[k], 0));
  return SGW_OK;
}

// Launches the persistent kernel with as many blocks as fit on the device at
// once (the cooperative launch refuses more), so every block reaches the
// grid barriers.  extra_blocks > 0 makes each barrier wait for blocks that
// do not exist (the wait-limit check).
template <bool SSSP, int W, int L>
int launch_persist_t(sgw_batch *b, uint32_t extra_blocks, unsigned long long wait_ns) {
  int per_sm = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_b_persist<SSSP, W, L>, kBThreads, 0));
  if (per_sm < 1) return sgw::fail(SGW_ECUDA, "persistent batch kernel does not fit on an SM");
  const uint32_t grid = (uint32_t)b->num_sms * (uint32_t)std::min(per_sm, 8);
  BPersist a;
  a.s = state_of(b, SSSP);
  a.max_iters = b->max_iters;
  a.expect_blocks = grid + extra_blocks;
  a.wait_ns = wait_ns;
  a.ctr = b->d_ctr;
  void *args[] = {&a};
  CK(cudaLaunchCooperativeKernel((const void *)k_b_persist<SSSP, W, L>, dim3(grid), dim3(kBThreads), args, 0,
                                 b->s));
  return SGW_OK;
}

int launch_persist(sgw_batch *b, bool sssp, uint32_t extra_blocks, unsigned long long wait_ns) {
  if (b->lanes == 64) {
    if (b->W == 1) return sssp ? launch_persist_t<true, 1, 64>(b, extra_blocks, wait_ns)
                               : launch_persist_t<false, 1, 64>(b, extra_blocks, wait_ns);
    return sssp ? launch_persist_t<true, 2, 64>(b, extra_blocks, wait_ns)
                : launch_persist_t<false, 2, 64>(b, extra_blocks, wait_ns);
  }
  if (b->W == 1) return sssp ? launch_persist_t<true, 1, 32>(b, extra_blocks, wait_ns)
                             : launch_persist_t<false, 1, 32>(b, extra_blocks, wait_ns);
  return sssp ? launch_persist_t<true, 2, 32>(b, extra_blocks, wait_ns)
              : launch_persist_t<false, 2, 32>(b, extra_blocks, wait_ns);
}

// A grid barrier waits at most this long before the kernel gives up; a
// barrier of a healthy run waits for the slowest block of one phase (well
// under 100 ms on the largest graphs measured).
constexpr unsigned long long kBarrierWaitNs = 2000000000ull;

int batch_run(sgw_batch *b, int algo, const uint32_t *sources, uint32_t nsrc, void *out, uint32_t answer_bytes,
              sgw_batch_stats *stats, bool persistent, uint32_t extra_blocks, unsigned long long wait_ns);

// Default form per algorithm, measured with 7, 32 and 64 queries on R-MAT 14 to
// 24.  SSSP, 64 queries, persistent against graph: 1.76 and 1.84 ms on 2^18,
// 5.55 and 6.15 on 2^20, 22.0 and 25.0 on 2^22, 86.6 and 101 on 2^24; below 2^17
// the graph is ahead (0.75 and 0.71 ms on 2^16, 0.43 and 0.42 on 2^14).  BFS: 0.29
// and 0.25 ms on 2^18, 0.59 and 0.44 on 2^20, 7.5 and 5.5 on 2^24, equal on 2^14.
// So SSSP takes the persistent kernel and BFS the graph.
bool use_persistent(const sgw_batch *b, int algo) {
  return b->form == 1 || (b->form == 0 && algo == SGW_SSSP);
}

}  // namespace

extern "C" {

int sgw_batch_create(const sgw_graph *g, const sgw_engine_opts *opts, uint32_t lanes, sgw_batch **out) {
  sgw::clear_error();
  if (!g || !out) return sgw::fail(SGW_EINVAL, "null argument");
  *out = nullptr;
  if (lanes != 32 && lanes != 64) return sgw::fail(SGW_EINVAL, "lanes must be 32 or 64");
  sgw_engine_opts o;
  sgw_engine_opts_default(&o);
  if (opts) o = *opts;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return sgw::fail(SGW_ECUDA, "no CUDA device");
  }
  CK(cudaSetDevice(o.device));
  sgw_batch *b = new (std::nothrow) sgw_batch();
  if (!b) return sgw::fail(SGW_ENOMEM, "batch object");
  b->g = g;
  b->device = o.device;
  b->n = g->n;
  b->m = g->m;
  b->lanes = lanes;
  b->unit_log2 = (o.flags & SGW_OPT_BATCH_WIDE_UNITS) ? kBWideUnitLog2 : b_unit_log2(g->n, g->m);
  b->min_units = o.chunk_edges ? std::max<uint32_t>(1, o.chunk_edges >> b->unit_log2) : 0;
  if ((o.flags & SGW_OPT_BATCH_PERSISTENT) && (o.flags & SGW_OPT_BATCH_GRAPH)) {
    delete b;
    return sgw::fail(SGW_EINVAL, "SGW_OPT_BATCH_PERSISTENT and SGW_OPT_BATCH_GRAPH exclude each other");
  }
  b->form = (o.flags & SGW_OPT_BATCH_PERSISTENT) ? 1 : (o.flags & SGW_OPT_BATCH_GRAPH) ? 2 : 0;
  {
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, o.device) != cudaSuccess || !coop) {
      cudaGetLastError();
      if (b->form == 1) {
        delete b;
        return sgw::fail(SGW_EINVAL, "device %d has no cooperative launch", o.device);
      }
      b->form = 2;
    }
  }
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, o.device) != cudaSuccess) { delete b; return sgw::fail(SGW_ECUDA, "props"); }
  b->num_sms = prop.multiProcessorCount;
  // resident edge records: packed when the weights fit beside the ids
  uint32_t *packed = nullptr;
  size_t packed_bytes = 0;
  const void *src_edges = g->edges;
  b->W = g->weighted ? 2 : 1;
  if (g->weighted && !(o.flags & SGW_OPT_NO_PACK) && sgw::pack_weighted(g, &packed, &packed_bytes, &b->pbits)) {
    b->W = 1;
    src_edges = packed;
  }
  b->stage_vertices = std::min<uint32_t>(g->n, 1u << 22);
  const bool wide = g->node_pointer64 != nullptr;
  const size_t nbase = (g->n >> sgw::kOffGroupLog2) + 2;
  const size_t need = al(4ull * (g->n + 1)) + (wide ? al(8 * nbase) : 0) + al((size_t)g->m * 4 * b->W) + al((size_t)g->n * lanes * 4) +
                      al(8ull * g->n) + al(sizeof(BMask) * (size_t)g->n) + 2 * al(4ull * g->n) + al(64) + al(256) +
                      al((size_t)b->stage_vertices * lanes * 4);
  if (o.budget_bytes && need > o.budget_bytes) {
    sgw::host_free(packed);
    delete b;
    return sgw::fail(SGW_EBUDGET, "graph and %u query lanes need %zu B > budget %llu B", lanes, need,
                     (unsigned long long)o.budget_bytes);
  }
  auto cleanup = [&](int st) { sgw::host_free(packed); sgw_batch_destroy(b); return st; };
  if (cudaMalloc(&b->d_arena, need) != cudaSuccess) { cudaGetLastError(); return cleanup(sgw::fail(SGW_ECUDA, "cudaMalloc(%zu)", need)); }
  b->arena_bytes = need;
  char *p = b->d_arena;
  auto take = [&](size_t bytes) { char *r = p; p += al(bytes); return r; };
  b->d_off = (uint32_t *)take(4ull * (g->n + 1));
  if (wide) b->d_obase = (unsigned long long *)take(8 * nbase);
  b->d_edges = (uint32_t *)take((size_t)g->m * 4 * b->W);
  b->d_dist = (uint32_t *)take((size_t)g->n * lanes * 4);
  b->d_cur = (unsigned long long *)take(8ull * g->n);
  b->d_mask = (BMask *)take(sizeof(BMask) * (size_t)g->n);
  b->d_rows = (uint32_t *)take(4ull * g->n);
  b->d_unit = (uint32_t *)take(4ull * g->n);
  b->d_ctr = (uint32_t *)take(64);
  b->d_src = (uint32_t *)take(256);
  b->d_stage = (uint32_t *)take((size_t)b->stage_vertices * lanes * 4);
  b->max_iters = 4u * g->n + 64u;  // label-correcting rounds never exceed this
  if (cudaStreamCreateWithFlags(&b->s, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&b->t0) != cudaSuccess || cudaEventCreate(&b->t1) != cudaSuccess ||
      cudaMallocHost(&b->h_ctr, 64) != cudaSuccess ||
      cudaHostAlloc((void **)&b->h_out, (size_t)g->n * lanes * 4, cudaHostAllocPortable) != cudaSuccess)
    return cleanup(sgw::fail(SGW_ECUDA, "stream/event/pinned setup"));
  cudaError_t ce;
  if (!wide) {
    ce = cudaMemcpyAsync(b->d_off, g->node_pointer, 4ull * (g->n + 1), cudaMemcpyHostToDevice, b->s);
  } else {
    std::vector<uint32_t> lo((size_t)g->n + 1);
    std::vector<unsigned long long> base(nbase);
    if (!sgw::device_offsets(g, lo.data(), base.data()))
      return cleanup(sgw::fail(SGW_ERANGE, "1024 consecutive vertices hold 2^32 edges or more"));
    ce = cudaMemcpy(b->d_off, lo.data(), 4 * lo.size(), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemcpy(b->d_obase, base.data(), 8 * base.size(), cudaMemcpyHostToDevice);
  }
  if (ce == cudaSuccess && g->m)
    ce = cudaMemcpyAsync(b->d_edges, src_edges, (size_t)g->m * 4 * b->W, cudaMemcpyHostToDevice, b->s);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(b->s);
  sgw::host_free(packed);
  packed = nullptr;
  if (ce != cudaSuccess) return cleanup(sgw::fail(SGW_ECUDA, "graph upload: %s", cudaGetErrorString(ce)));
  int st = build_graph<false>(b);
  if (st == SGW_OK && g->weighted) st = build_graph<true>(b);
  if (st != SGW_OK) { sgw_batch_destroy(b); return st; }
  *out = b;
  return SGW_OK;
}

int sgw_batch_destroy(sgw_batch *b) {
  if (!b) return SGW_OK;
  cudaSetDevice(b->device);
  if (b->s) cudaStreamSynchronize(b->s);
  for (int k = 0; k < 2; ++k) {
    if (b->exec[k]) cudaGraphExecDestroy(b->exec[k]);
    if (b->graph[k]) cudaGraphDestroy(b->graph[k]);
  }
  if (b->t0) cudaEventDestroy(b->t0);
  if (b->t1) cudaEventDestroy(b->t1);
  if (b->s) cudaStreamDestroy(b->s);
  if (b->h_ctr) cudaFreeHost(b->h_ctr);
  if (b->h_out) cudaFreeHost(b->h_out);
  if (b->d_arena) cudaFree(b->d_arena);
  cudaGetLastError();
  delete b;
  return SGW_OK;
}

int sgw_batch_results(const sgw_batch *b, const uint32_t **results) {
  if (!b || !results) return sgw::fail(SGW_EINVAL, "null argument");
  *results = b->h_out;
  return SGW_OK;
}

uint32_t sgw_batch_unit_edges(uint32_t n, uint64_t m) { return 1u << b_unit_log2(n, m); }

int sgw_batch_device_bytes(const sgw_batch *b, uint64_t *bytes) {
  if (!b || !bytes) return sgw::fail(SGW_EINVAL, "null argument");
  *bytes = b->arena_bytes;
  return SGW_OK;
}

int sgw_batch_run(sgw_batch *b, int algo, const uint32_t *sources, uint32_t nsrc, uint32_t *out,
                  sgw_batch_stats *stats) {
  sgw::clear_error();
  if (!b) return sgw::fail(SGW_EINVAL, "null argument");
  return batch_run(b, algo, sources, nsrc, out, 4, stats, use_persistent(b, algo), 0, kBarrierWaitNs);
}

int sgw_batch_run_u16(sgw_batch *b, int algo, const uint32_t *sources, uint32_t nsrc, uint16_t *out,
                      sgw_batch_stats *stats) {
  sgw::clear_error();
  if (!b) return sgw::fail(SGW_EINVAL, "null argument");
  return batch_run(b, algo, sources, nsrc, out, 2, stats, use_persistent(b, algo), 0, kBarrierWaitNs);
}

int sgw_batch_check_wait_timeout(sgw_batch *b, uint64_t wait_ns) {
  sgw::clear_error();
  if (!b) return sgw::fail(SGW_EINVAL, "null argument");
  if (wait_ns == 0 || wait_ns > 1000000000ull) return sgw::fail(SGW_EINVAL, "wait_ns outside 1..1e9");
  const uint32_t src = 0;
  return batch_run(b, SGW_BFS, &src, 1, nullptr, 4, nullptr, true, 1, wait_ns);
}

}  // extern "C"

namespace {

int batch_run(sgw_batch *b, int algo, const uint32_t *sources, uint32_t nsrc, void *out, uint32_t answer_bytes,
              sgw_batch_stats *stats, bool persistent, uint32_t extra_blocks, unsigned long long wait_ns) {
  if (!b || !sources) return sgw::fail(SGW_EINVAL, "null argument");
  if (!out) out = b->h_out;  // results stay in the batch's pinned buffer
  if (nsrc == 0 || nsrc > b->lanes) return sgw::fail(SGW_ERANGE, "1..%u sources per batch", b->lanes);
  if (algo != SGW_BFS && algo != SGW_SSSP) return sgw::fail(SGW_EINVAL, "batches run BFS or SSSP");
  if (algo == SGW_SSSP && !b->g->weighted) return sgw::fail(SGW_EINVAL, "SSSP needs a weighted graph");
  for (uint32_t i = 0; i < nsrc; ++i)
    if (sources[i] >= b->n) return sgw::fail(SGW_EINVAL, "source %u out of range", sources[i]);
  CK(cudaSetDevice(b->device));
  const auto w0 = std::chrono::steady_clock::now();
  CK(cudaMemcpyAsync(b->d_src, sources, 4ull * nsrc, cudaMemcpyHostToDevice, b->s));
  CK(cudaEventRecord(b->t0, b->s));
  const bool sssp = algo == SGW_SSSP;
  const uint32_t fill = (uint32_t)b->num_sms * 8;
  if (b->lanes == 64) {
    if (sssp) k_b_fill<64, true><<<fill, 256, 0, b->s>>>(b->d_dist, b->d_mask, b->n);
    else k_b_fill<64, false><<<fill, 256, 0, b->s>>>(b->d_dist, b->d_mask, b->n);
    if (sssp) k_b_seed<64, true><<<1, 64, 0, b->s>>>(b->d_src, nsrc, b->d_dist, b->d_mask, b->d_ctr);
    else k_b_seed<64, false><<<1, 64, 0, b->s>>>(b->d_src, nsrc, b->d_dist, b->d_mask, b->d_ctr);
  } else {
    if (sssp) k_b_fill<32, true><<<fill, 256, 0, b->s>>>(b->d_dist, b->d_mask, b->n);
    else k_b_fill<32, false><<<fill, 256, 0, b->s>>>(b->d_dist, b->d_mask, b->n);
    if (sssp) k_b_seed<32, true><<<1, 64, 0, b->s>>>(b->d_src, nsrc, b->d_dist, b->d_mask, b->d_ctr);
    else k_b_seed<32, false><<<1, 64, 0, b->s>>>(b->d_src, nsrc, b->d_dist, b->d_mask, b->d_ctr);
  }
  CK(cudaGetLastError());
  if (persistent) {
    const int st = launch_persist(b, sssp, extra_blocks, wait_ns);
    if (st != SGW_OK) return st;
  } else {
    CK(cudaGraphLaunch(b->exec[sssp ? 1 : 0], b->s));
  }
  CK(cudaEventRecord(b->t1, b->s));
  // lane-major results, staged through a transposed device tile
  const size_t ab = answer_bytes;
  char *outb = static_cast<char *>(out);
  for (uint32_t v0 = 0; v0 < b->n; v0 += b->stage_vertices) {
    const uint32_t len = std::min(b->stage_vertices, b->n - v0);
    const uint32_t blocks = (len + 31) / 32;
    uint16_t *st16 = reinterpret_cast<uint16_t *>(b->d_stage);
    if (!sssp) {
      const BState s = state_of(b, false);
      const uint32_t lb = (len + 255) / 256;
      if (ab == 2) {
        if (b->lanes == 64) k_b_levels<64, uint16_t><<<lb, 256, 0, b->s>>>(s, v0, len, nsrc, st16, b->d_ctr);
        else k_b_levels<32, uint16_t><<<lb, 256, 0, b->s>>>(s, v0, len, nsrc, st16, b->d_ctr);
      } else {
        if (b->lanes == 64) k_b_levels<64, uint32_t><<<lb, 256, 0, b->s>>>(s, v0, len, nsrc, b->d_stage, b->d_ctr);
        else k_b_levels<32, uint32_t><<<lb, 256, 0, b->s>>>(s, v0, len, nsrc, b->d_stage, b->d_ctr);
      }
    } else if (ab == 2) {
      if (b->lanes == 64) k_b_transpose16<64><<<blocks, 256, 0, b->s>>>(b->d_dist, v0, len, nsrc, st16, b->d_ctr + 10);
      else k_b_transpose16<32><<<blocks, 256, 0, b->s>>>(b->d_dist, v0, len, nsrc, st16, b->d_ctr + 10);
    } else {
      if (b->lanes == 64) k_b_transpose<64><<<blocks, 256, 0, b->s>>>(b->d_dist, v0, len, nsrc, b->d_stage, nullptr);
      else k_b_transpose<32><<<blocks, 256, 0, b->s>>>(b->d_dist, v0, len, nsrc, b->d_stage, nullptr);
    }
    CK(cudaGetLastError());
    CK(cudaMemcpy2DAsync(outb + ab * v0, ab * b->n, b->d_stage, ab * len, ab * len, nsrc,
                         cudaMemcpyDeviceToHost, b->s));
  }
  CK(cudaMemcpyAsync(b->h_ctr, b->d_ctr, 64, cudaMemcpyDeviceToHost, b->s));
  CK(cudaStreamSynchronize(b->s));
  if (b->h_ctr[3] == 2) return sgw::fail(SGW_ETIMEOUT, "iteration limit reached");
  if (b->h_ctr[3] == 4) return sgw::fail(SGW_ETIMEOUT, "grid barrier wait timed out");
  if (b->h_ctr[10]) return sgw::fail(SGW_ERANGE, "a distance does not fit 16 bits: use sgw_batch_run");
  if (stats) {
    float ms = 0;
    cudaEventElapsedTime(&ms, b->t0, b->t1);
    stats->iterations = b->h_ctr[2];
    stats->queries = nsrc;
    stats->ms_device = ms;
    stats->ms_wall = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - w0).count();
    stats->d2h_bytes = ab * b->n * nsrc;
  }
  return SGW_OK;
}

}  // namespace

