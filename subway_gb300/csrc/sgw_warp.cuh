// Warp-level building blocks shared by the engine's and the batch kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace sgw {

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// First thing in a kernel that may be launched while its predecessor in the
// stream still runs (programmatic dependent launch): waits for the predecessor
// and its writes.  chain_open() then lets the successor's blocks be placed at
// once, where they wait in turn; only the short kernels do that, since blocks
// waiting beside a wide relaxation keep the registers that the next gather's
// blocks need (PageRank-async 3.0 against 2.8 ms).
// Such a kernel's inputs change while it runs, up to its wait: no parameter is
// `__restrict__`, and __ldg is for arrays that no kernel of the stream writes
// (node pointers, the host chunk table); both would allow a load before the
// wait.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Warp-inclusive scan of a u32.
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  return x;
}

// Edges each thread keeps in flight in the expansion loops: the record and
// destination-value loads of kRelaxUnroll edges are issued before any of
// their compares and atomics, so a warp waits on one memory round trip per
// kRelaxUnroll edges instead of per edge.
constexpr int kRelaxUnroll = 4;

// Expansion of up to 32 sources by one warp, shared by the warp kernels.  Lane
// i owns `d` edges that start at edge `boff` of the device buffer and carries
// `val`.  The sources that have edges are packed by rank into shared memory,
// and a bit per edge position marks where each one starts, kExpandSeg
// positions at a time; lane i of a 32-edge window then finds its edge's owner
// as (owners before the window) + (start bits up to its own) - 1: a broadcast
// word, a popcount and one 8-byte shared load.  f(position in the buffer,
// owner's value, which exist) is called for U edges of a lane at a time.
//
// What bounds the relaxation of a large frontier is instructions, not memory:
// the earlier owner search (warp votes, __fns and three shuffles per window)
// took most of them.  Relaxation per run, before and after: SSWP-async on
// R-MAT of 1.3 M vertices and 16 M 8-byte records in memory 1.37 and 0.98 ms,
// SSSP-async on R-MAT 2^25 (0.53 G edges, learned schedule) 14.9 and 12.4 ms.
constexpr uint32_t kExpandSeg = 2048;
template <class V>
struct WarpExpand {
  struct Own { uint32_t delta; V val; };
  uint32_t bits[kExpandSeg / 32];
  Own own[32];
};

template <int U = kRelaxUnroll, class V, class F>
__device__ __forceinline__ uint32_t warp_expand(WarpExpand<V> &s, int lane, uint32_t d, uint32_t boff, V val, F f,
                                                bool align = false) {
  uint32_t incl = warp_incl_scan(d, lane);
  uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  if (total == 0) return 0;
  const uint32_t edges = total;
  const bool own = d > 0;
  const uint32_t owners = __ballot_sync(0xffffffffu, own);
  uint32_t skip = 0;  // align: positions before the first edge that put the windows on multiples of 32
  if (align) {
    skip = __shfl_sync(0xffffffffu, boff, __ffs(owners) - 1) & 31u;
    incl += skip;
    total += skip;
  }
  const uint32_t excl = incl - d;
  const uint32_t le = lanemask_lt() | (1u << lane);
  if (own) {
    typename WarpExpand<V>::Own o;
    o.delta = boff - excl;  // buffer position of edge j of the tile: delta + j (mod 2^32)
    o.val = val;
    s.own[__popc(owners & (le >> 1))] = o;
  }
  uint32_t base = 0xffffffffu;  // owners that start before the window, minus one
  for (uint32_t seg = 0; seg < total; seg += kExpandSeg) {
    __syncwarp();
#pragma unroll
    for (uint32_t w = 0; w < kExpandSeg / 32; w += 32) s.bits[w + lane] = 0;
    __syncwarp();
    if (own && excl - seg < kExpandSeg) atomicOr(&s.bits[(excl - seg) >> 5], 1u << ((excl - seg) & 31u));
    __syncwarp();
    const uint32_t end = min(total - seg, kExpandSeg);
    for (uint32_t w0 = 0; w0 < end; w0 += 32u * U) {
      uint32_t pos[U];
      V sv[U];
      bool ok[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const uint32_t word = s.bits[w0 / 32u + q];
        const uint32_t j = w0 + 32u * q + lane;
        ok[q] = j < end && seg + j >= skip;
        const uint32_t r = base + __popc(word & le);
        base += __popc(word);
        if (ok[q]) {
          const typename WarpExpand<V>::Own o = s.own[r];
          pos[q] = o.delta + seg + j;
          sv[q] = o.val;
        }
      }
      f(pos, sv, ok);
    }
  }
  __syncwarp();  // the tables are rewritten by the next tile
  return edges;
}

}  // namespace sgw
