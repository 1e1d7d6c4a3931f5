// Persistent scheduling of the gridding and degridding kernels.
//
// One launch takes up to DDFG_TABLE_FACETS facet descriptors as a __grid_constant__ parameter
// table.  The facets are split into packs of balanced size.  A CTA walks the packs in order: it
// stages a pack's descriptors in shared memory, then each of its warps takes work of that pack
// until none is left:
//   * large blocks, one at a time, from the pack's counter in device memory (the longest work first);
//   * the stripes (32 consecutive blocks) of the CTA's chunks, about four fifths of all, from a
//     ticket in shared memory: the warps of a CTA work side by side on one run of the map and share
//     its tap tables, model cells and visibilities in L1;
//   * the last fifth from the pack's counter, which evens out what the chunks cost.
// Without counters (the unbatched calls) large blocks and the last fifth go round robin.
// Warps meet at a barrier only between packs: with a barrier per item of a CTA a tenth of the
// warps' time (a sixth on averaged blocks) went into waiting for its slowest warp; with small
// items handed to single warps instead, neighbouring stripes fell on different SMs and half of the
// L1 hits were lost (averaged degridding a sixth slower).  The pack-major order keeps the grids of
// one pack at a time live in L2.
#pragma once
#include "ddfg_common.cuh"

namespace ddfg {

struct FacetTable {
  ddfg_facet f[DDFG_TABLE_FACETS];
};

struct Sched {
  int nfacets;               // facets of this launch
  int npacks;
  int max_pack;              // most facets in one pack (shared-memory sizing)
  // Gridding: a facet's shared accumulators are small_copies copies of its weight and Jones sums (one a
  // warp, or one that the CTA's warps share), then its per-channel Jones sums.
  int acc_stride;            // doubles of one facet's accumulators, 0 for the other kernels
  int small_stride;          // doubles of a copy
  int small_copies;          // warps of a CTA, or 1
  int warp_stride;           // doubles from a warp's copy to the next warp's: small_stride, or 0
  int chan_sums;             // 1: the shared accumulators hold the per-channel Jones sums
  long long nstripes;        // stripes of 32 blocks
  int chunk;                 // stripes of a CTA's chunk
  int chunks;                // chunks a CTA
  int spread;                // 1: a CTA's chunks are neighbours, 0: the CTAs' chunks interleave
  int near;                  // 1: the CTA's stripes are neighbours and its warps take turns
  long long tail;            // first stripe of the last fifth
  int run;                   // its stripes an item
  long long large_items;     // large blocks
  unsigned int *counter;     // a counter a pack (zeroed before the launch), or NULL: round robin
};

// Host: the chunks and items of a launch of ctas CTAs of `warps` warps.  batch->stripes_per_item
// sets the chunk (0: 64 stripes of single visibilities, 16 of averaged blocks, whose stripes differ so
// much that longer chunks leave CTAs behind -- averaged gridding 42.9 ms with 64, 35.2 with 16; 256
// channels 26.3 with 64, 27.1 with 16 -- or an eighth of a CTA's stripes where that is less).
inline void sched_split(Sched &sc, const ddfg_batch *batch, int ctas, int warps, bool averaged) {
  const long long per_cta = sc.nstripes / ctas;
  long long chunk = batch && batch->stripes_per_item > 0 ? batch->stripes_per_item : averaged ? 16 : 64;
  if (chunk > per_cta / 8) chunk = per_cta / 8;
  if (chunk < warps) chunk = warps;
  sc.chunk = (int)chunk;
  // a CTA with less than two stripes a warp takes them all one by one
  sc.chunks = per_cta < 2 * warps ? 0 : (int)(per_cta * 4 / (5 * chunk));
  sc.near = 0;
  sc.spread = batch && (batch->flags & 4) ? 1 : 0;
  sc.tail = (long long)ctas * sc.chunks * sc.chunk;
  sc.run = sc.chunks > 0 && sc.nstripes - sc.tail > 8LL * ctas * warps ? 2 : 1;
}

// Host: zeroes the counters of a call's launches before the first that uses them (`n` from sc.counter
// on).  A launch with less than two stripes a warp and no large blocks has nothing to even out: it goes
// round robin, without the memset and one or two round trips a warp to one address.  Where it gathers
// and has at least a stripe a warp, a CTA's stripes are neighbours, which share model cells and taps in
// L1; scattering, neighbours would add to the same cells at once (whole calls with one
// facet: degridding 223,000 visibilities 50.3 us with the counter, 45.2 round robin, 43.2 with
// neighbours; gridding 115,000 visibilities 46.2, 46.5 and 50.7).
inline int sched_counters(Sched &sc, bool gathers, int warps_launched, bool &zeroed, int n, cudaStream_t stream) {
  if (sc.chunks == 0 && sc.large_items == 0) {
    sc.counter = nullptr;
    sc.near = gathers && sc.nstripes >= warps_launched ? 1 : 0;
  }
  if (!sc.counter || zeroed) return 0;
  const cudaError_t e = cudaMemsetAsync(sc.counter, 0, sizeof(unsigned int) * n, stream);
  if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "queue counters: %s", cudaGetErrorString(e));
  zeroed = true;
  return 0;
}

__device__ __forceinline__ int pack_first(const Sched &sc, int p) {
  return (int)(((long long)p * sc.nfacets) / sc.npacks);
}

// A warp's work: stripes [s0, s1), or large block number s0.
struct Work {
  bool large;
  long long s0, s1;
};

// A warp's walk over the work of one pack.
struct WarpWork {
  unsigned int held;  // the first item of the last fifth this warp got
  int phase;          // 0 large blocks, 1 chunks, 2 the last fifth
  unsigned int seq;   // items taken round robin
  __device__ __forceinline__ void start(const Sched &sc) {
    phase = sc.large_items > 0 ? 0 : 1;
    held = 0xffffffffu;
    seq = 0;
  }
  __device__ __forceinline__ unsigned int item(const Sched &sc, int pack, int lane) {
    unsigned int it = blockIdx.x + gridDim.x * ((threadIdx.x >> 5) + (blockDim.x >> 5) * seq);
    if (!sc.counter) ++seq;  // neighbouring items to different SMs
    else if (lane == 0) it = atomicAdd(sc.counter + pack, 1u);
    return __shfl_sync(0xffffffffu, it, 0);
  }
  // All lanes call it; false when the pack is done.
  __device__ __forceinline__ bool next(const Sched &sc, int pack, unsigned int *ticket, int lane, Work &w) {
    w.large = false;
    if (phase == 0) {
      held = item(sc, pack, lane);
      if (held < sc.large_items) {
        w.large = true;
        w.s0 = held;
        w.s1 = w.s0 + 1;
        return true;
      }
      phase = 1;
    }
    if (phase == 1) {
      unsigned int t = 0;
      if (sc.chunks > 0 && lane == 0) t = atomicAdd(ticket, 1u);
      t = __shfl_sync(0xffffffffu, t, 0);
      const unsigned int c = t / (unsigned)sc.chunk, o = t - c * (unsigned)sc.chunk;
      if (c < (unsigned)sc.chunks) {
        const long long at = sc.spread ? (long long)blockIdx.x * sc.chunks + c : blockIdx.x + (long long)gridDim.x * c;
        w.s0 = at * sc.chunk + o;
        w.s1 = w.s0 + 1;
        return true;
      }
      phase = 2;
    }
    if (sc.near) {
      const long long hi = (blockIdx.x + 1) * sc.nstripes / gridDim.x;
      w.s0 = blockIdx.x * sc.nstripes / gridDim.x + (threadIdx.x >> 5) + (blockDim.x >> 5) * seq++;
      w.s1 = w.s0 + 1;
      return w.s0 < hi;
    }
    const unsigned int it = held != 0xffffffffu ? held : item(sc, pack, lane);
    held = 0xffffffffu;
    w.s0 = sc.tail + (it - sc.large_items) * sc.run;
    w.s1 = min(w.s0 + sc.run, sc.nstripes);
    return w.s0 < sc.nstripes;
  }
};

// Copies pack p's descriptors into shared memory (all threads call it).
__device__ __forceinline__ int stage_pack(const FacetTable &tab, const Sched &sc, int p, ddfg_facet *sf,
                                          double *s_n0m1) {
  const int f0 = pack_first(sc, p), f1 = pack_first(sc, p + 1);
  const int n = f1 - f0;
  const int words = n * (int)(sizeof(ddfg_facet) / sizeof(int));
  const int *src = (const int *)&tab.f[f0];
  int *dst = (int *)sf;
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const ddfg_facet &f = tab.f[f0 + i];
    s_n0m1[i] = sqrt(1. - f.l0 * f.l0 - f.m0 * f.m0) - 1.;
  }
  return n;
}

}  // namespace ddfg
