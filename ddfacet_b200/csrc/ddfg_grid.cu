// BDA W-projection gridder for B200 (sm_100a).
//
// Restates DDFacet's gridder<> (DDFacet/Gridder/gridder.h:78-377) as persistent, facet-inner kernels
// (ddfg_queue.cuh):
//
//  * one lane owns one BDA block (a baseline, rows r in R, channels [c0, c1)) and walks its
//    visibilities exactly like the reference's hot loop 1 (gridder.h:182-301): first-corr flag,
//    facet phasor exp(i nu angle) with an FP64 argument, per-antenna Jones J_p^H V J_q,
//    weights, smearing factor, and the block means of (u + w Cu, v + w Cv, w, nu) in FP64 in
//    the reference's summation order (so the integer grid indices agree bit-for-bit);
//  * the warp applies every facet of its pack to its stripe of 32 blocks in turn: the block's
//    facet-independent inputs come from DRAM once per pack, the facet-dependent record (position,
//    Jones, phasor, Stokes) is formed per facet, and the 32 lanes lay each record's S x S taps
//    (hot loop 2, gridder.h:353-375) onto the facet grid through a tile in shared memory (scatter,
//    ddfg_taps.cuh; into an FP64 accumulator when the facet has a grid_acc buffer, folded into the
//    float32 grid at the end of the call);
//  * per-band weight sums and the Jones normalisation sums are reduced per warp into shared
//    accumulators of the pack's facets and flushed when the CTA moves to another pack.
//
// Stokes I without smearing and with Jones terms as stored -- what a major cycle spends its time on --
// has kernels of its own (grid_single_i, grid_block_i; ddfg_single.cuh); the general ones
// (grid_single_q, grid_block_q) take everything.  Single-visibility maps (every block one row and one
// channel) load the visibility's inputs once per stripe (load_single); averaged blocks are walked per
// facet (their rows stay L1/L2-hot), and blocks of the optional large-block list are walked by a
// whole warp each.
//
// What bounds them (256 channels, 25 facets of 1485^2, 310 M facet-visibilities, FP64 sums): 38.5 ms
// with a reduction per tap and run, on the FP64 reduction rate of L2 (16 sectors a record, 125 G
// sectors/s); with tiles 26.3 ms at 52 instructions and 2.4 sectors a record, on instruction issue (50 %)
// and the shared-memory / L1 data path (61 %) together -- 24 warps an SM instead of 16 change
// nothing.  64 channels, 735^2: 16.7 ms to 8.1 ms.
#include <cuda_runtime.h>

#include "ddfg_common.cuh"
#include "ddfg_gridblock.cuh"
#include "ddfg_internal.h"
#include "ddfg_queue.cuh"
#include "ddfg_single.cuh"
#include "ddfg_taps.cuh"

namespace ddfg {

constexpr int kBlockWarps = 12;  // warps an SM of the averaged-block kernels

// Adds the CTA's shared sums of the pack's npk facets to their float64 outputs.
__device__ __forceinline__ void flush_grid_sums(const ddfg_facet *sf, int npk, const double *s_acc, const Sched &sc,
                                                const ddfg_jones &js, int nchan) {
  for (int fi = 0; fi < npk; ++fi) {
    const ddfg_facet &f = sf[fi];
    const double *a = s_acc + (size_t)fi * sc.acc_stride;
    const double *a_chan = a + sc.small_copies * sc.small_stride;
    const int nsw = f.nband * f.npol;
    const int nsmall = nsw + (js.mode != 0 ? 2 * f.nband : 0);
    for (int i = threadIdx.x; i < nsmall; i += blockDim.x) {
      double v = 0.;
      for (int w = 0; w < sc.small_copies; ++w) v += a[w * sc.small_stride + i];
      double *dst = i < nsw ? f.sumwt + i : (f.sumjones ? f.sumjones + (i - nsw) : nullptr);
      if (i < nsw && !f.sumwt) dst = nullptr;
      if (dst && v != 0.) atomicAdd(dst, v);
    }
    if (js.mode != 0 && sc.chan_sums)
      for (int i = threadIdx.x; i < 2 * nchan; i += blockDim.x)
        if (f.sumjones_chan && a_chan[i] != 0.) atomicAdd(&f.sumjones_chan[i], a_chan[i]);
  }
}

// Single-visibility blocks: each warp loads its 32 visibilities' facet-independent inputs (map
// entries, uvw, flags, weights, visibilities, Jones indices) once and grids them onto every facet
// of the pack in turn.  ACC: facets may have FP64 accumulators.
template <int NPOL, int SLOTS, bool ACC>
__global__ void __launch_bounds__(256, NPOL == 2 && SLOTS == 4 ? 1 : 2) grid_single_q(const ddfg_vis vs, const ddfg_jones js,
                                                     const __grid_constant__ FacetTable tab, const GridParams gp,
                                                     const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Smem = ScatterSmem<NPOL, SLOTS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  Smem &ws = ((Smem *)smem_raw)[warp];
  ddfg_facet *sf = (ddfg_facet *)((Smem *)smem_raw + nwarps);
  double *s_n0m1 = (double *)(sf + sc.max_pack);
  double *s_acc = s_n0m1 + sc.max_pack;
  ws.clear(lane);
  __shared__ unsigned int ticket;
  for (int pack = 0; pack < sc.npacks; ++pack) {
    __syncthreads();
    if (threadIdx.x == 0) ticket = 0;
    const int npk = stage_pack(tab, sc, pack, sf, s_n0m1);
    for (int i = threadIdx.x; i < npk * sc.acc_stride; i += blockDim.x) s_acc[i] = 0.;
    __syncthreads();
    WarpWork work;
    work.start(sc);
    for (Work w; work.next(sc, pack, &ticket, lane, w);) {
      for (long long s = w.s0; s < w.s1; ++s) {
        const int64_t b = s * 32 + lane;
        SingleIn in;
        in.valid = false;
        if (b < vs.nblocks) load_single(vs, js, gp, b, in);
        const unsigned all = __ballot_sync(0xffffffffu, in.valid);
        if (!all) continue;
        const int band = __shfl_sync(0xffffffffu, in.gridchan, __ffs(all) - 1);
        const bool one_band = __all_sync(0xffffffffu, !in.valid || in.gridchan == band);
        const double wsum = warp_sum(in.valid ? in.fw : 0.);
        for (int fi = 0; fi < npk; ++fi) {
          const ddfg_facet &f = sf[fi];
          const int npol_used = min(gp.nvispol, f.npol);
          double *acc = s_acc + (size_t)fi * sc.acc_stride, *a = acc + warp * sc.warp_stride;  // this warp's sums
          GridRecord<NPOL> rec;
          grid_single_facet<NPOL>(in, vs, js, f, gp, s_n0m1[fi], rec);
          warp_add_single_sums<NPOL>(vs, js, f, rec, npol_used, all, one_band, wsum, sc.warp_stride != 0, a,
                                     a + f.nband * f.npol,
                                     sc.chan_sums ? acc + sc.small_copies * sc.small_stride : nullptr);
          scatter<NPOL, SLOTS, false, false, ACC>(rec, f, npol_used, ws, lane);
        }
      }
    }
    __syncthreads();
    flush_grid_sums(sf, npk, s_acc, sc, js, vs.nchan);
  }
}

// The same for Stokes I from the diagonal correlations, without smearing and with Jones terms as
// stored (ddfg_single.cuh).  BANDS: facets have several bands.
template <int SLOTS, bool BANDS>
__global__ void __launch_bounds__(256) grid_single_i(const ddfg_vis vs, const ddfg_jones js,
                                                     const __grid_constant__ FacetTable tab, const GridParams gp,
                                                     const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Smem = ScatterSmem<1, SLOTS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  Smem &ws = ((Smem *)smem_raw)[warp];
  JonesProduct<true> *keep = (JonesProduct<true> *)((Smem *)smem_raw + nwarps) + warp * sc.max_pack;
  FacetI *sfi = (FacetI *)((JonesProduct<true> *)((Smem *)smem_raw + nwarps) + nwarps * sc.max_pack);
  ddfg_facet *sf = (ddfg_facet *)(sfi + sc.max_pack);
  double *s_acc = (double *)(sf + sc.max_pack);
  ws.clear(lane);
  __shared__ unsigned int ticket;
  for (int pack = 0; pack < sc.npacks; ++pack) {
    __syncthreads();
    if (threadIdx.x == 0) ticket = 0;
    const int npk = stage_pack_i(tab, sc, js, pack, sf, sfi);
    for (int i = threadIdx.x; i < npk * sc.acc_stride; i += blockDim.x) s_acc[i] = 0.;
    __syncthreads();
    JonesUse ju;
    ju.forget();
    WarpWork work;
    work.start(sc);
    for (Work w; work.next(sc, pack, &ticket, lane, w);) {
      for (long long s = w.s0; s < w.s1; ++s) {
        const int64_t b = s * 32 + lane;
        SingleIn in;
        in.valid = false;
        JonesAt at;
        at.o0 = at.o1 = 0;
        if (b < vs.nblocks) load_single<false>(vs, js, gp, b, in);
        if (in.valid && js.mode != 0) at = jones_at(js, in.irow, in.ch);
        const unsigned all = __ballot_sync(0xffffffffu, in.valid);
        if (!all) continue;
        const int use = ju.stripe(js, in.valid, all, at);
        const int band = __shfl_sync(0xffffffffu, in.gridchan, __ffs(all) - 1);
        const bool one_band = __all_sync(0xffffffffu, !in.valid || in.gridchan == band);
        const double wsum = warp_sum(in.valid ? in.fw : 0.);
        for (int fi = 0; fi < npk; ++fi) {
          const FacetI &f = sfi[fi];
          float2 t0 = in.vm.v[0], t3 = in.vm.v[3];
          GridRecord<1> rec;
          rec.bb = 0.f;
          if (use) {
            const JonesProduct<true> jp = jones_for<true>(js, use, ju, in.valid, at, f.jones_dir, keep + fi, lane);
            t0 = jp.first(in.vm);
            t3 = jp.second(in.vm);
            rec.bb = jp.bb;
          }
          rec.valid = in.valid && in.gridchan < f.nband &&
                      geometry_i(f, dadd(in.U, dmul(in.W, f.cu)), dadd(in.V, dmul(in.W, f.cv)), in.W, in.recip, rec.g);
          const float2 corr = phasor_turns(-in.nu * (in.U * f.l0 + in.V * f.m0 + in.W * f.n0m1) * kInvC);
          const float2 wgt = cscale(corr, 0.5f * (float)in.fw);
          rec.stokes[0] = cfma(t3, wgt, cmul(t0, wgt));
          rec.gridchan = in.gridchan;
          rec.weight = rec.sumsqw = in.fw;
          rec.sumjones = (double)rec.bb * in.fw;
          rec.ch0 = in.ch;
          rec.single_chan = true;
          double *acc = s_acc + (size_t)fi * sc.acc_stride, *a = acc + warp * sc.warp_stride;  // this warp's sums
          warp_add_single_sums<1>(vs, js, sf[fi], rec, 1, all, one_band, wsum, sc.warp_stride != 0, a,
                                  a + f.nband * f.npol,
                                  sc.chan_sums ? acc + sc.small_copies * sc.small_stride : nullptr);
          scatter<1, SLOTS, false, false, true, BANDS>(rec, sf[fi], 1, ws, lane);
        }
      }
    }
    __syncthreads();
    flush_grid_sums(sf, npk, s_acc, sc, js, vs.nchan);
  }
}

// Averaged BDA blocks: each warp walks its 32 blocks for every facet of the pack in turn
// (grid_block_record resets its Jones cache per block, so the order is free); a block's rows,
// visibilities, flags and weights come from DRAM once per pack and from L1/L2 for the other
// facets.  A large-block item gives its block to the whole warp: lane 0 walks the FP64 means in the
// reference's order, the warp the rest (grid_block_record_warp).  The block walk needs ~170
// registers: twelve warps an SM, as three CTAs of four or (where one facet's sums need it) one of twelve.
template <int NPOL, int SLOTS, bool ACC>
__global__ void __launch_bounds__(kBlockWarps * 32, 1) grid_block_q(const ddfg_vis vs, const ddfg_jones js,
                                                       const __grid_constant__ FacetTable tab, const GridParams gp,
                                                       const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Smem = ScatterSmem<NPOL, SLOTS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Smem &ws = ((Smem *)smem_raw)[warp];
  ddfg_facet *sf = (ddfg_facet *)((Smem *)smem_raw + (blockDim.x >> 5));
  double *s_n0m1 = (double *)(sf + sc.max_pack);
  double *s_acc = s_n0m1 + sc.max_pack;
  JonesCache jc;
  ws.clear(lane);
  __shared__ unsigned int ticket;
  for (int pack = 0; pack < sc.npacks; ++pack) {
    __syncthreads();
    if (threadIdx.x == 0) ticket = 0;
    const int npk = stage_pack(tab, sc, pack, sf, s_n0m1);
    for (int i = threadIdx.x; i < npk * sc.acc_stride; i += blockDim.x) s_acc[i] = 0.;
    __syncthreads();
    WarpWork work;
    work.start(sc);
    for (Work w; work.next(sc, pack, &ticket, lane, w);) {
      const bool large = w.large;
      int64_t bl = 0;
      if (large) {
        bl = vs.large_blocks[w.s0];
        // entries that are out of range or not above the threshold belong to the stripes
        if (bl < 0 || bl >= vs.nblocks || block_nvis(vs, bl) <= vs.large_min_vis) continue;
        if (vs.sparsification && !vs.sparsification[bl]) continue;
      }
      for (long long s = w.s0; s < w.s1; ++s) {
        const int64_t b = large ? bl : s * 32 + lane;
        // blocks above the large-block threshold are the large items' work
        const bool mine = !large && b < vs.nblocks && !(vs.nlarge > 0 && block_nvis(vs, b) > vs.large_min_vis);
        for (int fi = 0; fi < npk; ++fi) {
          const ddfg_facet &f = sf[fi];
          const int npol_used = min(gp.nvispol, f.npol);
          double *acc = s_acc + (size_t)fi * sc.acc_stride, *a = acc + warp * sc.warp_stride;
          double *a_chan = acc + sc.small_copies * sc.small_stride;
          GridRecord<NPOL> rec;
          rec.valid = false;
          rec.single_chan = true;
          if (large) {
            BlockMeans bm{};
            if (lane == 0) bm = grid_block_means(vs, f, bl);
            grid_block_record_warp<NPOL>(vs, js, f, gp, bl, bm, s_n0m1[fi], 0, lane, npol_used, a_chan, rec);
          } else if (mine) {
            grid_block_record<NPOL>(vs, js, f, gp, b, s_n0m1[fi], rec, jc);
          }
          warp_add_block_sums<NPOL>(vs, js, f, gp, b, rec, npol_used, a, a + f.nband * f.npol, a_chan, jc,
                                    large && !rec.single_chan);
          scatter<NPOL, SLOTS, false, true, ACC>(rec, f, npol_used, ws, lane);
        }
      }
    }
    __syncthreads();
    flush_grid_sums(sf, npk, s_acc, sc, js, vs.nchan);
  }
}

// The visibilities of a block that `first`, first + step, ... number (rows, then channels): their
// weighted, phased and Jones-corrected sum and their weights' and Jones weights' sums, with the
// per-channel Jones sums.  The products are FP32, their sum FP64: in FP32 2048 visibilities that add up
// in phase lost 6e-7 of their sum.
struct BlockSums {
  double2 t;
  double weight, sumjones;
};
template <bool STRIDED>
__device__ __forceinline__ BlockSums block_sums_i(const ddfg_vis &vs, const ddfg_jones &js, const FacetI &f,
                                                  const BlockRange &r, int first, int step, double *s_chan) {
  BlockSums o;
  o.t = make_double2(0., 0.);
  o.weight = o.sumjones = 0.;
  LaneJones<true> lj;
  lj.forget();
  const int nch = r.ch1 - r.ch0;
  int inx = STRIDED ? first / nch : 0, ch = r.ch0 + (STRIDED ? first - inx * nch : 0);
  while (inx < r.nrows) {
    const int64_t irow = r.rows[inx];
    const double *up = vs.uvw + 3 * irow;
    const double dot = up[0] * f.l0 + up[1] * f.m0 + up[2] * f.n0m1;
    for (; ch < r.ch1; ch += step) {
      const int64_t at = irow * vs.nchan + ch;
      if (vs.flags[at * vs.ncorr]) continue;
      const float w = vs.weights[at];
      if (js.mode != 0) lj.at(js, irow, ch, f.jones_dir);
      const M2 v = load_vis(vs, at * vs.ncorr);
      const float2 wgt = cscale(phasor_turns(-vs.freqs[ch] * dot * kInvC), 0.5f * w);
      const float2 t0 = js.mode != 0 ? lj.jp.first(v) : v.v[0], t3 = js.mode != 0 ? lj.jp.second(v) : v.v[3];
      const float2 t = cfma(t3, wgt, cmul(t0, wgt));
      o.t.x += (double)t.x;
      o.t.y += (double)t.y;
      o.weight += (double)w;
      if (js.mode != 0) {
        const double j = (double)lj.jp.bb * (double)w;
        o.sumjones += j;
        if (s_chan) {
          atomicAdd(&s_chan[ch], j);
          atomicAdd(&s_chan[vs.nchan + ch], (double)w);
        }
      }
    }
    if (STRIDED) {
      const int over = ch - r.ch1;
      inx += 1 + over / nch;
      ch = r.ch0 + over % nch;
    } else {
      ++inx;
      ch = r.ch0;
    }
  }
  return o;
}

// The same as grid_block_q for Stokes I from the diagonal correlations, without smearing and with
// per-visibility Jones terms as stored.  Each lane first walks its block's means and forms its
// footprint, then the sums of the blocks that have one (so the per-channel Jones sums need no second
// walk).  One third of grid_block_q's code: that kernel ran at 0.9 instructions a cycle and SM on
// averaged blocks, waiting for instructions most of the time.
template <int SLOTS>
__global__ void __launch_bounds__(kBlockWarps * 32, 1) grid_block_i(const ddfg_vis vs, const ddfg_jones js,
                                                       const __grid_constant__ FacetTable tab, const GridParams gp,
                                                       const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Smem = ScatterSmem<1, SLOTS>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  Smem &ws = ((Smem *)smem_raw)[warp];
  FacetI *sfi = (FacetI *)((Smem *)smem_raw + nwarps);
  ddfg_facet *sf = (ddfg_facet *)(sfi + sc.max_pack);
  double *s_acc = (double *)(sf + sc.max_pack);
  ws.clear(lane);
  __shared__ unsigned int ticket;
  for (int pack = 0; pack < sc.npacks; ++pack) {
    __syncthreads();
    if (threadIdx.x == 0) ticket = 0;
    const int npk = stage_pack_i(tab, sc, js, pack, sf, sfi);
    for (int i = threadIdx.x; i < npk * sc.acc_stride; i += blockDim.x) s_acc[i] = 0.;
    __syncthreads();
    WarpWork work;
    work.start(sc);
    for (Work w; work.next(sc, pack, &ticket, lane, w);) {
      const bool large = w.large;
      int64_t bl = 0;
      if (large) {
        bl = vs.large_blocks[w.s0];
        // entries that are out of range or not above the threshold belong to the stripes
        if (bl < 0 || bl >= vs.nblocks || block_nvis(vs, bl) <= vs.large_min_vis) continue;
      }
      for (long long s = w.s0; s < w.s1; ++s) {
        const int64_t b = large ? bl : s * 32 + lane;
        bool mine = b < vs.nblocks && !(vs.sparsification && !vs.sparsification[b < vs.nblocks ? b : 0]);
        BlockRange r;
        r.nrows = r.ch0 = r.ch1 = 0;
        int gridchan = -1;
        if (mine) {
          r = block_range(vs, b);
          // blocks above the large-block threshold are the large items' work
          if (large) mine = lane == 0;
          else mine = !(vs.nlarge > 0 && (int64_t)r.nrows * (r.ch1 - r.ch0) > vs.large_min_vis);
          gridchan = r.ch1 > r.ch0 ? vs.chan_map[r.ch0] : -1;
        }
        BlockMeans lm;  // a large block's means on facet fi & ~31 + lane: a facet a lane, not one after the other
        for (int fi = 0; fi < npk; ++fi) {
          const FacetI &f = sfi[fi];
          if (large && (fi & 31) == 0 && fi + lane < npk)
            lm = block_means_i(vs, sfi[fi + lane].cu, sfi[fi + lane].cv, r.rows, r.nrows, r.ch0, r.ch1);
          double *acc = s_acc + (size_t)fi * sc.acc_stride, *a = acc + warp * sc.warp_stride;  // this warp's sums
          double *s_chan = sf[fi].sumjones_chan ? acc + sc.small_copies * sc.small_stride : nullptr;
          GridRecord<1> rec;
          rec.valid = false;
          BlockMeans m;
          if (large) {
            m.u = __shfl_sync(0xffffffffu, lm.u, fi & 31);
            m.v = __shfl_sync(0xffffffffu, lm.v, fi & 31);
            m.w = __shfl_sync(0xffffffffu, lm.w, fi & 31);
            m.nu = __shfl_sync(0xffffffffu, lm.nu, fi & 31);
            m.nvis = __shfl_sync(0xffffffffu, lm.nvis, fi & 31);
            m.last_ch = __shfl_sync(0xffffffffu, lm.last_ch, fi & 31);
          }
          if (mine && gridchan >= 0 && gridchan < f.nband) {
            if (!large) m = block_means_i(vs, f.cu, f.cv, r.rows, r.nrows, r.ch0, r.ch1);
            if (m.nvis > 0) {
              const double rw = m.nvis == 1 && vs.recip_wvl ? vs.recip_wvl[m.last_ch] : m.nu / kC;
              rec.valid = geometry_i(f, m.u, m.v, m.w, rw, rec.g);
            }
          }
          BlockSums o;
          if (large) {
            if (!__shfl_sync(0xffffffffu, rec.valid, 0)) continue;
            o = block_sums_i<true>(vs, js, f, r, lane, 32, s_chan);
            o.t = make_double2(warp_sum(o.t.x), warp_sum(o.t.y));
            o.weight = warp_sum(o.weight);
            o.sumjones = warp_sum(o.sumjones);
          } else if (rec.valid) {
            o = block_sums_i<false>(vs, js, f, r, 0, 1, s_chan);
          }
          if (rec.valid) {
            rec.stokes[0] = make_float2((float)o.t.x, (float)o.t.y);
            rec.gridchan = gridchan;
            rec.weight = rec.sumsqw = o.weight;
            rec.sumjones = o.sumjones;
          }
          warp_add_sums<1>(js, sf[fi], rec, 1, a, a + f.nband * f.npol);
          scatter<1, SLOTS, false, true>(rec, sf[fi], 1, ws, lane);
        }
      }
    }
    __syncthreads();
    flush_grid_sums(sf, npk, s_acc, sc, js, vs.nchan);
  }
}

// grid = fl(grid + acc); acc = 0, for every facet of the table that has an FP64 accumulator.
__global__ void fold_acc_kernel(const __grid_constant__ FacetTable tab, int nfacets) {
  const int fi = blockIdx.y;
  if (fi >= nfacets) return;
  const ddfg_facet &f = tab.f[fi];
  if (!f.grid_acc) return;
  float2 *grid = (float2 *)f.grid;
  double2 *acc = (double2 *)f.grid_acc;
  const int64_t n = (int64_t)f.nband * f.npol * f.ny * f.nx;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double2 a = acc[i];
    if (a.x != 0. || a.y != 0.) {
      const float2 g = grid[i];
      grid[i] = make_float2((float)((double)g.x + a.x), (float)((double)g.y + a.y));
      acc[i] = make_double2(0., 0.);
    }
  }
}

}  // namespace ddfg

using namespace ddfg;

namespace {

// Whether grid_single_i / grid_block_i take the call: Stokes I from XX/YY or RR/LL visibilities,
// per-visibility Jones terms for averaged blocks.
bool grid_is_i(const ddfg_vis *vs, const ddfg_jones *js, const GridParams &gp) {
  return !gp.dopsf && !vs->uvw_dt && jones_as_stored(js) && (vs->single_vis_blocks || js->mode != 2) &&
         (gp.policy == G_I_LIN2 || gp.policy == G_I_CIRC2 || gp.policy == G_I_LIN4 || gp.policy == G_I_CIRC4);
}

// Shared memory of a CTA besides what a facet of its pack takes, and that.
template <int NP, int SL>
size_t grid_smem(int warps) { return warps * sizeof(ScatterSmem<NP, SL>); }
size_t grid_facet_smem(int warps, int acc_stride, bool stokes_i, bool single) {
  return sizeof(ddfg_facet) + sizeof(double) * ((size_t)acc_stride + 1) + (stokes_i ? sizeof(FacetI) : 0) +
         (stokes_i && single ? warps * sizeof(JonesProduct<true>) : 0);
}

template <int NP, int SL>
int launch_grid_table(const ddfg_vis *vs, const ddfg_jones *js, const FacetTable &tab, const GridParams &gp,
                      Sched sc, int threads, const ddfg_batch *batch, bool acc, bool &zeroed, int counters,
                      cudaStream_t stream) {
  const bool single = vs->single_vis_blocks != 0, stokes_i = NP == 1 && grid_is_i(vs, js, gp);
  const size_t smem = grid_smem<NP, SL>(threads / 32) +
                      (size_t)sc.max_pack * grid_facet_smem(threads / 32, sc.acc_stride, stokes_i, single);
  constexpr bool one = NP == 1;  // one plane: one kernel for both kinds of grid
  bool bands = false;
  for (int i = 0; i < sc.nfacets; ++i) bands = bands || tab.f[i].nband > 1;
  const void *kern = stokes_i ? (!single ? (const void *)grid_block_i<SL>
                                 : bands ? (const void *)grid_single_i<SL, true>
                                         : (const void *)grid_single_i<SL, false>)
                     : acc ? (single ? (const void *)grid_single_q<NP, SL, true> : (const void *)grid_block_q<NP, SL, true>)
                           : (single ? (const void *)grid_single_q<NP, SL, one> : (const void *)grid_block_q<NP, SL, one>);
  int per_sm = 0;
  int rc = ddfg_kernel_prepare(kern, threads, smem, &per_sm);
  if (rc) return rc;
  if (batch && batch->ctas_per_sm > 0) per_sm = min(per_sm, (int)batch->ctas_per_sm);
  const int ctas = ddfg_num_ctas(per_sm);
  sched_split(sc, batch, ctas, threads / 32, !single);
  if ((rc = sched_counters(sc, false, ctas * (threads / 32), zeroed, counters, stream))) return rc;
  if (stokes_i && single && bands) grid_single_i<SL, true><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else if (stokes_i && single) grid_single_i<SL, false><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else if (stokes_i) grid_block_i<SL><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else if (single && acc) grid_single_q<NP, SL, true><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else if (single) grid_single_q<NP, SL, one><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else if (acc) grid_block_q<NP, SL, true><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  else grid_block_q<NP, SL, one><<<ctas, threads, smem, stream>>>(*vs, *js, tab, gp, sc);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "grid launch: %s", cudaGetErrorString(e));
  return DDFG_OK;
}

}  // namespace

int ddfg_launch_grid(const ddfg_vis *vs, const ddfg_jones *js, const ddfg_facet *facets, int nfacets, int policy,
                     int nvispol, int dopsf, const ddfg_batch *batch, cudaStream_t stream) {
  int max_support = 1, max_band = 1;
  bool any_acc = false;
  for (int i = 0; i < nfacets; ++i) {
    max_support = max(max_support, facets[i].max_support);
    max_band = max(max_band, facets[i].nband * (facets[i].npol + 2));
    any_acc = any_acc || facets[i].grid_acc != nullptr;
  }
  const int slots = tap_slots(max_support, nvispol);
  GridParams gp;
  gp.policy = policy;
  gp.nvispol = nvispol;
  gp.dopsf = dopsf;
  gp.freq_mean0 = vs->freq_mean;
  const bool single = vs->single_vis_blocks != 0, stokes_i = nvispol == 1 && grid_is_i(vs, js, gp);
  const bool chan_sums = js->mode != 0 && (!single || vs->nchan <= kSharedChannels);
  // A CTA's warps, copies of the weight and Jones sums and shared memory: two CTAs of eight warps an SM
  // (single visibilities) or three of four (averaged blocks), each with its warps' tiles and the sums of a
  // pack.  A copy a warp, or one that the warps share (atomics) where that makes fewer packs: with hundreds
  // of bands.  Where not even one facet's sums fit (averaged blocks of thousands of channels), all of an
  // SM's shared memory goes to one CTA, with the warps of three or, where their tiles leave too little, of
  // one.
  struct Shape {
    int warps, copies;
    size_t smem;
  };
  const int warps = single ? 8 : 4;
  const size_t smem = (single ? 110 : 74) * 1024;
  const Shape shapes[] = {
      {warps, warps, smem}, {warps, 1, smem}, {single ? warps : kBlockWarps, 1, 225 * 1024}, {warps, 1, 225 * 1024}};
  int want = (batch && batch->facets_per_pack > 0) ? batch->facets_per_pack : 16;
  want = max(1, min(want, nfacets));
  const Shape *shape = nullptr;
  int acc_stride = 0, fit = 0;
  for (const Shape &sh : shapes) {
    if (shape && (fit == want || sh.smem > shape->smem || sh.warps < shape->warps)) break;
    const int stride = sh.copies * max_band + (chan_sums ? 2 * vs->nchan : 0);
    const size_t per_facet = grid_facet_smem(sh.warps, stride, stokes_i, single);
    const size_t scatter = nvispol == 1   ? (slots == 2 ? grid_smem<1, 2>(sh.warps) : grid_smem<1, 4>(sh.warps))
                           : nvispol == 2 ? grid_smem<2, 2>(sh.warps)
                           : nvispol == 3 ? grid_smem<3, 2>(sh.warps)
                                          : grid_smem<4, 2>(sh.warps);
    const int n = sh.smem < scatter ? 0 : (int)min((sh.smem - scatter) / per_facet, (size_t)want);
    if (n < 1 || (shape && (nfacets + n - 1) / n >= (nfacets + fit - 1) / fit)) continue;
    shape = &sh;
    acc_stride = stride;
    fit = n;
  }
  if (!shape) return ddfg_set_error(DDFG_ESIZE, "grid: too many bands/channels for the shared accumulators");
  want = fit;
  unsigned int *counters = batch && !(batch->flags & 1) ? (unsigned int *)batch->workspace : nullptr;  // one a pack
  bool zeroed = false;
  const int ngroups = (nfacets + DDFG_TABLE_FACETS - 1) / DDFG_TABLE_FACETS;
  const long long nstripes = (vs->nblocks + 31) / 32;
  const int nlarge = vs->single_vis_blocks ? 0 : (int)(vs->nlarge < (1LL << 30) ? vs->nlarge : (1LL << 30));
  FacetTable tab_tl;  // host staging of the parameter table (copied into the launch)
  for (int g = 0; g < ngroups; ++g) {
    const int f0 = (int)(((long long)g * nfacets) / ngroups), f1 = (int)(((long long)(g + 1) * nfacets) / ngroups);
    const int n = f1 - f0;
    for (int i = 0; i < n; ++i) tab_tl.f[i] = facets[f0 + i];
    Sched sc;
    sc.nfacets = n;
    sc.npacks = (n + want - 1) / want;
    sc.max_pack = (n + sc.npacks - 1) / sc.npacks;
    sc.acc_stride = acc_stride;
    sc.small_stride = max_band;
    sc.small_copies = shape->copies;
    sc.warp_stride = shape->copies > 1 ? max_band : 0;
    sc.chan_sums = chan_sums;
    sc.nstripes = nstripes;
    sc.large_items = nlarge;
    sc.counter = counters ? counters + f0 : nullptr;  // a launch has at most as many packs as facets
    int rc;
#define LG(NP, SL) rc = launch_grid_table<NP, SL>(vs, js, tab_tl, gp, sc, 32 * shape->warps, batch, any_acc, zeroed, nfacets - f0, stream)
    if (slots == 2) {
      switch (nvispol) {
        case 1: LG(1, 2); break;
        case 2: LG(2, 2); break;
        case 3: LG(3, 2); break;
        default: LG(4, 2); break;
      }
    } else if (nvispol == 1) {
      LG(1, 4);
    } else {
      LG(2, 4);
    }
#undef LG
    if (rc) return rc;
    if (any_acc) {
      int64_t cells = 0;
      for (int i = 0; i < n; ++i)
        {
          const int64_t c = (int64_t)tab_tl.f[i].nband * tab_tl.f[i].npol * tab_tl.f[i].ny * tab_tl.f[i].nx;
          if (c > cells) cells = c;
        }
      const int bx = (int)((cells + 255) / 256 < 1024 ? (cells + 255) / 256 : 1024);
      fold_acc_kernel<<<dim3(bx, n), 256, 0, stream>>>(tab_tl, n);
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "grid fold: %s", cudaGetErrorString(e));
    }
  }
  return DDFG_OK;
}
