// BDA W-projection degridder for B200 (sm_100a).
//
// Restates DDFacet's degridder<> (DDFacet/Gridder/degridder.h:55-267) as persistent, facet-inner
// kernels (ddfg_queue.cuh):
//
//  * one lane owns one BDA block: band, mean frequency over the block's channels and the
//    unweighted row means of (u + w Cu, v + w Cv, w) in FP64 (degridder.h:138-167), then the
//    W plane, grid location and oversampling phase (degridder.h:170-200);
//  * the warp gathers each block's S x S footprint cooperatively -- lanes on consecutive cells
//    of a CF row, one coalesced load per lane and tap -- and reduces the partial sums
//    (degridder.h:202-212);
//  * the owning lane converts Stokes to correlations, applies the per-block or per-visibility
//    Jones, the facet phasor exp(+i nu angle) (FP64 argument) and the smearing factor, and
//    subtracts the prediction from the visibilities (degridder.h:214-264).
//
// Every facet of a pack is applied to a stripe by the warp that owns it, so the read-modify-write
// of a visibility never races and the result does not depend on scheduling; the reference
// serialises the same update across facet processes with named semaphores (degridder.h:236-263).
// Single-visibility maps sum the pack's predictions in registers and subtract once per pack.
//
// What bounds them (256 channels, 16 facets a pack): the latency of taps and model cells from L2 (half of
// the cycles between issues), the L1 data path (67 %: four wavefronts for a record's taps, five when its
// model cells change, four for its lane partials) and issue (57 %, 53 instructions a record) together;
// 310 M facet-visibilities took 28.3 ms before records went through shared memory, runs kept their model
// cells and Stokes I had kernels of its own (ddfg_single.cuh), 24.4 ms since.  Averaged blocks (9 uneven
// facets): 24.3 ms to 15.2 ms, on the latency of the block walks.
#include <cuda_runtime.h>

#include "ddfg_common.cuh"
#include "ddfg_degridblock.cuh"
#include "ddfg_internal.h"
#include "ddfg_queue.cuh"
#include "ddfg_single.cuh"
#include "ddfg_taps.cuh"

namespace ddfg {

// Single-visibility blocks: the warp loads its 32 visibilities' facet-independent inputs once,
// sums the predictions of every facet of the pack in registers, and subtracts the sum from each
// visibility once (one read-modify-write per pack).
template <int NPOL, int SLOTS>
__global__ void __launch_bounds__(256, NPOL == 1 ? (SLOTS == 2 ? 3 : 1) : 1)
    degrid_single_q(const ddfg_vis vs, const ddfg_jones js, const __grid_constant__ FacetTable tab,
                    const DegridParams dp, const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ddfg_facet *sf = (ddfg_facet *)smem_raw;
  double *s_n0m1 = (double *)(sf + sc.max_pack);
  const int lane = threadIdx.x & 31;
  __shared__ GatherSmem<NPOL> s_gather[8];
  GatherSmem<NPOL> &ws = s_gather[threadIdx.x >> 5];
  const int npk = stage_pack(tab, sc, 0, sf, s_n0m1);  // one pack a launch
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = 0;
  __syncthreads();
  WarpWork work;
  work.start(sc);
  for (Work w; work.next(sc, 0, &ticket, lane, w);) {
    for (long long s = w.s0; s < w.s1; ++s) {
      const int64_t b = s * 32 + lane;
      DSingleIn in;
      in.valid = false;
      if (b < vs.nblocks) degrid_load_single(vs, js, b, in);
      if (!__any_sync(0xffffffffu, in.valid)) continue;
      M2 sum;
#pragma unroll
      for (int p = 0; p < 4; ++p) sum.v[p] = czero();
      bool any = false;
      for (int fi = 0; fi < npk; ++fi) {
        const ddfg_facet &f = sf[fi];
        BlockGeom g;
        const bool valid = degrid_single_geom_in(in, f, g);
        float2 mine[NPOL];
        gather<NPOL, SLOTS>(valid, g, in.gridchan, f, ws, lane, mine);
        if (valid) {
          const M2 vb = degrid_single_pred<NPOL>(in, vs, js, f, dp, s_n0m1[fi], mine);
#pragma unroll
          for (int p = 0; p < 4; ++p) sum.v[p] = cadd(sum.v[p], vb.v[p]);
          any = true;
        }
      }
      if (any) {
        float2 *vp = (float2 *)vs.vis + (in.irow * vs.nchan + in.ch) * (int64_t)vs.ncorr;
        if (vs.ncorr == 4) {
          float4 a = *(float4 *)vp, c = *(float4 *)(vp + 2);
          a.x -= sum.v[0].x; a.y -= sum.v[0].y; a.z -= sum.v[1].x; a.w -= sum.v[1].y;
          c.x -= sum.v[2].x; c.y -= sum.v[2].y; c.z -= sum.v[3].x; c.w -= sum.v[3].y;
          *(float4 *)vp = a;
          *(float4 *)(vp + 2) = c;
        } else if (vs.ncorr == 2) {
          vp[0] = csub(vp[0], sum.v[0]);
          vp[1] = csub(vp[1], sum.v[3]);
        } else {
          vp[0] = csub(vp[0], sum.v[0]);
        }
      }
    }
  }
}

// The same for Stokes I without smearing and with Jones terms as stored (ddfg_single.cuh).
template <int SLOTS>
__global__ void __launch_bounds__(256, SLOTS == 2 ? 3 : 2)
    degrid_single_i(const ddfg_vis vs, const ddfg_jones js, const __grid_constant__ FacetTable tab,
                    const DegridParams dp, const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  GatherSmem<1> &ws = ((GatherSmem<1> *)smem_raw)[warp];
  JonesProduct<false> *keep = (JonesProduct<false> *)((GatherSmem<1> *)smem_raw + nwarps) + warp * sc.max_pack;
  FacetI *sfi = (FacetI *)((JonesProduct<false> *)((GatherSmem<1> *)smem_raw + nwarps) + nwarps * sc.max_pack);
  ddfg_facet *sf = (ddfg_facet *)(sfi + sc.max_pack);
  const int npk = stage_pack_i(tab, sc, js, 0, sf, sfi);  // one pack a launch
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = 0;
  __syncthreads();
  JonesUse ju;
  ju.forget();
  WarpWork work;
  work.start(sc);
  for (Work w; work.next(sc, 0, &ticket, lane, w);) {
    for (long long s = w.s0; s < w.s1; ++s) {
      const int64_t b = s * 32 + lane;
      DSingleIn in;
      in.valid = false;
      JonesAt at;
      at.o0 = at.o1 = 0;
      if (b < vs.nblocks) degrid_load_single<false>(vs, js, b, in);
      if (in.valid && js.mode != 0) at = jones_at(js, in.irow, in.ch);
      const unsigned all = __ballot_sync(0xffffffffu, in.valid);
      if (!all) continue;
      const int use = ju.stripe(js, in.valid, all, at);
      float2 sum[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) sum[p] = czero();
      bool any = false;
      for (int fi = 0; fi < npk; ++fi) {
        const FacetI &f = sfi[fi];
        BlockGeom g;
        const bool valid = in.valid && in.gridchan < f.nband &&
                           geometry_i(f, dadd(in.U, dmul(in.W, f.cu)), dadd(in.V, dmul(in.W, f.cv)), in.W, in.recip, g);
        float2 t;
        gather<1, SLOTS, false>(valid, g, in.gridchan, sf[fi], ws, lane, &t);
        t = cmul(t, phasor_turns(in.nu * (in.U * f.l0 + in.V * f.m0 + in.W * f.n0m1) * kInvC));
        if (use) {
          const JonesProduct<false> jp = jones_for<false>(js, use, ju, in.valid, at, f.jones_dir, keep + fi, lane);
          if (valid) {
#pragma unroll
            for (int p = 0; p < 4; ++p) sum[p] = cadd(sum[p], cmul(t, jp.k[p]));
          }
        } else if (valid) {
          sum[0] = cadd(sum[0], t);
          sum[3] = cadd(sum[3], t);
        }
        any = any || valid;
      }
      if (any) {
        float2 *vp = (float2 *)vs.vis + (in.irow * vs.nchan + in.ch) * (int64_t)vs.ncorr;
        if (vs.ncorr == 4) {
          float4 a = *(float4 *)vp, c = *(float4 *)(vp + 2);
          a.x -= sum[0].x; a.y -= sum[0].y; a.z -= sum[1].x; a.w -= sum[1].y;
          c.x -= sum[2].x; c.y -= sum[2].y; c.z -= sum[3].x; c.w -= sum[3].y;
          *(float4 *)vp = a;
          *(float4 *)(vp + 2) = c;
        } else if (vs.ncorr == 2) {
          vp[0] = csub(vp[0], sum[0]);
          vp[1] = csub(vp[1], sum[3]);
        } else {
          vp[0] = csub(vp[0], sum[0]);
        }
      }
    }
  }
}

// Averaged BDA blocks: each lane reads its block's header once per stripe, then every facet of
// the pack forms the footprint, gathers and applies its prediction.  A large-block item gives its
// block to the whole warp: lane 0 forms the footprint (row means in the reference's order), the
// warp gathers the taps and applies the prediction lane-strided (degrid_block_apply_warp).
template <int NPOL, int SLOTS>
__global__ void __launch_bounds__(256) degrid_block_q(const ddfg_vis vs, const ddfg_jones js,
                                                      const __grid_constant__ FacetTable tab, const DegridParams dp,
                                                      const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ddfg_facet *sf = (ddfg_facet *)smem_raw;
  double *s_n0m1 = (double *)(sf + sc.max_pack);
  const int lane = threadIdx.x & 31;
  __shared__ GatherSmem<NPOL> s_gather[8];
  GatherSmem<NPOL> &ws = s_gather[threadIdx.x >> 5];
  const int npk = stage_pack(tab, sc, 0, sf, s_n0m1);  // one pack a launch
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = 0;
  __syncthreads();
  WarpWork work;
  work.start(sc);
  for (Work w; work.next(sc, 0, &ticket, lane, w);) {
    const bool large = w.large;
    int64_t bl = 0;
    if (large) {
      bl = vs.large_blocks[w.s0];
      if (bl < 0 || bl >= vs.nblocks || block_nvis(vs, bl) <= vs.large_min_vis) continue;
    }
    for (long long s = w.s0; s < w.s1; ++s) {
      const int64_t b = large ? bl : s * 32 + lane;
      const bool inrange = b < vs.nblocks;
      DegridBlock d;
      if (inrange) degrid_block_header(vs, b, d);
      // blocks above the large-block threshold are the large items' work
      const bool mine = large ? lane == 0
                              : inrange && !(vs.nlarge > 0 &&
                                             (int64_t)d.nrows * (d.ch1 - d.ch0) > vs.large_min_vis);
      for (int fi = 0; fi < npk; ++fi) {
        const ddfg_facet &f = sf[fi];
        BlockGeom g;
        const bool valid = mine && degrid_block_geom(vs, f, d, g);
        float2 pred[NPOL];
        gather<NPOL, SLOTS>(valid, g, d.gridchan, f, ws, lane, pred);
        if (large) {
          if (__shfl_sync(0xffffffffu, valid, 0)) degrid_block_apply_warp<NPOL>(vs, js, f, dp, d, pred, 0, lane);
        } else if (valid) {
          degrid_block_apply<NPOL>(vs, js, f, dp, d, pred);
        }
      }
    }
  }
}

// One visibility of an averaged block: vis -= s exp(+i nu angle) J0 J1^H (jp NULL: no Jones terms).
__device__ __forceinline__ void block_vis_i(const ddfg_vis &vs, const JonesProduct<false> *jp, float2 s, int64_t irow, int ch,
                                            double dot) {
  const float2 t = cmul(s, phasor_turns(vs.freqs[ch] * dot * kInvC));
  float2 *vp = (float2 *)vs.vis + (irow * vs.nchan + ch) * (int64_t)vs.ncorr;
  if (vs.ncorr == 4) {
    float4 a = *(float4 *)vp, c = *(float4 *)(vp + 2);
    float2 v0 = make_float2(a.x, a.y), v1 = make_float2(a.z, a.w), v2 = make_float2(c.x, c.y), v3 = make_float2(c.z, c.w);
    // products first: the visibility is rounded once
    if (jp) {
      v0 = csub(v0, cmul(t, jp->k[0]));
      v1 = csub(v1, cmul(t, jp->k[1]));
      v2 = csub(v2, cmul(t, jp->k[2]));
      v3 = csub(v3, cmul(t, jp->k[3]));
    } else {
      v0 = csub(v0, t);
      v3 = csub(v3, t);
    }
    *(float4 *)vp = make_float4(v0.x, v0.y, v1.x, v1.y);
    *(float4 *)(vp + 2) = make_float4(v2.x, v2.y, v3.x, v3.y);
  } else {
    vp[0] = csub(vp[0], jp ? cmul(t, jp->k[0]) : t);
    if (vs.ncorr == 2) vp[1] = csub(vp[1], jp ? cmul(t, jp->k[3]) : t);
  }
}

// The same as degrid_block_q for Stokes I without smearing and with per-visibility Jones terms as
// stored (ddfg_single.cuh).
template <int SLOTS>
__global__ void __launch_bounds__(256, 2) degrid_block_i(const ddfg_vis vs, const ddfg_jones js,
                                                         const __grid_constant__ FacetTable tab,
                                                         const DegridParams dp, const Sched sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  GatherSmem<1> &ws = ((GatherSmem<1> *)smem_raw)[warp];
  FacetI *sfi = (FacetI *)((GatherSmem<1> *)smem_raw + nwarps);
  ddfg_facet *sf = (ddfg_facet *)(sfi + sc.max_pack);
  const int npk = stage_pack_i(tab, sc, js, 0, sf, sfi);  // one pack a launch
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = 0;
  __syncthreads();
  WarpWork work;
  work.start(sc);
  for (Work w; work.next(sc, 0, &ticket, lane, w);) {
    const bool large = w.large;
    int64_t bl = 0;
    if (large) {
      bl = vs.large_blocks[w.s0];
      if (bl < 0 || bl >= vs.nblocks || block_nvis(vs, bl) <= vs.large_min_vis) continue;
    }
    for (long long s = w.s0; s < w.s1; ++s) {
      const int64_t b = large ? bl : s * 32 + lane;
      DegridBlock d;
      d.nrows = d.ch0 = d.ch1 = 0;
      if (b < vs.nblocks) degrid_block_header(vs, b, d);
      // blocks above the large-block threshold are the large items' work
      const bool mine = large ? lane == 0
                              : d.ch1 > d.ch0 && d.nrows > 0 &&
                                    !(vs.nlarge > 0 && (int64_t)d.nrows * (d.ch1 - d.ch0) > vs.large_min_vis);
      for (int fi = 0; fi < npk; ++fi) {
        const FacetI &f = sfi[fi];
        BlockGeom g;
        bool valid = false;
        if (mine && d.gridchan >= 0 && d.gridchan < f.nband) {
          const RowMeans m = degrid_row_means(vs, f.cu, f.cv, d);
          valid = geometry_i(f, m.u, m.v, m.w, m.recip, g);
        }
        float2 t;
        gather<1, SLOTS, false>(valid, g, d.gridchan, sf[fi], ws, lane, &t);
        bool apply = valid;
        if (large) {
          apply = __shfl_sync(0xffffffffu, valid, 0);
          t = make_float2(__shfl_sync(0xffffffffu, t.x, 0), __shfl_sync(0xffffffffu, t.y, 0));
        }
        if (apply) {
          LaneJones<false> lj;
          lj.forget();
          const int nch = d.ch1 - d.ch0, step = large ? 32 : 1;
          const int64_t total = (int64_t)d.nrows * nch;
          int inx = 0, ch = 0;
          for (int64_t k = large ? lane : 0; k < total; k += step) {
            if (large) {
              inx = (int)(k / nch);
              ch = (int)(k - (int64_t)inx * nch);
            }
            const int64_t irow = d.rows[inx];
            const double *up = vs.uvw + 3 * irow;
            if (js.mode != 0) lj.at(js, irow, d.ch0 + ch, f.jones_dir);
            block_vis_i(vs, js.mode != 0 ? &lj.jp : nullptr, t, irow, d.ch0 + ch,
                        up[0] * f.l0 + up[1] * f.m0 + up[2] * f.n0m1);
            if (++ch == nch) {
              ch = 0;
              ++inx;
            }
          }
        }
      }
    }
  }
}

}  // namespace ddfg

using namespace ddfg;

namespace {

template <int NP, int SL>
int launch_degrid_table(const ddfg_vis *vs, const ddfg_jones *js, const FacetTable &tab, const DegridParams &dp,
                        Sched sc, const ddfg_batch *batch, bool &zeroed, int counters, cudaStream_t stream) {
  const bool single = vs->single_vis_blocks != 0;
  bool stokes_i = NP == 1 && dp.policy == D_DIAG_FROM_I && !vs->uvw_dt && jones_as_stored(js) &&
                  (single || js->mode != 2);
  for (int i = 0; i < sc.nfacets; ++i) stokes_i = stokes_i && !far_bands(tab.f[i]);
  const size_t smem = stokes_i ? 8 * sizeof(GatherSmem<1>) + (sizeof(ddfg_facet) + sizeof(FacetI) +
                                                              (single ? 8 * sizeof(JonesProduct<false>) : 0)) *
                                                                 (size_t)sc.max_pack
                               : (sizeof(ddfg_facet) + sizeof(double)) * (size_t)sc.max_pack;
  const void *kern = stokes_i ? (single ? (const void *)degrid_single_i<SL> : (const void *)degrid_block_i<SL>)
                              : (single ? (const void *)degrid_single_q<NP, SL> : (const void *)degrid_block_q<NP, SL>);
  int per_sm = 0;
  int rc = ddfg_kernel_prepare(kern, 256, smem, &per_sm);
  if (rc) return rc;
  if (batch && batch->ctas_per_sm > 0) per_sm = min(per_sm, (int)batch->ctas_per_sm);
  const int ctas = ddfg_num_ctas(per_sm);
  sched_split(sc, batch, ctas, 8, !single);
  if ((rc = sched_counters(sc, true, ctas * 8, zeroed, counters, stream))) return rc;
  if (stokes_i && single) degrid_single_i<SL><<<ctas, 256, smem, stream>>>(*vs, *js, tab, dp, sc);
  else if (stokes_i) degrid_block_i<SL><<<ctas, 256, smem, stream>>>(*vs, *js, tab, dp, sc);
  else if (single) degrid_single_q<NP, SL><<<ctas, 256, smem, stream>>>(*vs, *js, tab, dp, sc);
  else degrid_block_q<NP, SL><<<ctas, 256, smem, stream>>>(*vs, *js, tab, dp, sc);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "degrid launch: %s", cudaGetErrorString(e));
  return DDFG_OK;
}

}  // namespace

int ddfg_launch_degrid(const ddfg_vis *vs, const ddfg_jones *js, const ddfg_facet *facets, int nfacets, int policy,
                       int nvispol, const ddfg_batch *batch, cudaStream_t stream) {
  DegridParams dp;
  dp.policy = policy;
  dp.nvispol = nvispol;
  int max_support = 1;
  for (int i = 0; i < nfacets; ++i) max_support = max(max_support, facets[i].max_support);
  const int slots = tap_slots(max_support, nvispol);
  // One launch per pack: two packs of one launch could update the same visibility at once.
  // Default: every facet of a call in one pack (each visibility read and written once).
  const int per_launch = (batch && batch->facets_per_pack > 0) ? min((int)batch->facets_per_pack, DDFG_TABLE_FACETS)
                                                               : DDFG_TABLE_FACETS;
  const int ngroups = (nfacets + per_launch - 1) / per_launch;  // <= DDFG_MAX_FACETS
  // counters after the gridder's (a grid and a degrid call may share one workspace)
  unsigned int *counters = batch && !(batch->flags & 1) ? (unsigned int *)batch->workspace + kGridCounters : nullptr;
  bool zeroed = false;
  const long long nstripes = (vs->nblocks + 31) / 32;
  const int nlarge = vs->single_vis_blocks ? 0 : (int)(vs->nlarge < (1LL << 30) ? vs->nlarge : (1LL << 30));
  FacetTable tab;
  for (int g = 0; g < ngroups; ++g) {
    const int f0 = (int)(((long long)g * nfacets) / ngroups), f1 = (int)(((long long)(g + 1) * nfacets) / ngroups);
    const int n = f1 - f0;
    for (int i = 0; i < n; ++i) tab.f[i] = facets[f0 + i];
    Sched sc;
    sc.nfacets = n;
    sc.npacks = 1;
    sc.max_pack = n;
    sc.acc_stride = 0;
    sc.small_stride = 0;
    sc.chan_sums = 0;
    sc.nstripes = nstripes;
    sc.large_items = nlarge;
    sc.counter = counters ? counters + g : nullptr;
    int rc;
#define LD(NP, SL) rc = launch_degrid_table<NP, SL>(vs, js, tab, dp, sc, batch, zeroed, ngroups - g, stream)
    if (slots == 2) {
      switch (nvispol) {
        case 1: LD(1, 2); break;
        case 2: LD(2, 2); break;
        case 3: LD(3, 2); break;
        default: LD(4, 2); break;
      }
    } else if (nvispol == 1) {
      LD(1, 4);
    } else {
      LD(2, 4);
    }
#undef LD
    if (rc) return rc;
  }
  return DDFG_OK;
}
