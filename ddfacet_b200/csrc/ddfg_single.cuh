// Stokes I without smearing: the case most of a major cycle's work is (one Stokes plane,
// per-antenna Jones terms taken as stored or none), with everything that does not depend on the
// visibility formed once.
//
// The general walk spends most of its instructions outside the taps: 64-bit Jones offsets, two 2 x 2
// products, four square roots for the Jones weight, an FP64 division and three 64-bit conversions a
// facet and visibility.  Here
//   * a pack's descriptors are staged with their derived FP64 constants;
//   * the two Jones matrices enter as one: gridding needs tr(J0^H V J1) = tr(V J1 J0^H), degridding
//     J0 (s 1) J1^H = s J0 J1^H.  A stripe is usually 32 channels of one row, which share their Jones
//     terms, and so do the row's other stripes: a warp keeps each facet's product (and weight) in
//     shared memory until the antennas, time slot or Jones channel change;
//   * the W plane's division is done only where a product with the reciprocal could round to another
//     integer.
// The integer indices are those of block_geometry, bit for bit.
#pragma once
#include "ddfg_common.cuh"
#include "ddfg_queue.cuh"

namespace ddfg {

struct FacetI {
  double cu, cv, l0, m0, n0m1;
  double scx, scy, hx, hy;                 // nx incr, n / 2 (gridder.h:142)
  double nwm1, ref_wave, wmax, rcp_wmax;
  const int32_t *cf_support;
  const int64_t *cf_offset;
  int64_t jones_dir;                       // first element of the facet's direction in the Jones array
  int32_t nx, ny, nw, overs, nband, npol;
};

// The facet's Jones product (and, gridding, its weight) of a warp's current row.  Gridding sums many
// visibilities under one product, so its rounding would not average out as those of their own
// products do: it is formed in FP64 and kept as two FP32 parts (one part: 7.3e-8 against 64 bits on
// averaged blocks, 5.1e-8 with a product a visibility).
template <bool GRID>
struct JonesProduct;
template <>
struct JonesProduct<false> {
  float2 k[4];
};
template <>
struct JonesProduct<true> {
  float2 k[4], lo[4];
  float bb;
  float pad[3];
  // The two terms of tr(V K): row by row, each rounded by itself.
  __device__ __forceinline__ float2 first(const M2 &v) const {
    return cfma(v.v[1], k[2], cfma(v.v[0], k[0], cfma(v.v[1], lo[2], cmul(v.v[0], lo[0]))));
  }
  __device__ __forceinline__ float2 second(const M2 &v) const {
    return cfma(v.v[3], k[3], cfma(v.v[2], k[1], cfma(v.v[3], lo[3], cmul(v.v[2], lo[1]))));
  }
};

// Whether the kernels of this file take a call's Jones terms.
inline bool jones_as_stored(const ddfg_jones *js) {
  return js->mode == 0 || (js->kms && !js->beam && js->interp_mode == 0 && js->apply_amp && js->apply_phase &&
                           !js->scale_jones && ((uintptr_t)js->kms & 15) == 0);
}

// Pack p's descriptors with their constants (all threads call it).
__device__ __forceinline__ int stage_pack_i(const FacetTable &tab, const Sched &sc, const ddfg_jones &js, int p,
                                            ddfg_facet *sf, FacetI *fi) {
  const int f0 = pack_first(sc, p), n = pack_first(sc, p + 1) - f0;
  const int words = n * (int)(sizeof(ddfg_facet) / sizeof(int));
  const int *src = (const int *)&tab.f[f0];
  for (int i = threadIdx.x; i < words; i += blockDim.x) ((int *)sf)[i] = src[i];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const ddfg_facet &f = tab.f[f0 + i];
    FacetI x;
    x.cu = f.cu; x.cv = f.cv; x.l0 = f.l0; x.m0 = f.m0;
    x.n0m1 = sqrt(1. - f.l0 * f.l0 - f.m0 * f.m0) - 1.;
    x.scx = dmul((double)f.nx, f.incr_x);
    x.scy = dmul((double)f.nx, f.incr_y);
    x.hx = (double)(f.nx / 2);
    x.hy = (double)(f.ny / 2);
    x.nwm1 = (double)f.nw - 1.0;
    x.ref_wave = f.ref_wave;
    x.wmax = f.wmax;
    x.rcp_wmax = 1. / f.wmax;
    x.cf_support = f.cf_support;
    x.cf_offset = f.cf_offset;
    x.jones_dir = js.mode != 0 ? (int64_t)f.idir_kms * js.kms_dims[2] * js.kms_dims[3] * 4 : 0;
    x.nx = f.nx; x.ny = f.ny; x.nw = f.nw; x.overs = f.overs; x.nband = f.nband; x.npol = f.npol;
    fi[i] = x;
  }
  return n;
}

// block_geometry from the staged constants.
__device__ __forceinline__ bool geometry_i(const FacetI &f, double umean, double vmean, double wmean,
                                           double recip_wvl, BlockGeom &g) {
  const double t = dmul(dmul(f.nwm1, fabs(wmean)), dmul(f.ref_wave, recip_wvl));
  double q = dmul(t, f.rcp_wmax);
  // q is within a few ulp of t / wmax: away from a half they round to the same integer
  if (!(fabs(q - rint(q)) < 0.499999)) q = t / f.wmax;
  const int iw = __double2int_rn(q);
  if (iw >= f.nw || iw < 0) return false;
  const int plane = wmean > 0. ? iw : f.nw + iw;
  const int S = __ldg(f.cf_support + plane), sup = (S - 1) / 2, O = f.overs;
  const double posx = dadd(dmul(dmul(f.scx, umean), recip_wvl), f.hx);
  const double posy = dadd(dmul(dmul(f.scy, vmean), recip_wvl), f.hy);
  const int lx = __double2int_rn(posx), ly = __double2int_rn(posy);
  if (lx < sup || lx >= f.nx - sup || ly < sup || ly >= f.ny - sup) return false;
  const int mid = (S * O - 1) / 2 - sup * O;
  const int io = __double2int_rn(dmul(dsub((double)ly, posy), (double)O)) + mid;
  const int jo = __double2int_rn(dmul(dsub((double)lx, posx), (double)O)) + mid;
  const int k = io * O + jo;
  if (k < 0 || k >= O * O) return false;
  g.locx = lx;
  g.locy = ly;
  g.sup = sup;
  g.S = S;
  g.cfoff = (int)(__ldg(f.cf_offset + plane) + (int64_t)k * S * S);
  return true;
}

// Element offsets of a visibility's two Jones matrices for direction 0.
struct JonesAt {
  int64_t o0, o1;
};
__device__ __forceinline__ JonesAt jones_at(const ddfg_jones &js, int64_t irow, int ichan) {
  const int64_t nd = js.kms_dims[1], na = js.kms_dims[2], nch = js.kms_dims[3];
  const int64_t t = js.kms_tmap[irow], c = js.kms_cmap[ichan];
  JonesAt x;
  x.o0 = (((t * nd) * na + js.a0[irow]) * nch + c) * 4;
  x.o1 = (((t * nd) * na + js.a1[irow]) * nch + c) * 4;
  return x;
}

__device__ __forceinline__ M2 load_jones(const ddfg_jones &js, int64_t off) {
  const float4 *p = (const float4 *)((const float2 *)js.kms + off);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  M2 m;
  m.v[0] = make_float2(a.x, a.y);
  m.v[1] = make_float2(a.z, a.w);
  m.v[2] = make_float2(b.x, b.y);
  m.v[3] = make_float2(b.z, b.w);
  return m;
}

// J1 J0^H (GRID) or J0 J1^H of a visibility for one facet, and its weight (JonesServer.cc:193-298).
template <bool GRID>
__device__ __forceinline__ JonesProduct<GRID> jones_product(const ddfg_jones &js, const JonesAt &at, int64_t dir) {
  const M2 j0 = load_jones(js, at.o0 + dir), j1 = load_jones(js, at.o1 + dir);
  JonesProduct<GRID> r;
  if constexpr (GRID) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {  // K_ij = sum_m J1_im conj(J0_jm)
        double x = 0., y = 0.;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const float2 a = j1.v[2 * i + m], c = j0.v[2 * j + m];
          x = fma((double)a.x, (double)c.x, fma((double)a.y, (double)c.y, x));
          y = fma((double)a.y, (double)c.x, fma(-(double)a.x, (double)c.y, y));
        }
        const float2 k = make_float2((float)x, (float)y);
        r.k[2 * i + j] = k;
        r.lo[2 * i + j] = make_float2((float)(x - (double)k.x), (float)(y - (double)k.y));
      }
    r.bb = jones_weight(j0, j1);
  } else {
    const M2 m = m2_times(j0, m2_herm(j1));
#pragma unroll
    for (int i = 0; i < 4; ++i) r.k[i] = m.v[i];
  }
  return r;
}

// A warp's use of its per-facet Jones products: 0 none, 1 a product per lane, 2 one for the stripe,
// to be formed and kept, 3 one for the stripe, kept already.
struct JonesUse {
  int64_t o0, o1;  // the kept products' offsets
  __device__ __forceinline__ void forget() { o0 = o1 = -1; }
  // All lanes call it; valid lanes pass their offsets.
  __device__ __forceinline__ int stripe(const ddfg_jones &js, bool valid, unsigned all, const JonesAt &at) {
    if (js.mode == 0) return 0;
    const int lead = __ffs(all) - 1;
    const int64_t l0 = __shfl_sync(0xffffffffu, at.o0, lead), l1 = __shfl_sync(0xffffffffu, at.o1, lead);
    if (!__all_sync(0xffffffffu, !valid || (at.o0 == l0 && at.o1 == l1))) return 1;
    const bool kept = l0 == o0 && l1 == o1;
    o0 = l0;
    o1 = l1;
    return kept ? 3 : 2;
  }
};

// The product of this lane's visibility for facet fi; all lanes call it (lanes without a visibility
// get a product nobody uses).
template <bool GRID>
__device__ __forceinline__ JonesProduct<GRID> jones_for(const ddfg_jones &js, int use, const JonesUse &u, bool valid,
                                                        const JonesAt &at, int64_t dir, JonesProduct<GRID> *keep,
                                                        int lane) {
  if (use == 3) return *keep;
  if (use == 1 && !valid) return JonesProduct<GRID>{};
  JonesAt x = at;
  if (use == 2) {
    x.o0 = u.o0;
    x.o1 = u.o1;
  }
  const JonesProduct<GRID> r = jones_product<GRID>(js, x, dir);
  if (use == 2) {
    __syncwarp();
    if (lane == 0) *keep = r;
    __syncwarp();
  }
  return r;
}

// ----------------------------------------------------------------------------------------
// Averaged blocks
// ----------------------------------------------------------------------------------------

// Rows [rows, rows + nrows) and channels [ch0, ch1) of a block.
struct BlockRange {
  const int32_t *rows;
  int nrows, ch0, ch1;
};
__device__ __forceinline__ BlockRange block_range(const ddfg_vis &vs, int64_t b) {
  const int64_t start = vs.block_start[b];
  BlockRange r;
  r.nrows = vs.bda_map[2 + b] - 2;
  r.ch0 = vs.bda_map[start];
  r.ch1 = vs.bda_map[start + 1];
  r.rows = vs.bda_map + start + 2;
  return r;
}

// A lane's Jones product, formed again where its antennas, time slot or channel change.
template <bool GRID>
struct LaneJones {
  int64_t o0, o1;
  JonesProduct<GRID> jp;
  __device__ __forceinline__ void forget() { o0 = o1 = -1; }
  __device__ __forceinline__ void at(const ddfg_jones &js, int64_t irow, int ch, int64_t dir) {
    const JonesAt x = jones_at(js, irow, ch);
    if (x.o0 == o0 && x.o1 == o1) return;
    o0 = x.o0;
    o1 = x.o1;
    jp = jones_product<GRID>(js, x, dir);
  }
};

// A visibility as a 2 x 2 matrix, padded as the gridder reads it.
__device__ __forceinline__ M2 load_vis(const ddfg_vis &vs, int64_t doff) {
  const float2 *vp = (const float2 *)vs.vis + doff;
  M2 m;
  if (vs.ncorr == 4) {
    const float4 a = *(const float4 *)vp, c = *(const float4 *)(vp + 2);
    m.v[0] = make_float2(a.x, a.y);
    m.v[1] = make_float2(a.z, a.w);
    m.v[2] = make_float2(c.x, c.y);
    m.v[3] = make_float2(c.z, c.w);
  } else {  // two correlations
    m.v[0] = vp[0];
    m.v[1] = m.v[2] = czero();
    m.v[3] = vp[1];
  }
  return m;
}

}  // namespace ddfg
