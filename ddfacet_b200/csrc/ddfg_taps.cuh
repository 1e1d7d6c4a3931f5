// Warp-cooperative tap loops: laying a warp's records onto a facet grid (scatter) and gathering a
// warp's footprints from a model grid.
//
// A record is a block's footprint (S x S cells at an origin), its tap table and its values.  The
// lanes take its taps t = lane + 32 k; SLOTS taps a lane and pass, so footprints of more than 32
// SLOTS taps are walked in several passes and SLOTS sets registers, not the largest support.
// Records travel through the warp's shared memory (broadcast loads) instead of through four to six
// shuffles each, compacted so that the loops run over valid records only, four in flight: their
// loads are issued first, then their products in order.  Records of different supports (W planes
// of one stripe) are walked support by support.
#pragma once
#include <type_traits>

#include "ddfg_common.cuh"
#include "ddfg_gridblock.cuh"

namespace ddfg {

// Cells of a facet's bands together do not fit an int32 index: records are then taken band by band.
__host__ __device__ __forceinline__ bool far_bands(const ddfg_facet &f) {
  return f.nband > 1 && (int64_t)f.nband * f.npol * f.ny * f.nx > 0x7fffffff;
}

// Taps a lane and pass for the largest support of a launch: supports up to 8 fit two; wider ones take
// four, or two where the Stokes planes multiply the registers.
inline int tap_slots(int max_support, int npol) { return max_support <= 8 || npol > 2 ? 2 : 4; }

// Row t / S of tap t < S^2 (S <= 63); any value in range for taps past the footprint.
__device__ __forceinline__ int tap_row(int t, int S) {
  return __float2int_rz(__fdividef((float)t + 0.5f, (float)S));
}

// ----------------------------------------------------------------------------------------
// Scatter, one Stokes plane: runs in registers, stripes in a shared-memory tile
// ----------------------------------------------------------------------------------------
// Consecutive blocks of a map are neighbouring channels or times of one baseline: their footprints
// coincide in runs and otherwise overlap.  A run is summed in registers; a finished run is added to
// the warp's tile of shared memory that covers the records' bounding box (plain loads and stores:
// the lanes of one run own different cells, a __syncwarp orders runs); the tile reaches the grid
// once, one addition a touched cell.  A B200 takes 120-130 G 32-byte sectors a second of FP64
// reductions wherever they fall, which bounded the gridder when every run went to the grid (16
// sectors a record on 256 channels, 31 on 64).
//
// The tile holds FP64 sums for a facet with an FP64 accumulator, FP32 sums otherwise, so a run reaches
// the same sum as it would in the grid.  (FP32 tiles under FP64 grids would be 3 % faster on 256
// channels and raise the error against 64 bits from 4.9e-8 to 6.4e-8.)  It is kept all zero between
// uses: what adds it to the grid clears it.  Its pitch is a multiple of 16 (FP64: 8) cells plus the
// support where that fits: the rows of a footprint then fall on distinct banks.
template <int CELLS>
struct alignas(16) TileSmem {
  double2 tile[CELLS];
  int4 rec[32];  // byte offset of the footprint's origin in the tile, tap table offset, value
};

// Shared-memory accesses by 32-bit address.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float2 lds_f2(unsigned a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double2 lds_d2(unsigned a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double lds_d(unsigned a) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int4 lds_i4(unsigned a) {
  int4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts_f2(unsigned a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts_d2(unsigned a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void sts_d(unsigned a, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// *p += v unless v is zero.
__device__ __forceinline__ void red_add_f64(double *p, double v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.neu.f64 p, %1, 0d0000000000000000;\n\t@p red.global.add.f64 [%0], %1;\n\t}" ::"l"(
                   p),
               "d"(v)
               : "memory");
}

// v onto complex128 cell `cell` of acc (none if negative) for every lane of the warp: lanes 2i and
// 2i+1 swap halves so that each reduction carries whole cells.  A cell's two doubles in one
// instruction are one sector operation instead of two, and the sectors are what FP64 reductions
// cost: 7 x 7 footprints, 249 G cells/s against 126 G cells/s with one instruction for the real and
// one for the imaginary parts.  Cells ca and cb are the pair's first and second.
template <typename T2>
__device__ __forceinline__ void red_add_pair_f64(double *acc, int ca, int cb, T2 v, int lane) {
  const bool odd = lane & 1;
  const auto got = __shfl_xor_sync(0xffffffffu, odd ? v.x : v.y, 1);
  double *d = acc + (lane & 1);
  if (ca >= 0) red_add_f64(d + 2 * (size_t)ca, odd ? got : v.x);
  if (cb >= 0) red_add_f64(d + 2 * (size_t)cb, odd ? v.y : got);
}
__device__ __forceinline__ void red_add_cells_f64(double *acc, int cell, float2 v, int lane) {
  const int other = __shfl_xor_sync(0xffffffffu, cell, 1);
  red_add_pair_f64(acc, lane & 1 ? other : cell, lane & 1 ? cell : other, v, lane);
}

// Adds the products of n records (a multiple of four) of support S to the tile, taps first ..
// first + 32 SLOTS - 1.  Bit j of runs: record j starts a run.  F64: an FP64 tile; RUN64: the runs'
// sums in FP64 too (of products rounded to FP32).
template <int SLOTS, bool CONJ, bool F64, bool RUN64>
__device__ __forceinline__ void tile_pass(unsigned tile, unsigned recs, int n, unsigned runs, int S, int first,
                                          int pitch, const float2 *cfd, int lane) {
  bool on[SLOTS];
  unsigned cell[SLOTS];
  using Sum = typename std::conditional<RUN64, double2, float2>::type;
  Sum acc[SLOTS];
  float2 c[4][SLOTS];
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) {
    const int t = first + lane + 32 * k, sy = tap_row(t, S);
    on[k] = t < S * S;
    cell[k] = tile + (F64 ? 16 : 8) * (sy * pitch + t - sy * S);
    acc[k].x = acc[k].y = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) c[r][k] = czero();
  }
  cfd += first + lane;
  unsigned cur = 0;
  auto flush = [&]() {  // the run's sums to the tile
    __syncwarp();
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      const unsigned a = cell[k] + cur;
      if (on[k]) {
        if (F64) {
          const double2 t = lds_d2(a);
          sts_d2(a, make_double2(t.x + (double)acc[k].x, t.y + (double)acc[k].y));
        } else {
          const float2 t = lds_f2(a);
          sts_f2(a, make_float2(t.x + (float)acc[k].x, t.y + (float)acc[k].y));
        }
      }
      acc[k].x = acc[k].y = 0;
    }
  };
  for (int i = 0; i < n; i += 4) {
    int4 q[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      q[r] = lds_i4(recs + 16 * (i + r));
      const float2 *p = cfd + q[r].y;
#pragma unroll
      for (int k = 0; k < SLOTS; ++k)
        if (on[k]) c[r][k] = __ldg(p + 32 * k);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (runs >> (i + r) & 1) flush();  // the same for all lanes
      cur = q[r].x;
      const float2 v = make_float2(__int_as_float(q[r].z), __int_as_float(q[r].w));
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) {
        if constexpr (RUN64) {
          const float2 t = cmul(CONJ ? cconj(c[r][k]) : c[r][k], v);
          acc[k].x += (double)t.x;
          acc[k].y += (double)t.y;
        } else {
          acc[k] = CONJ ? cfma_conj(c[r][k], v, acc[k]) : cfma(c[r][k], v, acc[k]);
        }
      }
    }
  }
  flush();
  __syncwarp();
}

// Adds the tile's bw x bh cells to the grid at cell `origin` and clears them, row by row.
__device__ __forceinline__ void tile_to_grid(unsigned tile, int bw, int bh, int pitch, const ddfg_facet &f,
                                             size_t origin, int lane) {
  if (f.grid_acc) {
    // a lane a double: a cell's two halves in one instruction are one sector operation
    for (int j = lane; j < 2 * bw; j += 32) {
      unsigned t = tile + 8 * j;
      double *d = (double *)f.grid_acc + 2 * origin + j;
#pragma unroll 4
      for (int r = 0; r < bh; ++r) {
        const double v = lds_d(t);
        sts_d(t, 0.);
        red_add_f64(d, v);
        t += 16 * pitch;
        d += 2 * (ptrdiff_t)f.nx;
      }
    }
  } else {
    for (int j = lane; j < bw; j += 32) {
      unsigned t = tile + 8 * j;
      float2 *d = (float2 *)f.grid + origin + j;
#pragma unroll 4
      for (int r = 0; r < bh; ++r) {
        const float2 v = lds_f2(t);
        sts_f2(t, czero());
        if (v.x != 0.f || v.y != 0.f) red_add(d, v);
        t += 8 * pitch;
        d += f.nx;
      }
    }
  }
  __syncwarp();
}

// Adds the warp's 32 records to facet f (gridder.h:353-362): into the FP64 accumulator when the
// facet has one, else into the float32 grid.  CONJ lays down conj(CF) (the adjoint of the
// degridder's gather).  sm: the warp's own, its tile zero.  Must be called by all 32 lanes.
// Segments of up to this many records skip the tile (10,800 visibilities of 8 channels on one facet,
// channels up to 12 cells apart, with the window below: 32 us to 22 us).
constexpr int kFewRecords = 2;
// A stripe of bands with no more than this many records each skips it as a whole (64 channels in as many
// bands: 1.36 ms band by band, 1.09 ms so).
constexpr int kFewInBand = 2;

// A run on its way to an FP64 accumulator: averaged blocks' runs are long (0.1 cells a block) and are summed
// in FP64; single visibilities of one support up to 16 have runs of about three, whose sum in FP32 loses
// less than the products' own roundings; those of wide or mixed supports take no runs.
// BANDS: facets may have several bands.
template <int SLOTS, bool CONJ, bool BLOCKS, bool BANDS, int CELLS>
__device__ __forceinline__ void scatter_tile(const GridRecord<1> &rec, const ddfg_facet &f, TileSmem<CELLS> &sm,
                                             int lane) {
  const unsigned tile = smem_addr(sm.tile), recs = smem_addr(sm.rec);
  constexpr int W = CELLS >= 625 ? 25 : 22;  // W x W cells fit
  static_assert(W * W <= CELLS, "tile");
  unsigned mask = __ballot_sync(0xffffffffu, rec.valid);
  const int bx = rec.g.locx - rec.g.sup, by = rec.g.locy - rec.g.sup;
  unsigned other = 0;  // records of another support
  while (mask) {
    // the records of one support and band that the tile covers together
    const int lead = __ffs(mask) - 1;
    const int S = __shfl_sync(0xffffffffu, rec.g.S, lead);
    const int band = BANDS ? __shfl_sync(0xffffffffu, rec.gridchan, lead) : 0;
    const bool like = (mask >> lane & 1) && rec.g.S == S && (!BANDS || rec.gridchan == band);
    unsigned seg = __ballot_sync(0xffffffffu, like);
    bool few = false;
    if (!BLOCKS && !BANDS) {
      other |= seg ^ mask;
    } else if (!BLOCKS && seg != mask) {
      const unsigned same = __ballot_sync(0xffffffffu, (mask >> lane & 1) && rec.g.S == S);
      other |= same ^ mask;
      if (same != seg) {
        const bool in = same >> lane & 1;
        const int bands = __reduce_max_sync(0xffffffffu, in ? rec.gridchan : -1) -
                          __reduce_min_sync(0xffffffffu, in ? rec.gridchan : 0x7fffffff) + 1;
        few = __popc(same) <= kFewInBand * bands;
        if (few) seg = same;
      }
    }
    int x0 = __reduce_min_sync(0xffffffffu, like ? bx : 0x7fffffff);
    int y0 = __reduce_min_sync(0xffffffffu, like ? by : 0x7fffffff);
    int bw = __reduce_max_sync(0xffffffffu, like ? bx : -1) - x0 + S;
    int bh = __reduce_max_sync(0xffffffffu, like ? by : -1) - y0 + S;
    if (!few && bw * bh > CELLS) {
      // not all of them: those in a W x W window that starts a cell behind the first record and
      // opens towards the last one (a baseline's records move one way)
      const int last = 31 - __clz(seg), slack = W - S > 1 ? 1 : 0;
      const int lx = __shfl_sync(0xffffffffu, bx, lead), ly = __shfl_sync(0xffffffffu, by, lead);
      const int xa = __shfl_sync(0xffffffffu, bx, last) >= lx ? lx - slack : lx + slack - (W - S);
      const int ya = __shfl_sync(0xffffffffu, by, last) >= ly ? ly - slack : ly + slack - (W - S);
      const bool in = like && (W < S ? lane == lead : (unsigned)(bx - xa) <= (unsigned)(W - S) &&
                                                          (unsigned)(by - ya) <= (unsigned)(W - S));
      seg = __ballot_sync(0xffffffffu, in);
      x0 = __reduce_min_sync(0xffffffffu, in ? bx : 0x7fffffff);
      y0 = __reduce_min_sync(0xffffffffu, in ? by : 0x7fffffff);
      bw = __reduce_max_sync(0xffffffffu, in ? bx : -1) - x0 + S;
      bh = __reduce_max_sync(0xffffffffu, in ? by : -1) - y0 + S;
    }
    mask &= ~seg;
    const float2 *const cfd = (const float2 *)f.cf_data;
    if (few || bw * bh > CELLS || (!BLOCKS && __popc(seg) <= kFewRecords)) {
      // a support wider than the tile, or too few records to pay for it: tap by tap
      for (; seg; seg &= seg - 1) {
        const int src = __ffs(seg) - 1;
        const float2 *const taps = cfd + __shfl_sync(0xffffffffu, rec.g.cfoff, src);
        const float2 s = make_float2(__shfl_sync(0xffffffffu, rec.stokes[0].x, src),
                                     __shfl_sync(0xffffffffu, rec.stokes[0].y, src));
        const int b = BLOCKS || !BANDS ? band : __shfl_sync(0xffffffffu, rec.gridchan, src);
        const size_t at = ((size_t)(b * f.npol) * f.ny + __shfl_sync(0xffffffffu, by, src)) * f.nx +
                          __shfl_sync(0xffffffffu, bx, src);
        for (int t = lane; t < ((S * S + 31) & ~31); t += 32) {
          const bool on = t < S * S;
          const float2 c = on ? __ldg(taps + t) : czero();
          const float2 v = cmul(s, CONJ ? cconj(c) : c);
          const int sy = tap_row(t, S), cell = sy * f.nx + t - sy * S;
          if (f.grid_acc) red_add_cells_f64((double *)f.grid_acc + 2 * at, on ? cell : -1, v, lane);
          else if (on) red_add((float2 *)f.grid + at + cell, v);
        }
      }
      continue;
    }
    const size_t origin = ((size_t)(band * f.npol) * f.ny + y0) * f.nx + x0;
    const bool f64 = f.grid_acc != nullptr;
    int pitch = bw + ((S - bw) & (f64 ? 7 : 15));
    if (pitch * bh > CELLS) pitch = bw;
    const int n = __popc(seg), n4 = (n + 3) & ~3;
    if ((seg >> lane) & 1) {
      const int at = __popc(seg & ((1u << lane) - 1u));
      const float2 s = rec.stokes[0];
      const int to = (f64 ? 16 : 8) * ((by - y0) * pitch + bx - x0);
      sm.rec[at] = make_int4(to, rec.g.cfoff, __float_as_int(s.x), __float_as_int(s.y));
      if (at == n - 1)  // copies of the last record with a zero value fill the last group of four
        for (int j = n; j < n4; ++j) sm.rec[j] = make_int4(to, rec.g.cfoff, 0, 0);
    }
    __syncwarp();
    unsigned runs =
        __ballot_sync(0xffffffffu, lane > 0 && lane < n && sm.rec[lane].x != sm.rec[lane > 0 ? lane - 1 : 0].x);
    if (!BLOCKS && ((SLOTS > 2 && S > 16) || other) && f64) runs = 0xffffffffu;  // no runs: into the FP64 tile
    const int step = SLOTS == 2 || S <= 8 ? 64 : 32 * SLOTS;
    for (int first = 0; first < S * S; first += step) {
      if (SLOTS == 2 || S <= 8) {
        if (f64) tile_pass<2, CONJ, true, BLOCKS>(tile, recs, n4, runs, S, first, pitch, cfd, lane);
        else tile_pass<2, CONJ, false, false>(tile, recs, n4, runs, S, first, pitch, cfd, lane);
      } else {
        if (f64) tile_pass<SLOTS, CONJ, true, BLOCKS>(tile, recs, n4, runs, S, first, pitch, cfd, lane);
        else tile_pass<SLOTS, CONJ, false, false>(tile, recs, n4, runs, S, first, pitch, cfd, lane);
      }
    }
    tile_to_grid(tile, bw, bh, pitch, f, origin, lane);
  }
}

// ----------------------------------------------------------------------------------------
// Scatter, several Stokes planes: the footprint in registers as a torus
// ----------------------------------------------------------------------------------------
// A tile would need a plane's space four times; the planes share tap loads and addresses, so here
// the registers do the merging.  A lane owns the torus positions t (t < S^2): of any S x S window
// exactly one cell (x, y) has (y mod S) S + (x mod S) = t, so the lane's cell for the next record is
// the same one as long as the window still covers it.  The lane keeps adding into registers and
// reaches memory only when the window leaves its cell: a move by one column costs S additions a
// plane, not S^2.

// x mod S for 0 <= x < 2^26, magic = torus_magic(S).
__device__ __forceinline__ unsigned torus_magic(int S) { return 0xffffffffu / (unsigned)S + 1u; }
__device__ __forceinline__ int torus_mod(int x, int S, unsigned magic) {
  return S > 1 ? x - (int)__umulhi((unsigned)x, magic) * S : 0;
}

// A lane's torus positions of one pass and their place in the current window.
template <int SLOTS>
struct TorusLane {
  int cx[SLOTS], cy[SLOTS];
  bool on[SLOTS];
  int off[SLOTS];   // tap index (row-major in the window) of the position
  int cell[SLOTS];  // its cell index in the grid, -1 for positions past S^2
  __device__ __forceinline__ void set(int S, int first) {
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      const int t = first + 32 * k;
      on[k] = t < S * S;
      const int tt = on[k] ? t : 0;  // idle positions read tap 0 and never reach the grid
      cy[k] = tap_row(tt, S);
      cx[k] = tt - cy[k] * S;
      cell[k] = -1;
      off[k] = 0;
    }
  }
  // Moves the window to the origin with cell index base and (bx mod S, by mod S) = (m & 255, m >> 8).
  __device__ __forceinline__ void move(int base, int m, int S, int nx) {
    const int mx = m & 255, my = m >> 8;
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      const int dx = cx[k] - mx, dy = cy[k] - my;
      const int tx = (int)min((unsigned)dx, (unsigned)(dx + S)), ty = (int)min((unsigned)dy, (unsigned)(dy + S));
      off[k] = ty * S + tx;
      cell[k] = on[k] ? base + ty * nx + tx : -1;
    }
  }
};

template <int NPOL>
struct alignas(16) TorusSmem {
  int4 rec[32];  // cell index of the window's origin, tap table offset, the first Stokes value
  int mod[32];
  float2 st[NPOL > 1 ? NPOL - 1 : 1][32];
};

// One pass of the torus over n records (n a multiple of four) of support S, into the float32 grid.
template <int NPOL, int SLOTS, bool CONJ>
__device__ __forceinline__ void torus_pass(const TorusSmem<NPOL> &sm, int n, int S, int first,
                                           const ddfg_facet &f, size_t origin, int npol_used, int lane) {
  float2 *const grid = (float2 *)f.grid + origin;
  const float2 *const cfd = (const float2 *)f.cf_data;
  const int nx = f.nx;
  const size_t plane = (size_t)f.nx * f.ny;
  TorusLane<SLOTS> tl;
  tl.set(S, first + lane);
  int cell[SLOTS];  // the cells the sums below belong to
  float2 a[NPOL][SLOTS];
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) {
    cell[k] = -1;
#pragma unroll
    for (int p = 0; p < NPOL; ++p) a[p][k] = czero();
  }
  auto flush = [&](int k, int to) {  // slot k's sums to cell `to` (-1: this lane has none to flush)
#pragma unroll
    for (int p = 0; p < NPOL; ++p) {
      if (p >= npol_used) break;
      if (to >= 0) red_add(grid + p * plane + to, a[p][k]);
    }
  };
  int cur = -1, ahead = -1;  // origin of the sums, origin of the records being loaded
  for (int i = 0; i < n; i += 4) {
    int4 q[4];
    float2 c[4][SLOTS];
    int to[4][SLOTS];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      q[r] = sm.rec[i + r];
      if (q[r].x != ahead) {  // the same for all lanes
        ahead = q[r].x;
        tl.move(ahead, sm.mod[i + r], S, nx);
      }
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) {
        to[r][k] = tl.cell[k];
        c[r][k] = __ldg(cfd + (q[r].y + tl.off[k]));
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (q[r].x != cur) {
        cur = q[r].x;
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) {
          const bool leave = to[r][k] != cell[k];
          flush(k, leave ? cell[k] : -1);  // not inside the branch: 1.55 ms instead of 1.25
          if (leave) {
            cell[k] = to[r][k];
#pragma unroll
            for (int p = 0; p < NPOL; ++p) a[p][k] = czero();
          }
        }
      }
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        const float2 v = p == 0 ? make_float2(__int_as_float(q[r].z), __int_as_float(q[r].w)) : sm.st[p > 0 ? p - 1 : 0][i + r];
#pragma unroll
        for (int k = 0; k < SLOTS; ++k)
          a[p][k] = CONJ ? cfma_conj(c[r][k], v, a[p][k]) : cfma(c[r][k], v, a[p][k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < SLOTS; ++k) flush(k, cell[k]);
}

// All passes over n records of support S into the facet's FP64 accumulator, which takes every run by
// itself.  RUN64: the run's FP32 products are summed in FP64.  A record at a time (its successor's taps in
// flight) and out of line: with four at once, as in torus_pass, the additions of eight cells stand in the
// code four times, and the kernel waits for its instructions (four planes, supports up to 23, FP64 runs:
// 15.8 ms, 5.2 ms this way; with both kinds of grid in one loop the float32 one takes 2.47 ms instead of
// 1.25).
template <int NPOL, bool RUN64>
__device__ __noinline__ void torus_acc(const TorusSmem<NPOL> &sm, int n, int S, const ddfg_facet &f, size_t origin,
                                       int npol_used, int lane) {
  using Sum = typename std::conditional<RUN64, double2, float2>::type;
  double *const acc = (double *)f.grid_acc + 2 * origin;
  const float2 *const cfd = (const float2 *)f.cf_data;
  const int nx = f.nx;
  const size_t plane = (size_t)f.nx * f.ny;
  for (int first = 0; first < S * S; first += 64) {
    TorusLane<2> tl;
    tl.set(S, first + lane);
    int cell[2] = {-1, -1}, to[2];
    Sum a[NPOL][2];
    float2 c[2];
    int cur = -1, ahead = -1;
    auto load = [&](int i) {
      const int4 q = sm.rec[i];
      if (q.x != ahead) {  // the same for all lanes
        ahead = q.x;
        tl.move(ahead, sm.mod[i], S, nx);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        to[k] = tl.cell[k];
        c[k] = __ldg(cfd + (q.y + tl.off[k]));
      }
    };
    auto flush = [&]() {
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int other = __shfl_xor_sync(0xffffffffu, cell[k], 1);
        const int ca = lane & 1 ? other : cell[k], cb = lane & 1 ? cell[k] : other;
#pragma unroll
        for (int p = 0; p < NPOL; ++p) {
          if (p >= npol_used) break;
          red_add_pair_f64(acc + 2 * p * plane, ca, cb, a[p][k], lane);
        }
      }
    };
    load(0);
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const int4 q = sm.rec[i];
      const float2 tap[2] = {c[0], c[1]};
      const int at[2] = {to[0], to[1]};
      if (i + 1 < n) load(i + 1);
      if (q.x != cur) {
        if (cur >= 0) flush();
        cur = q.x;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          cell[k] = at[k];
#pragma unroll
          for (int p = 0; p < NPOL; ++p) a[p][k].x = a[p][k].y = 0;
        }
      }
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        const float2 v = p == 0 ? make_float2(__int_as_float(q.z), __int_as_float(q.w)) : sm.st[p > 0 ? p - 1 : 0][i];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if constexpr (RUN64) {
            const float2 t = cmul(tap[k], v);
            a[p][k].x += (double)t.x;
            a[p][k].y += (double)t.y;
          } else {
            a[p][k] = cfma(tap[k], v, a[p][k]);
          }
        }
      }
    }
    flush();
  }
}

// Adds the warp's 32 records to facet f (gridder.h:353-362): into the FP64 accumulator when the
// facet has one, else into the float32 grid.  CONJ lays down conj(CF) (the adjoint of the
// degridder's gather).  sm: the warp's own.  Must be called by all 32 lanes.
template <int NPOL, int SLOTS, bool CONJ, bool BLOCKS, bool ACC>
__device__ __forceinline__ void scatter_torus(const GridRecord<NPOL> &rec, const ddfg_facet &f, int npol_used,
                                              TorusSmem<NPOL> &sm, int lane) {
  unsigned mask = __ballot_sync(0xffffffffu, rec.valid);
  bool mixed = false;  // several supports
  const bool far = far_bands(f);
  while (mask) {
    const int lead = __ffs(mask) - 1, S = __shfl_sync(0xffffffffu, rec.g.S, lead);
    const int band = far ? __shfl_sync(0xffffffffu, rec.gridchan, lead) : 0;
    const size_t origin = (size_t)band * f.npol * f.ny * f.nx;
    const bool mine = rec.valid && rec.g.S == S && (!far || rec.gridchan == band);
    const unsigned sub = __ballot_sync(0xffffffffu, mine);
    mixed = mixed || sub != mask;
    mask &= ~sub;
    const int n = __popc(sub), n4 = (n + 3) & ~3;
    int base = 0, mod = 0, cfo = 0;
    if (mine) {
      const int bx = rec.g.locx - rec.g.sup, by = rec.g.locy - rec.g.sup;
      const unsigned magic = torus_magic(S);
      base = (((rec.gridchan - band) * f.npol) * f.ny + by) * f.nx + bx;
      mod = torus_mod(bx, S, magic) | torus_mod(by, S, magic) << 8;
      cfo = rec.g.cfoff;
      const int at = __popc(sub & ((1u << lane) - 1u));
      sm.rec[at] = make_int4(base, cfo, __float_as_int(rec.stokes[0].x), __float_as_int(rec.stokes[0].y));
      sm.mod[at] = mod;
#pragma unroll
      for (int p = 1; p < NPOL; ++p) sm.st[p > 0 ? p - 1 : 0][at] = rec.stokes[p];
    }
    // up to three copies of the last record with zero values fill the last group of four
    const int last = 31 - __clz(sub);
    base = __shfl_sync(0xffffffffu, base, last);
    cfo = __shfl_sync(0xffffffffu, cfo, last);
    mod = __shfl_sync(0xffffffffu, mod, last);
    if (lane < n4 - n) {
      sm.rec[n + lane] = make_int4(base, cfo, 0, 0);
      sm.mod[n + lane] = mod;
#pragma unroll
      for (int p = 1; p < NPOL; ++p) sm.st[p > 0 ? p - 1 : 0][n + lane] = czero();
    }
    __syncwarp();
    if (ACC && f.grid_acc) {
      if (BLOCKS || S > 16 || mixed) torus_acc<NPOL, true>(sm, n, S, f, origin, npol_used, lane);
      else torus_acc<NPOL, false>(sm, n, S, f, origin, npol_used, lane);
    } else if (SLOTS > 2 && S <= 8) {
      torus_pass<NPOL, 2, CONJ>(sm, n4, S, 0, f, origin, npol_used, lane);
    } else {
      for (int first = 0; first < S * S; first += 32 * SLOTS)
        torus_pass<NPOL, SLOTS, CONJ>(sm, n4, S, first, f, origin, npol_used, lane);
    }
    __syncwarp();
  }
}

template <int NPOL, int SLOTS>
struct ScatterSmem {
  TorusSmem<NPOL> torus;
  __device__ __forceinline__ void clear(int) {}
};
// Tiles of 22 x 22 cells for supports up to 8 (a 7 x 7 footprint's travel of 15 cells), 25 x 25
// for wider ones: two CTAs of eight warps an SM.
template <int SLOTS>
struct ScatterSmem<1, SLOTS> {
  static constexpr int kCells = SLOTS == 2 ? 512 : 640;
  TileSmem<kCells> tile;
  __device__ __forceinline__ void clear(int lane) {
    for (int i = lane; i < kCells; i += 32) tile.tile[i] = make_double2(0., 0.);
    __syncwarp();
  }
};

// The warp's records onto facet f.  sm: the warp's own, cleared once (clear) before the first call.  ACC:
// facets may have FP64 accumulators (several planes only, where that code costs the other path registers).
// BANDS: facets may have several bands (one plane only).
template <int NPOL, int SLOTS, bool CONJ = false, bool BLOCKS = false, bool ACC = !CONJ, bool BANDS = true>
__device__ __forceinline__ void scatter(const GridRecord<NPOL> &rec, const ddfg_facet &f, int npol_used,
                                        ScatterSmem<NPOL, SLOTS> &sm, int lane) {
  if constexpr (NPOL == 1) scatter_tile<SLOTS, CONJ, BLOCKS, BANDS>(rec, f, sm.tile, lane);
  else scatter_torus<NPOL, SLOTS, CONJ, BLOCKS, ACC>(rec, f, npol_used, sm.torus, lane);
}

// ----------------------------------------------------------------------------------------
// Gather
// ----------------------------------------------------------------------------------------
// A run of records with one footprint origin loads its model cells once and keeps them in
// registers; every record costs its tap loads, its products and one partial sum a lane.

template <int NPOL>
struct alignas(16) GatherSmem {
  float2 part[8][32];    // lane partial sums of eight (record, plane) rows
  float2 out[32][NPOL];  // sums
  int2 rec[32];          // cell index of the footprint's origin, tap table offset
};

// The 8 rows of sm.part summed over lanes: four lanes a row, each over eight partials (read so that
// a quarter warp's 16-byte loads fall on distinct banks), then two shuffles.  Lanes 4 j get row j.
__device__ __forceinline__ float2 sum_rows(const float2 (*part)[32], int lane) {
  const int row = lane >> 2, quarter = lane & 3;
  const float4 *p = (const float4 *)&part[row][quarter * 8];
  float2 t = czero();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = p[(i + (quarter >> 1) + 2 * row) & 3];
    t = cadd(t, make_float2(v.x + v.z, v.y + v.w));
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
    t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
  }
  return t;
}

// The lane partials of records i .. i + GROUP - 1 to their rows of sm.part; with the last rows of a
// reduction, their sums to sm.out.
template <int NPOL, int GROUP>
__device__ __forceinline__ void gather_store(GatherSmem<NPOL> &sm, const float2 (*t)[NPOL], int i, int n, int lane) {
  constexpr int ROWS = 8 / NPOL;  // records of one reduction: 8, 4, 2, 2
#pragma unroll
  for (int r = 0; r < GROUP; ++r)
#pragma unroll
    for (int p = 0; p < NPOL; ++p) sm.part[((i + r) % ROWS) * NPOL + p][lane] = t[r][p];
  if ((i + GROUP) % ROWS == 0 || i + GROUP >= n) {
    __syncwarp();
    const float2 v = sum_rows(sm.part, lane);
    const int row = lane >> 2, rec = i / ROWS * ROWS + row / NPOL;
    if ((lane & 3) == 0 && row < ROWS * NPOL && rec < n) sm.out[rec][row % NPOL] = v;
    __syncwarp();
  }
}

// Sums n records (a multiple of four) of support S <= 8: a run's model cells stay in registers.
template <int NPOL>
__device__ __forceinline__ void gather_narrow(GatherSmem<NPOL> &sm, int n, int S, const ddfg_facet &f,
                                              const float2 *grid, int lane) {
  constexpr int GROUP = NPOL == 1 ? 4 : NPOL == 2 ? 4 : 2;  // records in flight
  const size_t plane = (size_t)f.nx * f.ny;
  bool on[2];
  const float2 *cell[2];
  float2 held[NPOL][2], c[GROUP][2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int t = lane + 32 * k, sy = tap_row(t, S);
    on[k] = t < S * S;
    cell[k] = grid + (sy * f.nx + t - sy * S);
#pragma unroll
    for (int p = 0; p < NPOL; ++p) held[p][k] = czero();
#pragma unroll
    for (int r = 0; r < GROUP; ++r) c[r][k] = czero();
  }
  const float2 *const cfd = (const float2 *)f.cf_data + lane;
  int cur = -1;
  for (int i = 0; i < n; i += GROUP) {
    float2 g[GROUP][NPOL][2], t[GROUP][NPOL];
    bool moved[GROUP];
#pragma unroll
    for (int r = 0; r < GROUP; ++r) {
      const int2 q = sm.rec[i + r];
      moved[r] = q.x != cur;  // the same for all lanes
      if (moved[r]) {
        cur = q.x;
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int p = 0; p < NPOL; ++p) g[r][p][k] = on[k] ? __ldg(cell[k] + cur + p * plane) : czero();
      }
      const float2 *p = cfd + q.y;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (on[k]) c[r][k] = __ldg(p + 32 * k);
    }
#pragma unroll
    for (int r = 0; r < GROUP; ++r) {
      if (moved[r]) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int p = 0; p < NPOL; ++p) held[p][k] = g[r][p][k];
      }
#pragma unroll
      for (int p = 0; p < NPOL; ++p) t[r][p] = cfma(c[r][1], held[p][1], cmul(c[r][0], held[p][0]));
    }
    gather_store<NPOL, GROUP>(sm, t, i, n, lane);
  }
}

// The same for any support: four records at a time over all their taps, 32 SLOTS a round, so that a
// record still costs one partial sum a lane.  Records of a round on one origin share its cells.
template <int NPOL, int SLOTS>
__device__ __forceinline__ void gather_wide(GatherSmem<NPOL> &sm, int n, int S, const ddfg_facet &f,
                                            const float2 *grid, int lane) {
  constexpr int GROUP = NPOL <= 2 ? 4 : 2;
  const size_t plane = (size_t)f.nx * f.ny;
  const float2 *const cfd = (const float2 *)f.cf_data + lane;
  const int row0 = tap_row(lane, S), col0 = lane - row0 * S, drow = tap_row(32, S), dcol = 32 - drow * S;
  for (int i = 0; i < n; i += GROUP) {
    int2 q[GROUP];
    float2 t[GROUP][NPOL];
#pragma unroll
    for (int r = 0; r < GROUP; ++r) {
      q[r] = sm.rec[i + r];
#pragma unroll
      for (int p = 0; p < NPOL; ++p) t[r][p] = czero();
    }
    int row = row0, col = col0;
    for (int first = 0; first < S * S; first += 32 * SLOTS) {
      float2 c[GROUP][SLOTS], g[NPOL][SLOTS];
      int at[SLOTS];
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) {
        const bool on = first + 32 * k + lane < S * S;
        at[k] = on ? row * f.nx + col : -1;
        col += dcol;
        row += drow;
        if (col >= S) {
          col -= S;
          ++row;
        }
#pragma unroll
        for (int r = 0; r < GROUP; ++r) c[r][k] = on ? __ldg(cfd + q[r].y + first + 32 * k) : czero();
      }
#pragma unroll
      for (int r = 0; r < GROUP; ++r) {
        if (r == 0 || q[r].x != q[r > 0 ? r - 1 : 0].x) {  // the same for all lanes
#pragma unroll
          for (int k = 0; k < SLOTS; ++k)
#pragma unroll
            for (int p = 0; p < NPOL; ++p) g[p][k] = at[k] >= 0 ? __ldg(grid + q[r].x + at[k] + p * plane) : czero();
        }
#pragma unroll
        for (int p = 0; p < NPOL; ++p)
#pragma unroll
          for (int k = 0; k < SLOTS; ++k) t[r][p] = cfma(c[r][k], g[p][k], t[r][p]);
      }
    }
    gather_store<NPOL, GROUP>(sm, t, i, n, lane);
  }
}

// The sums over every valid record's taps on facet f (degridder.h:202-212); the sum of lane r's
// record ends in its mine[].  sm: the warp's own.  Must be called by all 32 lanes.  FAR: the facet may have
// far_bands (the Stokes I kernels do without: 2 to 3 % of degrid_single_i).
template <int NPOL, int SLOTS, bool FAR = true>
__device__ __forceinline__ void gather(bool valid, const BlockGeom &g, int gridchan, const ddfg_facet &f,
                                       GatherSmem<NPOL> &sm, int lane, float2 *mine) {
#pragma unroll
  for (int p = 0; p < NPOL; ++p) mine[p] = czero();
  unsigned mask = __ballot_sync(0xffffffffu, valid);
  const bool far = FAR && far_bands(f);
  while (mask) {
    const int lead = __ffs(mask) - 1, S = __shfl_sync(0xffffffffu, g.S, lead);
    const int band = far ? __shfl_sync(0xffffffffu, gridchan, lead) : 0;
    const float2 *const grid = (const float2 *)f.grid + (size_t)band * f.npol * f.ny * f.nx;
    const bool own = valid && g.S == S && (!far || gridchan == band);
    const unsigned sub = __ballot_sync(0xffffffffu, own);
    mask &= ~sub;
    const int n = __popc(sub), n4 = (n + 3) & ~3;
    const int at = __popc(sub & ((1u << lane) - 1u));
    if (own) {
      const int2 q = make_int2((((gridchan - band) * f.npol) * f.ny + g.locy - g.sup) * f.nx + g.locx - g.sup,
                               g.cfoff);
      sm.rec[at] = q;
      if (at == n - 1)  // copies of the last record fill the last group of four
        for (int j = n; j < n4; ++j) sm.rec[j] = q;
    }
    __syncwarp();
    if (S <= 8) gather_narrow<NPOL>(sm, n4, S, f, grid, lane);
    else gather_wide<NPOL, SLOTS>(sm, n4, S, f, grid, lane);
    if (own) {
#pragma unroll
      for (int p = 0; p < NPOL; ++p) mine[p] = sm.out[at][p];
    }
    __syncwarp();
  }
}

}  // namespace ddfg
