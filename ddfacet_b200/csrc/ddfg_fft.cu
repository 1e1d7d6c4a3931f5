// Per-facet transforms between grids and images, and stitching into the main image.
//
//  * grid -> dirty facet image: GridToIm (ClassDDEGridMachine.py:1186-1190) is
//    Grid *= OverS^2; fftshift(ifft2(ifftshift(Grid))) * N^2 (ModFFTW.py:584-599), i.e. the
//    unnormalised inverse DFT of the centred grid.  One shift+scale kernel, a batched cuFFT
//    C2C inverse over every (band, pol) plane, one shift kernel back (ddfg_facet_to_image: the
//    same kernel that stitches).
//  * stitching: FacetsToIm_Channel (ClassFacetMachine.py:1331-1416): real part times InvSphe times
//    the facet's spatial weight over (sum of weights x sqrt(sum of Jones)), zero where the taper
//    is below 1e-3, flipped and transposed ([::-1,:].T), cropped with GiveEdges (GiveEdges.py:
//    29-80) and added into the main image; then the main image is divided by the facet norm
//    (:1411-1414).  One fused kernel per facet; facets are added one after the other on the
//    stream, so overlapping padded facets add in a fixed order.
//  * model image -> facet grid: GiveModelTessel(ToGrid=True) (ClassImToGrid.py:138-264): crop
//    the padded facet box, divide by the facet norm, multiply by the spatial weight, divide by
//    the taper (zero where it is below 1e-3), transpose and flip (.T[::-1,:]), scale by
//    (OverS N)^2 and take fftshift(fft2(ifftshift(.))) / N^2 (ModFFTW.py:557-582).  One fused
//    gather+shift kernel, cuFFT forward, one shift+scale kernel.
//
// The facet's 2-D arrays (taper, spatial weight) are [N][N] float32 in the orientation named in
// each entry point.  cuFFT is the only library call; every other pass is a kernel here.
#include <cuda_runtime.h>
#include <cufft.h>

#include "ddfg_common.cuh"
#include "ddfg_internal.h"

struct ddfg_fft_plan {
  cufftHandle h;
  int n, batch;
};

namespace {

// (i + s) mod n for 0 <= i < n, 0 <= s < n
__device__ __forceinline__ int wrap(int i, int s, int n) {
  const int j = i + s;
  return j >= n ? j - n : j;
}

// out[p][y][x] = in[p][(y + s) % n][(x + s) % n] * scale: ifftshift with s = n / 2, fftshift with
// s = n - n / 2.  A block moves one row (blockIdx.x), so the index needs one division a block instead
// of three 64-bit ones an element: 42 MB each way in 35 us before, 13 us now.
__global__ void __launch_bounds__(256) shift_scale_kernel(const float2 *__restrict__ in, float2 *__restrict__ out,
                                                          int n, int s, float scale) {
  const int p = blockIdx.x / n, y = blockIdx.x - p * n;
  const float2 *src = in + ((int64_t)p * n + wrap(y, s, n)) * n;
  float2 *dst = out + (int64_t)blockIdx.x * n;
#pragma unroll 4
  for (int x = threadIdx.x; x < n; x += 256) {
    const float2 v = src[wrap(x, s, n)];
    dst[x] = make_float2(v.x * scale, v.y * scale);
  }
}

struct Edges {
  int x0m, x1m, y0m, y1m, x0f, x1f, y0f, y1f;
};

// GiveEdges(xc, yc, M, n//2, n//2, n) (GiveEdges.py:29-80), no parity argument.
Edges give_edges(int xc, int yc, int m, int n) {
  Edges e;
  const int mx0 = xc - n / 2;
  e.x0m = mx0 > 0 ? mx0 : 0;
  e.x0f = e.x0m - mx0;
  const int mx1 = xc + n / 2;
  int x1m = mx1 < m - 1 ? mx1 : m - 1;
  e.x1f = n - (mx1 - x1m);
  e.x1m = x1m + 1;
  const int my0 = yc - n / 2;
  e.y0m = my0 > 0 ? my0 : 0;
  e.y0f = e.y0m - my0;
  const int my1 = yc + n / 2;
  int y1m = my1 < m - 1 ? my1 : m - 1;
  e.y1f = n - (my1 - y1m);
  e.y1m = y1m + 1;
  return e;
}

// The facet's transposed passes run over 32 x 32 tiles that turn in shared memory, so that both the
// facet's rows and the image's are read and written along their own direction (on two 1625^2 planes:
// shifting and stitching 35 + 53 us to 41 us in one kernel, gathering 57 us to 29 us).
constexpr int kTurn = 32, kTurnRows = 8;  // a block: kTurn x kTurnRows threads

// SumWeights[band][pol] sqrt(SumJonesNorm[band]) of a plane (ClassFacetMachine.py:1066-1076,
// 1385-1391); sumjones [2][nband], NULL or all zero: no Jones normalisation.
__device__ __forceinline__ double plane_weight(const double *sumwt, const double *sumjones, int nband, int npol,
                                               int plane) {
  double w = sumwt[plane];
  if (sumjones) {
    bool any = false;
    for (int i = 0; i < 2 * nband; ++i) any = any || sumjones[i] != 0.;
    if (any) {
      const int band = plane / npol;
      const double den = sumjones[nband + band];
      const double norm = sumjones[band] / (den == 0. ? 1. : den);
      w *= sqrt(norm == 0. ? 1. : norm);
    }
  }
  return w == 0. ? 1. : w;
}

// image[b][p][x0m + a][y0m + c] += Im[n-1-(y0f+c)][x0f+a]
// with Im[r][q] = Re(dirty[b][p][r][q]) * invsphe[r][q] * sw[r][q] / w[b][p], 0 where sphe < 1e-3.
// SHIFT: dirty is first filled from the transform, dirty[r][q] = work[(r - h) mod n][(q - h) mod n]
// (fftshift), all of it.
template <bool SHIFT>
__global__ void __launch_bounds__(256) stitch_kernel(float2 *__restrict__ dirty, const float2 *__restrict__ work,
                                                     int nband, int npol, int n, const float *__restrict__ sphe,
                                                     const float *__restrict__ invsphe, const float *__restrict__ sw,
                                                     const double *__restrict__ sumwt,
                                                     const double *__restrict__ sumjones, float *__restrict__ image,
                                                     int m, Edges e) {
  __shared__ float turn[kTurn][kTurn + 1];
  const int h = n / 2, plane = blockIdx.z, q0 = blockIdx.x * kTurn, r0 = blockIdx.y * kTurn;
  __shared__ double s_w;
  if (threadIdx.x == 0 && threadIdx.y == 0) s_w = plane_weight(sumwt, sumjones, nband, npol, plane);
  __syncthreads();
  const double w = s_w;
  float2 *d = dirty + (int64_t)plane * n * n;
  const int q = q0 + threadIdx.x;
#pragma unroll
  for (int k = threadIdx.y; k < kTurn; k += kTurnRows) {
    const int r = r0 + k;
    if (r >= n || q >= n) continue;
    const int64_t at = (int64_t)r * n + q;
    float2 v;
    if (SHIFT) {
      v = work[(int64_t)plane * n * n + (int64_t)wrap(r, n - h, n) * n + wrap(q, n - h, n)];
      d[at] = v;
    } else {
      v = d[at];
    }
    const float s = sphe[at];
    // numexpr evaluates Im*InvSPhe*SpacialWeigth/weights in float64 (ClassFacetMachine.py:1393-1396)
    turn[threadIdx.x][k] = s < 1e-3f ? 0.f : (float)((double)v.x * (double)invsphe[at] * (double)sw[at] / w);
  }
  __syncthreads();
  // image row a of column q = x0f + a, image column c of row r = n - 1 - (y0f + c)
  const int r = r0 + threadIdx.x, c = n - 1 - r - e.y0f;
  if (r >= n || c < 0 || c >= e.y1m - e.y0m) return;
#pragma unroll
  for (int k = threadIdx.y; k < kTurn; k += kTurnRows) {
    const int a = q0 + k - e.x0f;
    if (a >= 0 && a < e.x1m - e.x0m && q0 + k < n)
      image[plane * (int64_t)m * m + (int64_t)(e.x0m + a) * m + (e.y0m + c)] += turn[k][threadIdx.x];
  }
}

__global__ void __launch_bounds__(256) normalise_kernel(float *image, int planes, int m,
                                                        const float *__restrict__ norm) {
  const int64_t mm = (int64_t)m * m, i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= mm) return;
  const float d = norm[i];
#pragma unroll 4
  for (int p = 0; p < planes; ++p) image[p * mm + i] = image[p * mm + i] / d;
}

// work[p][y][x] = M2[p][(y+h)%n][(x+h)%n] * scale with M2[i][j] = ModelIm[j][n-1-i] and ModelIm
// the normalised crop of the main image (zero outside the GiveEdges box and where sphe < 1e-3).
__global__ void __launch_bounds__(256) model_gather_kernel(const float *__restrict__ image, int m,
                                                           const float *__restrict__ norm, const float *__restrict__ sw,
                                                           const float *__restrict__ sphe, int n, Edges e, float scale,
                                                           float2 *__restrict__ work) {
  __shared__ float turn[kTurn][kTurn + 1];
  const int h = n / 2, plane = blockIdx.z, i0 = blockIdx.x * kTurn, j0 = blockIdx.y * kTurn;
  const int pc = n - 1 - (i0 + threadIdx.x);  // ModelIm[pr][pc]
#pragma unroll
  for (int k = threadIdx.y; k < kTurn; k += kTurnRows) {
    const int pr = j0 + k;
    float v = 0.f;
    if (pr >= e.x0f && pr < e.x1f && pr < n && pc >= 0 && pc >= e.y0f && pc < e.y1f) {
      const float s = sphe[(int64_t)pr * n + pc];
      if (!(s < 1e-3f)) {
        const int64_t mi = (int64_t)(e.x0m + (pr - e.x0f)) * m + (e.y0m + (pc - e.y0f));
        v = image[plane * (int64_t)m * m + mi] / norm[mi] * sw[(int64_t)pr * n + pc] / s;
      }
    }
    turn[threadIdx.x][k] = v;
  }
  __syncthreads();
  const int j = j0 + threadIdx.x;
  if (j >= n) return;
#pragma unroll
  for (int k = threadIdx.y; k < kTurn; k += kTurnRows) {
    const int i = i0 + k;
    if (i < n)
      work[(int64_t)plane * n * n + (int64_t)wrap(i, n - h, n) * n + wrap(j, n - h, n)] =
          make_float2(turn[k][threadIdx.x] * scale, 0.f);
  }
}

// The adjoint of model_gather_kernel with respect to the real image, accumulated:
// grad[p][x0m + a][y0m + c] += scale * Re(work[p][(i - h) mod n][(j - h) mod n]) * coef(pr, pc)
// with pr = x0f + a, pc = y0f + c, (i, j) = (n-1-pc, pr) and coef = sw / sphe / norm (0 where
// sphe < 1e-3): every image pixel of the facet box reads the one grid cell its value went to.
__global__ void model_gather_adjoint_kernel(const float2 *__restrict__ work, int planes, int m,
                                            const float *__restrict__ norm, const float *__restrict__ sw,
                                            const float *__restrict__ sphe, int n, Edges e, float scale,
                                            float *__restrict__ grad) {
  const int h = n / 2;
  const int wa = e.x1m - e.x0m, wb = e.y1m - e.y0m;
  const int64_t per = (int64_t)wa * wb, total = per * planes, nn = (int64_t)n * n;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = idx / per;
    const int64_t k = idx - p * per;
    const int a = (int)(k / wb), c = (int)(k - (int64_t)a * wb);
    const int pr = e.x0f + a, pc = e.y0f + c;
    const float s = sphe[(int64_t)pr * n + pc];
    if (s < 1e-3f) continue;
    const int y = wrap(n - 1 - pc, n - h, n), x = wrap(pr, n - h, n);
    const int64_t mi = (int64_t)(e.x0m + a) * m + (e.y0m + c);
    const float v = work[p * nn + (int64_t)y * n + x].x * scale;
    grad[p * (int64_t)m * m + mi] += v / norm[mi] * sw[(int64_t)pr * n + pc] / s;
  }
}

// One 32 x 32 tile a block over planes of n x n.
dim3 turn_grid(int n, int planes) {
  const unsigned t = (unsigned)((n + kTurn - 1) / kTurn);
  return dim3(t, t, (unsigned)planes);
}
const dim3 kTurnBlock(kTurn, kTurnRows);

int nctas_for(int64_t total) {
  const int64_t b = (total + 255) / 256;
  const int64_t cap = ddfg_num_ctas(8);
  return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}

}  // namespace

extern "C" int ddfg_fft_plan_create(int32_t n, int32_t batch, ddfg_fft_plan **out) {
  if (!out || n <= 0 || batch <= 0) return ddfg_set_error(DDFG_EINVAL, "fft_plan_create: bad argument");
  ddfg_fft_plan *p = new ddfg_fft_plan;
  p->n = n;
  p->batch = batch;
  int dims[2] = {n, n};
  cufftResult r = cufftPlanMany(&p->h, 2, dims, nullptr, 1, n * n, nullptr, 1, n * n, CUFFT_C2C, batch);
  if (r != CUFFT_SUCCESS) {
    delete p;
    return ddfg_set_error(DDFG_ECUDA, "fft_plan_create: cufftPlanMany failed (%d)", (int)r);
  }
  *out = p;
  return DDFG_OK;
}

extern "C" int ddfg_fft_plan_destroy(ddfg_fft_plan *p) {
  if (!p) return DDFG_OK;
  cufftDestroy(p->h);
  delete p;
  return DDFG_OK;
}

extern "C" int ddfg_grid_to_image(ddfg_fft_plan *p, void *grid, double scale, void *work, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!p || !grid || !work) return ddfg_set_error(DDFG_EINVAL, "grid_to_image: null argument");
  const int rows = p->batch * p->n, h = p->n / 2;
  shift_scale_kernel<<<rows, 256, 0, stream>>>((const float2 *)grid, (float2 *)work, p->n, h, (float)scale);
  if (cufftSetStream(p->h, stream) != CUFFT_SUCCESS) return ddfg_set_error(DDFG_ECUDA, "grid_to_image: cufftSetStream");
  if (cufftExecC2C(p->h, (cufftComplex *)work, (cufftComplex *)work, CUFFT_INVERSE) != CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "grid_to_image: cufftExecC2C failed");
  shift_scale_kernel<<<rows, 256, 0, stream>>>((const float2 *)work, (float2 *)grid, p->n, p->n - h, 1.f);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "grid_to_image: %s", cudaGetErrorString(e));
  return DDFG_OK;
}

extern "C" int ddfg_fft_centred(ddfg_fft_plan *p, void *data, int32_t inverse, double scale, void *work,
                                void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!p || !data || !work) return ddfg_set_error(DDFG_EINVAL, "fft_centred: null argument");
  const int rows = p->batch * p->n, h = p->n / 2;
  shift_scale_kernel<<<rows, 256, 0, stream>>>((const float2 *)data, (float2 *)work, p->n, h, 1.f);
  if (cufftSetStream(p->h, stream) != CUFFT_SUCCESS) return ddfg_set_error(DDFG_ECUDA, "fft_centred: cufftSetStream");
  if (cufftExecC2C(p->h, (cufftComplex *)work, (cufftComplex *)work, inverse ? CUFFT_INVERSE : CUFFT_FORWARD) !=
      CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "fft_centred: cufftExecC2C failed");
  shift_scale_kernel<<<rows, 256, 0, stream>>>((const float2 *)work, (float2 *)data, p->n, p->n - h, (float)scale);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "fft_centred: %s", cudaGetErrorString(e));
  return DDFG_OK;
}

extern "C" int ddfg_stitch_facet(const void *dirty, int32_t nband, int32_t npol, int32_t n, const float *sphe,
                                 const float *invsphe, const float *sw_grid, const double *weights, float *image,
                                 int32_t m, int32_t xc, int32_t yc, void *stream_) {
  if (!dirty || !sphe || !invsphe || !sw_grid || !weights || !image || n <= 0 || m <= 0)
    return ddfg_set_error(DDFG_EINVAL, "stitch_facet: bad argument");
  const Edges e = give_edges(xc, yc, m, n);
  if (e.x1m <= e.x0m || e.y1m <= e.y0m) return DDFG_OK;  // facet box outside the image
  stitch_kernel<false><<<turn_grid(n, nband * npol), kTurnBlock, 0, (cudaStream_t)stream_>>>(
      (float2 *)dirty, nullptr, nband, npol, n, sphe, invsphe, sw_grid, weights, nullptr, image, m, e);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "stitch_facet: %s", cudaGetErrorString(err));
  return DDFG_OK;
}

extern "C" int ddfg_facet_to_image(ddfg_fft_plan *p, void *grid, double scale, int32_t nband, int32_t npol,
                                   const float *sphe, const float *invsphe, const float *sw_grid, const double *sumwt,
                                   const double *sumjones, float *image, int32_t m, int32_t xc, int32_t yc, void *work,
                                   void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!p || !grid || !work || !sphe || !invsphe || !sw_grid || !sumwt || !image || m <= 0 || nband <= 0 || npol <= 0)
    return ddfg_set_error(DDFG_EINVAL, "facet_to_image: bad argument");
  if (nband * npol != p->batch)
    return ddfg_set_error(DDFG_EINVAL, "facet_to_image: %d planes, the plan has %d", nband * npol, p->batch);
  const int n = p->n;
  Edges e = give_edges(xc, yc, m, n);
  if (e.x1m <= e.x0m || e.y1m <= e.y0m) e = Edges{};  // facet box outside the image
  shift_scale_kernel<<<p->batch * n, 256, 0, stream>>>((const float2 *)grid, (float2 *)work, n, n / 2, (float)scale);
  if (cufftSetStream(p->h, stream) != CUFFT_SUCCESS) return ddfg_set_error(DDFG_ECUDA, "facet_to_image: cufftSetStream");
  if (cufftExecC2C(p->h, (cufftComplex *)work, (cufftComplex *)work, CUFFT_INVERSE) != CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "facet_to_image: cufftExecC2C failed");
  stitch_kernel<true><<<turn_grid(n, p->batch), kTurnBlock, 0, stream>>>(
      (float2 *)grid, (const float2 *)work, nband, npol, n, sphe, invsphe, sw_grid, sumwt, sumjones, image, m, e);
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "facet_to_image: %s", cudaGetErrorString(err));
  return DDFG_OK;
}

extern "C" int ddfg_image_normalise(float *image, int32_t planes, int32_t m, const float *facet_norm, void *stream_) {
  if (!image || !facet_norm || planes <= 0 || m <= 0) return ddfg_set_error(DDFG_EINVAL, "image_normalise: bad argument");
  normalise_kernel<<<(unsigned)(((int64_t)m * m + 255) / 256), 256, 0, (cudaStream_t)stream_>>>(image, planes, m, facet_norm);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "image_normalise: %s", cudaGetErrorString(err));
  return DDFG_OK;
}

extern "C" int ddfg_image_to_grid(ddfg_fft_plan *p, const float *image, int32_t m, const float *norm_image,
                                  const float *sw_img, const float *sphe, int32_t xc, int32_t yc, double overs,
                                  void *grid_out, void *work, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!p || !image || !norm_image || !sw_img || !sphe || !grid_out || !work || m <= 0)
    return ddfg_set_error(DDFG_EINVAL, "image_to_grid: bad argument");
  const int n = p->n;
  const Edges e = give_edges(xc, yc, m, n);
  const double s = overs * (double)n;
  model_gather_kernel<<<turn_grid(n, p->batch), kTurnBlock, 0, stream>>>(image, m, norm_image, sw_img, sphe, n, e,
                                                                         (float)(s * s), (float2 *)work);
  if (cufftSetStream(p->h, stream) != CUFFT_SUCCESS) return ddfg_set_error(DDFG_ECUDA, "image_to_grid: cufftSetStream");
  if (cufftExecC2C(p->h, (cufftComplex *)work, (cufftComplex *)work, CUFFT_FORWARD) != CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "image_to_grid: cufftExecC2C failed");
  shift_scale_kernel<<<p->batch * n, 256, 0, stream>>>((const float2 *)work, (float2 *)grid_out, n, n - n / 2,
                                                       (float)(1.0 / ((double)n * n)));
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "image_to_grid: %s", cudaGetErrorString(err));
  return DDFG_OK;
}

extern "C" int ddfg_image_to_grid_adjoint(ddfg_fft_plan *p, const void *grid_grad, int32_t m, const float *norm_image,
                                          const float *sw_img, const float *sphe, int32_t xc, int32_t yc,
                                          double overs, float *image_grad, void *work, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (!p || !grid_grad || !norm_image || !sw_img || !sphe || !image_grad || !work || m <= 0)
    return ddfg_set_error(DDFG_EINVAL, "image_to_grid_adjoint: bad argument");
  const int n = p->n;
  const Edges e = give_edges(xc, yc, m, n);
  if (e.x1m <= e.x0m || e.y1m <= e.y0m) return DDFG_OK;  // facet box outside the image
  // adjoint of (fftshift, times 1/N^2): ifftshift, times 1/N^2
  shift_scale_kernel<<<p->batch * n, 256, 0, stream>>>((const float2 *)grid_grad, (float2 *)work, n, n / 2,
                                                       (float)(1.0 / ((double)n * n)));
  if (cufftSetStream(p->h, stream) != CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "image_to_grid_adjoint: cufftSetStream");
  // adjoint of the unnormalised forward DFT: the unnormalised inverse DFT
  if (cufftExecC2C(p->h, (cufftComplex *)work, (cufftComplex *)work, CUFFT_INVERSE) != CUFFT_SUCCESS)
    return ddfg_set_error(DDFG_ECUDA, "image_to_grid_adjoint: cufftExecC2C failed");
  const double s = overs * (double)n;
  const int64_t pix = (int64_t)(e.x1m - e.x0m) * (e.y1m - e.y0m) * p->batch;
  model_gather_adjoint_kernel<<<nctas_for(pix), 256, 0, stream>>>((const float2 *)work, p->batch, m, norm_image,
                                                                    sw_img, sphe, n, e, (float)(s * s), image_grad);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return ddfg_set_error(DDFG_ECUDA, "image_to_grid_adjoint: %s", cudaGetErrorString(err));
  return DDFG_OK;
}
