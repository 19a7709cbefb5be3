// Uniform weighting on the GPU.
//
// Reference behaviour:
//   grid_weight_to_griddata   processing_components/griddata/gridding.py:161-183
//   griddata_reweight         processing_components/griddata/gridding.py:213-230
//   weight_visibility         processing_components/imaging/weighting.py:19-40
//
// grid_weight_to_griddata adds each row's imaging weight (one value per
// polarisation) to its nearest grid cell grid[chan, :, pwg, pv, pu] and to
// sumwt[chan, :]; griddata_reweight then divides each row's weights by the
// real part of that cell when every polarisation's cell is non-zero.  The
// weight grid is real FP64 here (ARL keeps it in the real part of a complex
// grid); the row weights keep the precision of the path.
#include "common.cuh"
#include "dsmath.cuh"
#include "mapping.cuh"

namespace arlgpu {

void count_launch(unsigned n);

// Nearest-cell mapping of one row.  ARL's convolution_mapping asserts that
// the pixel, the w-plane, the cf plane and the channel are in range; the
// sub-pixel index is not used here.  The pixels and planes come from the plan's
// fixed-point decisions where those hold, else from map_raw: both give NumPy's
// indices, and the second takes about 40 FP64 operations at GB300's 2 a clock and SM.
__device__ __forceinline__ bool map_cell(double u, double v, double w, double f, const Geom &g, int *ch,
                                         int64_t *cell0) {
  int pu, pv, uf, vf, zg, zc, c;
  if (map_fixed(u, v, w, f, g, &pu, &pv, &uf, &vf, &zg, &zc, &c)) {
    if (pu < 0 || pu >= g.nx || pv < 0 || pv >= g.ny || zg < 0 || zc < 0 || c < 0) return false;
  } else {
    const RawMap m = map_raw(u, v, w, f, g);
    if (!(m.pu >= 0.0 && m.pu < g.nx && m.pv >= 0.0 && m.pv < g.ny && m.zg >= 0.0 && m.zg < g.nw && m.zc >= 0.0 &&
          m.zc < g.nz && m.ch >= 0.0 && m.ch < g.nchan && m.ch < g.cf_nchan))
      return false;
    pu = (int)m.pu;
    pv = (int)m.pv;
    zg = (int)m.zg;
    c = (int)m.ch;
  }
  *ch = c;
  // cell of polarisation 0; polarisation p is p * nw * ny * nx further
  *cell0 = (((int64_t)c * g.npol) * g.nw + zg) * g.ny * g.nx + (int64_t)pv * g.nx + pu;
  return true;
}

// K10a: weights onto the weight grid, and sumwt.  An FP64 addition to shared
// memory is a compare-and-swap loop, and the rows of a block all add to the few
// words of [nchan][npol]: each thread therefore sums in registers while its rows
// stay in one channel (every row of a one-channel image; the rows a thread
// takes lie a multiple of 2^13 apart, so with a power-of-two number of
// channels in row order too) and adds the sum when the channel changes and at
// the end, there after a sum over the warp when all its lanes hold one channel.
// Bound by the L2 atomics of the grid (35 to 75 G a second, measured).
// 10.05 M rows, one polarisation, 4096^2: 3161 -> 177 us.
template <typename W, int NPOL>
__global__ void __launch_bounds__(256)
k_grid_weight(const double *__restrict__ uvw, const double *__restrict__ freq, const W *__restrict__ wt, int64_t nvis,
              Geom g, double *__restrict__ wgrid, double *__restrict__ sumwt, unsigned long long *__restrict__ nbad,
              int shared_sum) {
  extern __shared__ double s_sum[];
  const int npol = NPOL ? NPOL : g.npol;
  const int nsum = g.nchan * npol;
  if (shared_sum) {
    for (int k = threadIdx.x; k < nsum; k += blockDim.x) s_sum[k] = 0.0;
    __syncthreads();
  }
  double *sums = shared_sum ? s_sum : sumwt;
  const int64_t pstride = (int64_t)g.nw * g.ny * g.nx;
  double acc[NPOL ? NPOL : 1];
#pragma unroll
  for (int p = 0; p < NPOL; ++p) acc[p] = 0.0;
  int cur = -1;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nvis; r += (int64_t)gridDim.x * blockDim.x) {
    int ch;
    int64_t c0;
    if (!map_cell(uvw[3 * r], uvw[3 * r + 1], uvw[3 * r + 2], freq[r], g, &ch, &c0)) {
      atomicAdd(nbad, 1ull);
      continue;
    }
    if (NPOL) {
      if (ch != cur) {
        if (cur >= 0)
#pragma unroll
          for (int p = 0; p < NPOL; ++p) {
            atomicAdd(&sums[cur * NPOL + p], acc[p]);
            acc[p] = 0.0;
          }
        cur = ch;
      }
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        const double w = (double)wt[r * NPOL + p];
        atomicAdd(&wgrid[c0 + p * pstride], w);
        acc[p] += w;
      }
    } else {
      for (int p = 0; p < npol; ++p) {
        const double w = (double)wt[r * npol + p];
        atomicAdd(&wgrid[c0 + p * pstride], w);
        atomicAdd(&sums[ch * npol + p], w);
      }
    }
  }
  if (NPOL) {
    const int lane = threadIdx.x & 31;
    const int c0 = __reduce_max_sync(0xffffffffu, cur);  // -1: no row in the warp
    if (c0 >= 0 && __all_sync(0xffffffffu, cur == c0 || cur < 0)) {
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        double t = acc[p];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) atomicAdd(&sums[c0 * NPOL + p], t);
      }
    } else if (cur >= 0) {
#pragma unroll
      for (int p = 0; p < NPOL; ++p) atomicAdd(&sums[cur * NPOL + p], acc[p]);
    }
  }
  if (shared_sum) {
    __syncthreads();
    for (int k = threadIdx.x; k < nsum; k += blockDim.x)
      if (s_sum[k] != 0.0) atomicAdd(&sumwt[k], s_sum[k]);
  }
}

// w / sum.  An FP64 division takes the FP64 unit 9 operations' time; a
// FP32 weight's quotient comes from a double-single one instead (46 bits before
// its one rounding to FP32) when the sum's magnitude leaves room for the
// low parts.  Where it lies within 1e-4 of half an ulp of a rounding boundary,
// so that those bits might not decide it (Ziv's test: the sum with the low part
// enlarged rounds otherwise), the division does: the result is always the FP64
// quotient's.
__device__ __forceinline__ double divide(double w, double sum) { return w / sum; }
__device__ __forceinline__ float divide(float w, double sum) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(sum);
  const int e = (int)(b >> 52) & 0x7ff;
  // weights from 1e-14 on: a quotient's low part stays a normal FP32 number, or its spacing below 1e-5 of its half ulp
  if (e < 1023 - 60 || e > 1023 + 60 || !(w == 0.f || (fabsf(w) > 1e-14f && fabsf(w) < 1e18f)))
    return (float)((double)w / sum);
  // sum as hi + lo from its bits: 24 leading bits, then the other 29
  const float hi = __uint_as_float((unsigned)((b >> 63) << 31) | (unsigned)(e - 1023 + 127) << 23 |
                                   ((unsigned)(b >> 29) & 0x7fffffu));
  if (w == 0.f) return __fdiv_rn(w, hi);  // a flagged row's zero keeps its sign
  const float unit = __uint_as_float((unsigned)((b >> 63) << 31) | (unsigned)(e - 1023 + 127 - 52) << 23);
  const dsf q = ds_div({w, 0.f}, quick_two_sum(hi, (float)((unsigned)b & 0x1fffffffu) * unit));
  if (__fadd_rn(q.hi, __fmul_rn(q.lo, 1.0001f)) != q.hi) return (float)((double)w / sum);
  return q.hi;
}

// K10b: each row's weights divided by its cells when all are non-zero.
// 10.05 M rows, one polarisation, 4096^2: 1249 -> 204 us.
template <typename W>
__global__ void __launch_bounds__(256)
k_reweight(const double *__restrict__ uvw, const double *__restrict__ freq, W *__restrict__ wt, int64_t nvis, Geom g,
           const double *__restrict__ wgrid) {
  const int64_t pstride = (int64_t)g.nw * g.ny * g.nx;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nvis; r += (int64_t)gridDim.x * blockDim.x) {
    int ch;
    int64_t c0;
    if (!map_cell(uvw[3 * r], uvw[3 * r + 1], uvw[3 * r + 2], freq[r], g, &ch, &c0)) continue;
    bool all = true;
    for (int p = 0; p < g.npol; ++p) all = all && wgrid[c0 + p * pstride] != 0.0;
    if (!all) continue;
    for (int p = 0; p < g.npol; ++p) wt[r * g.npol + p] = divide(wt[r * g.npol + p], wgrid[c0 + p * pstride]);
  }
}

static int blocks_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 152 * 32 ? 152 * 32 : b));
}

template <typename W>
static void launch_grid_weight(const double *uvw, const double *freq, const W *wt, int64_t nvis, const Geom &g,
                               double *wgrid, double *sumwt, unsigned long long *nb, int shared_sum, size_t smem,
                               cudaStream_t st) {
  const int blocks = blocks_for(nvis);
  switch (g.npol) {
    case 1: k_grid_weight<W, 1><<<blocks, 256, smem, st>>>(uvw, freq, wt, nvis, g, wgrid, sumwt, nb, shared_sum); break;
    case 2: k_grid_weight<W, 2><<<blocks, 256, smem, st>>>(uvw, freq, wt, nvis, g, wgrid, sumwt, nb, shared_sum); break;
    case 4: k_grid_weight<W, 4><<<blocks, 256, smem, st>>>(uvw, freq, wt, nvis, g, wgrid, sumwt, nb, shared_sum); break;
    default: k_grid_weight<W, 0><<<blocks, 256, smem, st>>>(uvw, freq, wt, nvis, g, wgrid, sumwt, nb, shared_sum);
  }
}

}  // namespace arlgpu

using namespace arlgpu;

extern "C" int arlgpu_grid_weights(const double *uvw, const double *frequency, const void *weight, int64_t nvis,
                                   int precision, const arlgpu_cf_desc *cd, double *wgrid, const arlgpu_grid_desc *gd,
                                   double *sumwt, int64_t *n_bad_dev, void *stream) {
  Geom g;
  ARL_TRY(make_geom(gd, cd, precision, nvis, &g));
  if (nvis < 0) return fail(ARLGPU_ERR_INVALID, "nvis < 0");
  if (!wgrid || !sumwt || !n_bad_dev || (nvis > 0 && (!uvw || !frequency || !weight)))
    return fail(ARLGPU_ERR_INVALID, "null array argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const size_t cells = (size_t)g.nchan * g.npol * g.nw * g.ny * g.nx;
  ARL_CUDA(cudaMemsetAsync(wgrid, 0, cells * sizeof(double), st));
  ARL_CUDA(cudaMemsetAsync(sumwt, 0, (size_t)g.nchan * g.npol * sizeof(double), st));
  ARL_CUDA(cudaMemsetAsync(n_bad_dev, 0, sizeof(int64_t), st));
  if (nvis == 0) return ARLGPU_OK;
  const int nsum = g.nchan * g.npol;
  const int shared_sum = nsum <= 4096;
  const size_t smem = shared_sum ? (size_t)nsum * sizeof(double) : 0;
  unsigned long long *nb = reinterpret_cast<unsigned long long *>(n_bad_dev);
  if (precision == ARLGPU_FP64)
    launch_grid_weight(uvw, frequency, static_cast<const double *>(weight), nvis, g, wgrid, sumwt, nb, shared_sum,
                       smem, st);
  else
    launch_grid_weight(uvw, frequency, static_cast<const float *>(weight), nvis, g, wgrid, sumwt, nb, shared_sum,
                       smem, st);
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

extern "C" int arlgpu_reweight(const double *uvw, const double *frequency, void *weight, int64_t nvis, int precision,
                               const arlgpu_cf_desc *cd, const double *wgrid, const arlgpu_grid_desc *gd,
                               void *stream) {
  Geom g;
  ARL_TRY(make_geom(gd, cd, precision, nvis, &g));
  if (nvis < 0) return fail(ARLGPU_ERR_INVALID, "nvis < 0");
  if (nvis == 0) return ARLGPU_OK;
  if (!uvw || !frequency || !weight || !wgrid) return fail(ARLGPU_ERR_INVALID, "null array argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == ARLGPU_FP64)
    k_reweight<double><<<blocks_for(nvis), 256, 0, st>>>(uvw, frequency, static_cast<double *>(weight), nvis, g,
                                                          wgrid);
  else
    k_reweight<float><<<blocks_for(nvis), 256, 0, st>>>(uvw, frequency, static_cast<float *>(weight), nvis, g,
                                                         wgrid);
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}
