// Row-wise visibility operators on the path (K10, K11).
//
// Reference behaviour:
//   phaserotate_visibility (tangent=True)   processing_components/visibility/base.py:295-334
//   simulate_point                          processing_library/util/coordinate_support.py:192-212
//   apply_gaintable, scalar gains           processing_components/calibration/operations.py:79-164 (:134-137)
#include "common.cuh"
#include "dsmath.cuh"

namespace arlgpu {

void count_launch(unsigned n);

// vis *= exp(-2 pi i s.uvw) (inverse) or its conjugate; s = (l, m, n - 1).
template <typename CT>
__global__ void k_phaserotate(CT *vis, const double *uvw, int64_t nvis, int npol, double l, double m, double n1,
                              int inverse) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nvis; r += (int64_t)gridDim.x * blockDim.x) {
    const double ph = -2.0 * M_PI * (uvw[3 * r] * l + uvw[3 * r + 1] * m + uvw[3 * r + 2] * n1);
    double s, c;
    sincos(ph, &s, &c);
    if (!inverse) s = -s;
    for (int p = 0; p < npol; ++p) {
      CT v = vis[r * npol + p];
      const double re = (double)v.x * c - (double)v.y * s, im = (double)v.x * s + (double)v.y * c;
      v.x = re;
      v.y = im;
      vis[r * npol + p] = v;
    }
  }
}

// Row of baseline (a1, a2), stored at [a2, a1]: V *= g[a2] conj(g[a1]).
// inverse uses 1/g where |g| > 0 and 1 elsewhere (operations.py:128-131).
template <typename CT>
__global__ void k_gains(CT *vis, int64_t nvis, int npol, const int32_t *a1, const int32_t *a2, const double2 *g,
                        int inverse) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nvis; r += (int64_t)gridDim.x * blockDim.x) {
    double2 ga = g[a2[r]], gb = g[a1[r]];
    if (inverse) {
      double na = ga.x * ga.x + ga.y * ga.y, nb = gb.x * gb.x + gb.y * gb.y;
      ga = na > 0.0 ? make_double2(ga.x / na, -ga.y / na) : make_double2(1.0, 0.0);
      gb = nb > 0.0 ? make_double2(gb.x / nb, -gb.y / nb) : make_double2(1.0, 0.0);
    }
    // m = ga * conj(gb)
    const double mr = ga.x * gb.x + ga.y * gb.y, mi = ga.y * gb.x - ga.x * gb.y;
    for (int p = 0; p < npol; ++p) {
      CT v = vis[r * npol + p];
      const double re = (double)v.x * mr - (double)v.y * mi, im = (double)v.x * mi + (double)v.y * mr;
      v.x = re;
      v.y = im;
      vis[r * npol + p] = v;
    }
  }
}

// chi^2 = sum_r,p w |Vobs - g[a2] conj(g[a1]) M|^2 and its conjugate-Wirtinger
// derivatives (row of baseline (a1, a2) stored at [a2, a1], the convention of
// apply_gaintable, calibration/operations.py:134-137): with R = Vobs - g2 conj(g1) M
// and Q = w R conj(M),
//   d/d conj(M)     = -w conj(g2) g1 R
//   d/d conj(g[a2]) = -g1 sum Q            (over rows and pols)
//   d/d conj(g[a1]) = -g2 conj(sum Q)
// Bound by the FP64 unit (2 operations a clock and SM), so the row's work is
// kept to 14 multiply-adds: a thread takes ROWS consecutive rows, forms the
// gain product once per run of one baseline (the channels of a time, in the
// usual row order) and sums Q over the run, and the two gain derivatives follow
// from the run's sum.  The a1 derivative is summed while a1 stays and then, when
// a warp's lanes all end on one a1 (baselines are ordered by a1), over the warp:
// an FP64 addition to shared memory is a compare-and-swap loop that 32 lanes on
// one word would run 32 times over.
// 15.6 M rows, 128 antennas, 8 channels: 3882 -> 790 us.
// ROWS is 8 where that gives more than every second SM a block, 4 down to 64 Ki rows,
// and 1 below, where few rows a thread keep its chain of waits short.  8 / 4 / 1 rows, us, 64
// antennas: 3,000 rows of one channel 33 / 21 / 16 (in random order 38 / 23 / 12),
// 100,000 rows 34 / 23 / 32 (39 / 25 / 27), 300,000 rows 35 / 40 / 66 (40 / 42 / 42).
template <typename CT> struct ChiPair { using T = double4; };
template <> struct ChiPair<float2> { using T = float4; };

template <typename CT, int NPOL, int ROWS>
__global__ void __launch_bounds__(256)
k_gain_chi2(const CT *__restrict__ vobs, const CT *__restrict__ m, const double *__restrict__ wt, int64_t nvis,
            int npol_arg, const int32_t *__restrict__ a1, const int32_t *__restrict__ a2,
            const double2 *__restrict__ g, int nant, double *__restrict__ chi2, CT *__restrict__ grad_m,
            double2 *__restrict__ grad_g, int pairs) {
  extern __shared__ double sg[];  // 2 * nant: re, im of the per-antenna sums
  for (int i = threadIdx.x; i < 2 * nant; i += blockDim.x) sg[i] = 0.0;
  __syncthreads();
  const int npol = NPOL ? NPOL : npol_arg, lane = threadIdx.x & 31;
  const int64_t nrun = (nvis + ROWS - 1) / ROWS;
  // whole warps loop together: the flush at the end of a run is a warp's
  const int64_t first = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~(int64_t)31;
  double local = 0.0;
  for (int64_t w0 = first; w0 < nrun; w0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t rb = (w0 + lane) * ROWS, re = min(rb + ROWS, nvis);
    int c1 = -1, c2 = -1;
    double2 g1{}, g2{};
    double gr = 0.0, gi = 0.0, qx = 0.0, qy = 0.0, dx = 0.0, dy = 0.0;
    auto end_pair = [&]() {  // the baseline's sum into both antennas
      if (grad_g && c2 >= 0) {
        atomicAdd(&sg[2 * c2], -(qx * g1.x - qy * g1.y));
        atomicAdd(&sg[2 * c2 + 1], -(qx * g1.y + qy * g1.x));
        dx -= qx * g2.x + qy * g2.y;
        dy -= qx * g2.y - qy * g2.x;
      }
      qx = qy = 0.0;
    };
    auto row = [&](int64_t k, CT vo, CT mo, CT *go) {
      const double mr = widen(mo.x), mi = widen(mo.y);
      const double rr = fma(-gr, mr, fma(gi, mi, widen(vo.x))), ri = fma(-gr, mi, fma(-gi, mr, widen(vo.y)));
      double sr = rr, si = ri;  // w R
      if (wt) {
        const double w = wt[k];
        sr *= w;
        si *= w;
      }
      local = fma(sr, rr, fma(si, ri, local));
      if (grad_m) {
        narrow(-fma(gr, sr, gi * si), &go->x);
        narrow(fma(gi, sr, -(gr * si)), &go->y);
      }
      qx = fma(sr, mr, fma(si, mi, qx));
      qy = fma(si, mr, fma(-sr, mi, qy));
    };
    auto pair = [&](int i1, int i2) {
      if (i1 == c1 && i2 == c2) return;
      end_pair();
      if (i1 != c1) {
        if (grad_g && c1 >= 0) {
          atomicAdd(&sg[2 * c1], dx);
          atomicAdd(&sg[2 * c1 + 1], dy);
        }
        dx = dy = 0.0;
        g1 = g[i1];
      }
      if (i2 != c2) g2 = g[i2];
      c1 = i1;
      c2 = i2;
      gr = g2.x * g1.x + g2.y * g1.y;  // g2 conj(g1)
      gi = g2.y * g1.x - g2.x * g1.y;
    };
    if (NPOL == 1 && ROWS % 2 == 0 && pairs && rb + ROWS <= nvis) {
      using P = typename ChiPair<CT>::T;
#pragma unroll
      for (int j = 0; j < ROWS; j += 2) {
        const int2 i1 = *reinterpret_cast<const int2 *>(a1 + rb + j), i2 = *reinterpret_cast<const int2 *>(a2 + rb + j);
        const P vo = *reinterpret_cast<const P *>(vobs + rb + j), mo = *reinterpret_cast<const P *>(m + rb + j);
        CT g0{}, g1o{};
        pair(i1.x, i2.x);
        row(rb + j, CT{vo.x, vo.y}, CT{mo.x, mo.y}, &g0);
        pair(i1.y, i2.y);
        row(rb + j + 1, CT{vo.z, vo.w}, CT{mo.z, mo.w}, &g1o);
        if (grad_m) *reinterpret_cast<P *>(grad_m + rb + j) = P{g0.x, g0.y, g1o.x, g1o.y};
      }
    } else {
      for (int64_t r = rb; r < re; ++r) {
        pair(a1[r], a2[r]);
        for (int p = 0; p < npol; ++p) {
          const int64_t k = r * npol + p;
          CT o{};
          row(k, vobs[k], m[k], &o);
          if (grad_m) grad_m[k] = o;
        }
      }
    }
    end_pair();
    if (grad_g) {
      const int top = __reduce_max_sync(0xffffffffu, c1);  // -1: a lane past the last row
      if (__all_sync(0xffffffffu, c1 == top || c1 < 0)) {
        for (int o = 16; o > 0; o >>= 1) {
          dx += __shfl_xor_sync(0xffffffffu, dx, o);
          dy += __shfl_xor_sync(0xffffffffu, dy, o);
        }
        if (lane == 0) {
          atomicAdd(&sg[2 * top], dx);
          atomicAdd(&sg[2 * top + 1], dy);
        }
      } else if (c1 >= 0) {
        atomicAdd(&sg[2 * c1], dx);
        atomicAdd(&sg[2 * c1 + 1], dy);
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if (lane == 0) atomicAdd(chi2, local);
  __syncthreads();
  if (grad_g)
    for (int i = threadIdx.x; i < nant; i += blockDim.x)
      if (sg[2 * i] != 0.0 || sg[2 * i + 1] != 0.0) {
        atomicAdd(&grad_g[i].x, sg[2 * i]);
        atomicAdd(&grad_g[i].y, sg[2 * i + 1]);
      }
}

template <typename CT, int ROWS>
static void launch_gain_chi2_rows(const CT *vo, const CT *mo, const double *wt, int64_t nvis, int npol,
                                  const int32_t *a1, const int32_t *a2, const double2 *g, int nant, double *chi2,
                                  CT *gm, double2 *grad_g, int pairs, cudaStream_t st) {
  const int64_t want = ((nvis + ROWS - 1) / ROWS + 255) / 256;
  const int blocks = (int)(want < 152 * 4 ? want : 152 * 4);
  const size_t smem = 2 * sizeof(double) * nant;
  if (npol == 1)
    k_gain_chi2<CT, 1, ROWS><<<blocks, 256, smem, st>>>(vo, mo, wt, nvis, npol, a1, a2, g, nant, chi2, gm, grad_g, pairs);
  else
    k_gain_chi2<CT, 0, ROWS><<<blocks, 256, smem, st>>>(vo, mo, wt, nvis, npol, a1, a2, g, nant, chi2, gm, grad_g, pairs);
}

template <typename CT>
static void launch_gain_chi2(const void *vobs, const void *model, const double *wt, int64_t nvis, int npol,
                             const int32_t *a1, const int32_t *a2, const double2 *g, int nant, double *chi2,
                             void *grad_m, double2 *grad_g, cudaStream_t st) {
  // two rows in one 16-byte access: the arrays' first elements decide, rows are taken an even number at a time
  auto at = [](const void *p, uintptr_t n) { return ((uintptr_t)p & (n - 1)) == 0; };
  const int pairs = sizeof(CT) == 8 && at(vobs, 16) && at(model, 16) && at(grad_m, 16) && at(a1, 8) && at(a2, 8);
  const CT *vo = static_cast<const CT *>(vobs), *mo = static_cast<const CT *>(model);
  CT *gm = static_cast<CT *>(grad_m);
  auto launch = nvis < 65536 ? launch_gain_chi2_rows<CT, 1>
                             : nvis <= 4 * 152 * 256 ? launch_gain_chi2_rows<CT, 4> : launch_gain_chi2_rows<CT, 8>;
  launch(vo, mo, wt, nvis, npol, a1, a2, g, nant, chi2, gm, grad_g, pairs, st);
}

// apply_gaintable with scalar gains on a BlockVisibility (one polarisation):
// cell [t][i][j][c] of the block, for a time t with a gain-table row
// k = time_row[t] >= 0, becomes V * g[k][i][c] conj(g[k][j][c]), where g is the
// gain or, for the inverse, 1/gain where |gain| > 0 and 1 elsewhere
// (operations.py:124-137); the cell is zeroed where the product of the two
// antennas' gain weights is 0 (:138-140).  Times with time_row[t] < 0 are
// left as they are.
template <typename CT>
__global__ void k_gaintable(CT *vis, int ntimes, int nant, int nchan, const int32_t *__restrict__ time_row,
                            const double2 *__restrict__ g, const double *__restrict__ gw, int inverse) {
  const int64_t ncell = (int64_t)ntimes * nant * nant * nchan;
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < ncell; q += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(q % nchan);
    int64_t r = q / nchan;
    const int j = (int)(r % nant);
    r /= nant;
    const int i = (int)(r % nant);
    const int t = (int)(r / nant);
    const int k = time_row[t];
    if (k < 0) continue;
    const int64_t gi = ((int64_t)k * nant + i) * nchan + c, gj = ((int64_t)k * nant + j) * nchan + c;
    double2 ga = g[gi], gb = g[gj];
    if (inverse) {
      const double na = ga.x * ga.x + ga.y * ga.y, nb = gb.x * gb.x + gb.y * gb.y;
      ga = na > 0.0 ? make_double2(ga.x / na, -ga.y / na) : make_double2(1.0, 0.0);
      gb = nb > 0.0 ? make_double2(gb.x / nb, -gb.y / nb) : make_double2(1.0, 0.0);
    }
    CT v = vis[q];
    if (gw[gi] * gw[gj] == 0.0) {
      v.x = 0;
      v.y = 0;
    } else {
      // m = ga conj(gb), then V m
      const double mr = ga.x * gb.x + ga.y * gb.y, mi = ga.y * gb.x - ga.x * gb.y;
      const double re = (double)v.x * mr - (double)v.y * mi, im = (double)v.x * mi + (double)v.y * mr;
      v.x = re;
      v.y = im;
    }
    vis[q] = v;
  }
}

static int nblk(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 152 * 32 ? 152 * 32 : b));
}

}  // namespace arlgpu

using namespace arlgpu;

extern "C" int arlgpu_phaserotate(void *vis, const double *uvw, int64_t nvis, int32_t npol, int precision, double l,
                                  double m, int inverse, void *stream) {
  if (nvis < 0 || npol < 1 || (nvis > 0 && (!vis || !uvw))) return fail(ARLGPU_ERR_INVALID, "bad arguments");
  if (nvis == 0) return ARLGPU_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const double n1 = sqrt(1.0 - l * l - m * m) - 1.0;
  if (precision == ARLGPU_FP64)
    k_phaserotate<double2><<<nblk(nvis), 256, 0, st>>>(static_cast<double2 *>(vis), uvw, nvis, npol, l, m, n1, inverse);
  else if (precision == ARLGPU_FP32C)
    k_phaserotate<float2><<<nblk(nvis), 256, 0, st>>>(static_cast<float2 *>(vis), uvw, nvis, npol, l, m, n1, inverse);
  else
    return fail(ARLGPU_ERR_INVALID, "bad precision");
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

extern "C" int arlgpu_apply_gains(void *vis, int64_t nvis, int32_t npol, int precision, const int32_t *a1,
                                  const int32_t *a2, const void *gains, int inverse, void *stream) {
  if (nvis < 0 || npol < 1 || (nvis > 0 && (!vis || !a1 || !a2 || !gains))) return fail(ARLGPU_ERR_INVALID, "bad arguments");
  if (nvis == 0) return ARLGPU_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const double2 *g = static_cast<const double2 *>(gains);
  if (precision == ARLGPU_FP64)
    k_gains<double2><<<nblk(nvis), 256, 0, st>>>(static_cast<double2 *>(vis), nvis, npol, a1, a2, g, inverse);
  else if (precision == ARLGPU_FP32C)
    k_gains<float2><<<nblk(nvis), 256, 0, st>>>(static_cast<float2 *>(vis), nvis, npol, a1, a2, g, inverse);
  else
    return fail(ARLGPU_ERR_INVALID, "bad precision");
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

extern "C" int arlgpu_apply_gaintable(void *vis, int32_t ntimes, int32_t nants, int32_t nchan, int precision,
                                      const int32_t *time_row, const void *gain, const double *gain_weight,
                                      int inverse, void *stream) {
  if (ntimes < 0 || nants < 1 || nchan < 1) return fail(ARLGPU_ERR_INVALID, "bad block shape");
  const int64_t ncell = (int64_t)ntimes * nants * nants * nchan;
  if (ncell == 0) return ARLGPU_OK;
  if (!vis || !time_row || !gain || !gain_weight) return fail(ARLGPU_ERR_INVALID, "null array argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const double2 *g = static_cast<const double2 *>(gain);
  if (precision == ARLGPU_FP64)
    k_gaintable<double2><<<nblk(ncell), 256, 0, st>>>(static_cast<double2 *>(vis), ntimes, nants, nchan, time_row, g,
                                                      gain_weight, inverse);
  else if (precision == ARLGPU_FP32C)
    k_gaintable<float2><<<nblk(ncell), 256, 0, st>>>(static_cast<float2 *>(vis), ntimes, nants, nchan, time_row, g,
                                                     gain_weight, inverse);
  else
    return fail(ARLGPU_ERR_INVALID, "bad precision");
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

extern "C" int arlgpu_gain_chi2(const void *vobs, const void *model, const double *weight, int64_t nvis, int32_t npol,
                                int precision, const int32_t *a1, const int32_t *a2, const void *gains, int32_t nant,
                                double *chi2, void *grad_model, void *grad_gains, void *stream) {
  if (nvis < 0 || npol < 1 || nant < 1 || !chi2 || (nvis > 0 && (!vobs || !model || !a1 || !a2 || !gains)))
    return fail(ARLGPU_ERR_INVALID, "bad arguments");
  if (nant > 4096) return fail(ARLGPU_ERR_UNSUPPORTED, "more than 4096 antennas");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ARL_CUDA(cudaMemsetAsync(chi2, 0, sizeof(double), st));
  if (grad_gains) ARL_CUDA(cudaMemsetAsync(grad_gains, 0, sizeof(double2) * nant, st));
  if (nvis == 0) return ARLGPU_OK;
  const double2 *g = static_cast<const double2 *>(gains);
  double2 *gg = static_cast<double2 *>(grad_gains);
  if (precision == ARLGPU_FP64)
    launch_gain_chi2<double2>(vobs, model, weight, nvis, npol, a1, a2, g, nant, chi2, grad_model, gg, st);
  else if (precision == ARLGPU_FP32C)
    launch_gain_chi2<float2>(vobs, model, weight, nvis, npol, a1, a2, g, nant, chi2, grad_model, gg, st);
  else
    return fail(ARLGPU_ERR_INVALID, "bad precision");
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}
