// Direct Fourier transform of point components, and its adjoint.
//
// Reference behaviour:
//   predict_skycomponent_visibility   processing_components/imaging/base.py:192-244
//   simulate_point                    processing_library/util/coordinate_support.py:192-212
//
// vis[r, p] += sum_k flux[k, chan[r], p] exp(-2 pi i (u l_k + v m_k + w n_k)),
// n_k = sqrt(1 - l_k^2 - m_k^2) - 1 supplied by the caller.  |u l| reaches 1e4
// turns and more on long baselines, so the phase needs far more than FP32: the
// FP64 path forms it in FP64 and reduces it to [-1/2, 1/2] turns before an FP64
// sincospi; the FP32C path forms it modulo one turn in 32-bit fixed point
// (k_dft_predict32), with an error below 2^-29 turns before the one rounding
// to FP32.
//
// The adjoint, image[k, p] += Re sum_r conj(exp(...)) x[r, p] (for rows of
// one channel map), gives the gradient of a DFT-predicted chi^2 with respect
// to the component fluxes; the gradient checks use it as a dense reference.
#include <algorithm>

#include "common.cuh"
#include "dsmath.cuh"

namespace arlgpu {

void count_launch(unsigned n);

constexpr int kTile = 128;  // components staged per shared-memory tile

template <typename R> struct Phasor;
template <> struct Phasor<float> {
  __device__ static __forceinline__ void at(double turns, float *c, float *s) {
    const float t = (float)(turns - rint(turns));
    sincospif(-2.f * t, s, c);
  }
};
template <> struct Phasor<double> {
  __device__ static __forceinline__ void at(double turns, double *c, double *s) {
    sincospi(-2.0 * (turns - rint(turns)), s, c);
  }
};

template <typename R, int NPOL>
__global__ void __launch_bounds__(256)
k_dft_predict(const double *__restrict__ uvw, const int32_t *__restrict__ chan, int64_t nvis,
              const double *__restrict__ lmn, const double *__restrict__ flux, int ncomp, int nchan,
              typename Cplx<R>::T *__restrict__ vis) {
  __shared__ double s_lmn[kTile][3];
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = r < nvis;
  double u = 0, v = 0, w = 0;
  int c = 0;
  if (live) {
    u = uvw[3 * r];
    v = uvw[3 * r + 1];
    w = uvw[3 * r + 2];
    c = chan ? chan[r] : 0;
  }
  R ar[NPOL], ai[NPOL];
#pragma unroll
  for (int p = 0; p < NPOL; ++p) ar[p] = ai[p] = 0;
  for (int k0 = 0; k0 < ncomp; k0 += kTile) {
    const int nk = min(kTile, ncomp - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < nk * 3; i += blockDim.x) s_lmn[i / 3][i % 3] = lmn[3 * k0 + i];
    __syncthreads();
    if (!live) continue;
    for (int k = 0; k < nk; ++k) {
      const double turns = fma(u, s_lmn[k][0], fma(v, s_lmn[k][1], w * s_lmn[k][2]));
      R cs, sn;
      Phasor<R>::at(turns, &cs, &sn);
      const double *fk = flux + ((int64_t)(k0 + k) * nchan + c) * NPOL;
#pragma unroll
      for (int p = 0; p < NPOL; ++p) {
        const R f = (R)fk[p];
        ar[p] += f * cs;
        ai[p] += f * sn;
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int p = 0; p < NPOL; ++p) {
    typename Cplx<R>::T o = vis[r * NPOL + p];
    o.x += ar[p];
    o.y += ai[p];
    vis[r * NPOL + p] = o;
  }
}

// ---------------------------------------------------------------------------
// FP32C predict.  What bounds it is issue slots per (row, component) pair: in
// FP64 the phase alone is 3 multiply-adds, a rounding and a subtraction, two
// conversions follow per flux, and GB300 retires 2 FP64 operations (arithmetic
// or conversion) a clock and SM against 128 FP32 ones.  Here
//   * u = Uhi + Ulo 2^-32 and l = Lhi 2^-31 + Llo 2^-63, signed 32-bit words;
//     Uhi Lhi (low word) + hi(Uhi Llo) + hi(Ulo Lhi) is u l modulo 2 turns in
//     units of 2^-31, so three axes cost three 32-bit products, six high words
//     and additions that wrap by themselves.  The dropped Ulo Llo is below a
//     unit, and so are the six truncations, whose mean (half a unit each) is
//     added back for the axes where both low words are there to be truncated: a row
//     or a component at the phase centre has phase zero exactly.  The mean is a byte
//     of the direction, picked by the row (a dot product of bytes took 316 us; 64-bit
//     sums of the six products, which halve the error, 363 us);
//   * sine and cosine are polynomials over an eighth of a turn on either side
//     of a quadrant's centre, the quadrant read from the phase's top bits;
//   * fluxes are converted once per block into shared memory.
// 2.67 M rows x 50 components: 1687 -> 264 us.
// Rows with a coordinate of 2^31 wavelengths or more (or not finite) and
// components whose direction cosines do not lie inside (-1, 1) take FP64 phases.
// ---------------------------------------------------------------------------
constexpr int kFluxWords = 6144;  // shared fluxes of one tile of components

struct FixDir {
  int lh, mh, nh, ll, ml, nl;
  // Byte b: the bits that b and low_words of the direction share; the top bit: FP64 phases.
  unsigned mean[2];
};

// x 2^scale, truncated, as hi 2^32 + lo in signed words: integer operations on
// the bits of x, because the FP64 rounding, scaling and conversions of a
// row's three coordinates took as long as 20 components.  False where
// |x| 2^scale reaches 2^63 or x is not finite.
__device__ __forceinline__ bool fix_words(double x, int scale, int *hi, int *lo) {
  const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
  const int s = 1085 - scale - (int)((xh >> 20) & 0x7ff);  // the mantissa, 10 bits up, moves right by s
  const unsigned long long m = ((unsigned long long)((xh & 0xfffffu) | 0x100000u) << 32 | xl) << 10;
  unsigned long long v = s < 64 ? m >> (s & 63) : 0;
  if (xh >> 31) v = 0 - v;
  *lo = (int)v;
  *hi = (int)((v + 0x80000000ull) >> 32);
  return s >= 0 && *hi != (int)0x80000000;  // the words' range, also after rounding hi
}

// A bit for each axis: its low word is not zero.
__device__ __forceinline__ unsigned low_words(int x, int y, int z) { return (x != 0) | (y != 0) << 1 | (z != 0) << 2; }

// cos and sin of 2 pi t, t = phase 2^-32 turns.
__device__ __forceinline__ void sincos_fix(int phase, float *c, float *s) {
  const unsigned q = ((unsigned)phase + 0x20000000u) >> 30;
  const float y = (float)(int)((unsigned)phase - (q << 30)) * 1.862645149230957e-9f;  // 2^-29
  sincos_quadrant(y, q, c, s);
}

template <int NPOL, int RPT>
__global__ void __launch_bounds__(256)
k_dft_predict32(const double *__restrict__ uvw, const int32_t *__restrict__ chan, int64_t nvis,
                const double *__restrict__ lmn, const double *__restrict__ flux, int ncomp, int nchan, int tile,
                float2 *__restrict__ vis) {
  __shared__ FixDir s_dir[kTile];
  __shared__ float s_flux[kFluxWords];
  const int64_t r0 = (int64_t)blockIdx.x * (256 * RPT) + threadIdx.x;  // rows r0 + 256 j
  const bool staged = tile > 0;
  const int per = nchan * NPOL, nt = staged ? tile : kTile;
  int uh[RPT], ul[RPT], vh[RPT], vl[RPT], wh[RPT], wl[RPT], c[RPT];
  unsigned sel[RPT];  // byte_perm's selector: the row's byte of FixDir::mean, then byte 0 (zero) three times
  bool fix = true;
  float ar[RPT][NPOL], ai[RPT][NPOL];
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int64_t r = min(r0 + 256 * j, nvis - 1);  // rows past the end repeat the last one and are not written
    fix = fix_words(uvw[3 * r], 32, &uh[j], &ul[j]) && fix;
    fix = fix_words(uvw[3 * r + 1], 32, &vh[j], &vl[j]) && fix;
    fix = fix_words(uvw[3 * r + 2], 32, &wh[j], &wl[j]) && fix;
    sel[j] = low_words(ul[j], vl[j], wl[j]);
    c[j] = chan ? chan[r] * NPOL : 0;
#pragma unroll
    for (int p = 0; p < NPOL; ++p) ar[j][p] = ai[j][p] = 0.f;
  }
  for (int k0 = 0; k0 < ncomp; k0 += nt) {
    const int nk = min(nt, ncomp - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < nk; i += 256) {
      FixDir d;
      const double *q = lmn + 3 * (int64_t)(k0 + i);
      bool ok = fix_words(q[0], 63, &d.lh, &d.ll);
      ok = fix_words(q[1], 63, &d.mh, &d.ml) && ok;
      ok = fix_words(q[2], 63, &d.nh, &d.nl) && ok;
      const unsigned has = low_words(d.ll, d.ml, d.nl);
      d.mean[0] = d.mean[1] = 0;
      for (unsigned b = 1; b < 8; ++b) d.mean[b >> 2] |= (unsigned)__popc(has & b) << (8 * (b & 3));
      d.mean[1] |= ok ? 0u : 0x80000000u;
      s_dir[i] = d;
    }
    if (staged)
      for (int i = threadIdx.x; i < nk * per; i += 256) s_flux[i] = (float)flux[(int64_t)k0 * per + i];
    __syncthreads();
    for (int k = 0; k < nk; ++k) {
      const FixDir d = s_dir[k];
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        float cs, sn;
        if (fix && (int)d.mean[1] >= 0) {
          const unsigned lo = (unsigned)uh[j] * d.lh + (unsigned)vh[j] * d.mh + (unsigned)wh[j] * d.nh;
          const unsigned hi = (unsigned)__mulhi(uh[j], d.ll) + (unsigned)__mulhi(ul[j], d.lh) +
                              (unsigned)__mulhi(vh[j], d.ml) + (unsigned)__mulhi(vl[j], d.mh) +
                              (unsigned)__mulhi(wh[j], d.nl) + (unsigned)__mulhi(wl[j], d.nh);
          sincos_fix((int)((lo + hi + __byte_perm(d.mean[0], d.mean[1], sel[j])) << 1), &cs, &sn);
          sn = -sn;
        } else {
          const double *q = lmn + 3 * (int64_t)(k0 + k), *x = uvw + 3 * min(r0 + 256 * j, nvis - 1);
          Phasor<float>::at(fma(x[0], q[0], fma(x[1], q[1], x[2] * q[2])), &cs, &sn);
        }
#pragma unroll
        for (int p = 0; p < NPOL; ++p) {
          const float f = staged ? s_flux[k * per + c[j] + p] : (float)flux[(int64_t)(k0 + k) * per + c[j] + p];
          ar[j][p] += f * cs;
          ai[j][p] += f * sn;
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int64_t r = r0 + 256 * j;
    if (r >= nvis) break;
#pragma unroll
    for (int p = 0; p < NPOL; ++p) {
      float2 o = vis[r * NPOL + p];
      o.x += ar[j][p];
      o.y += ai[j][p];
      vis[r * NPOL + p] = o;
    }
  }
}

// ---------------------------------------------------------------------------
// Channel of each row: the rank of its frequency among the rows' distinct ones
// (get_frequency_map with no image; numpy.unique's order: ascending, NaNs equal
// and last, the two zeros equal).  A table of at least twice as many slots as
// the components have channels holds the distinct values.  More values than
// channels are the caller's error; rows that pass the count's check together can
// fill the table then, so every probe is bounded by its size.
//   k_chan_first   empties the table and adds the first rows' values: with the
//                  channel the fastest axis, as rows are ordered, all of them
//   k_chan_insert  every other row's value (the row that claims a slot counts it)
//   k_chan_rank    each slot's number of smaller values
//   k_chan_rows    each row's slot -> its rank
// The pass costs a read of the frequencies each for insert and rows: 2.67 M
// rows take 25 us in all, where sorting them on the host took 88 ms.
// ---------------------------------------------------------------------------
constexpr unsigned long long kNoKey = ~0ull;  // no value maps to it: NaNs are made one positive NaN first

// Order-preserving integer of a double.
__device__ __forceinline__ unsigned long long chan_key(double f) {
  unsigned long long b = (unsigned long long)__double_as_longlong(f);
  if ((b << 1) > 0xffe0000000000000ull) b = 0x7ff8000000000000ull;  // any NaN
  if ((b << 1) == 0) b = 0;                                         // -0.0 as +0.0
  return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}

__device__ __forceinline__ unsigned chan_hash(unsigned long long k) {
  unsigned h = (unsigned)(k >> 32) * 0x9E3779B1u ^ (unsigned)k * 0x85EBCA77u;
  return h ^ (h >> 15);
}

// One row's value into the table.  A slot never changes once it holds a value,
// so a cached read of one is good; a slot that looks empty is read again past
// L1 before the atomic, so that the rows in flight when a value first appears do
// not all queue for one word.
__device__ __forceinline__ bool chan_add(unsigned long long k, int max_chan, unsigned long long *keys, unsigned mask,
                                         int32_t *count) {
  unsigned h = chan_hash(k) & mask;
  for (unsigned probe = 0; probe <= mask; ++probe, h = (h + 1) & mask) {
    unsigned long long have = keys[h];
    if (have == kNoKey) have = __ldcg(&keys[h]);
    if (have == kNoKey) {
      if (__ldcg(count) > max_chan) return false;  // too many already
      have = atomicCAS(&keys[h], kNoKey, k);
      if (have == kNoKey) {
        atomicAdd(count, 1);
        return true;
      }
    }
    if (have == k) return true;
  }
  return false;
}

constexpr int kChanFirst = 4096;  // rows that the first kernel adds

__global__ void __launch_bounds__(1024)
k_chan_first(const double *__restrict__ freq, int64_t n, int max_chan, unsigned long long *__restrict__ keys, int cap,
             int32_t *__restrict__ count) {
  for (int i = threadIdx.x; i < cap; i += blockDim.x) keys[i] = kNoKey;
  if (threadIdx.x == 0) *count = 0;
  __threadfence();
  __syncthreads();
  for (int r = threadIdx.x; r < min(n, (int64_t)kChanFirst); r += blockDim.x)
    if (!chan_add(chan_key(freq[r]), max_chan, keys, (unsigned)cap - 1, count)) return;
}

__global__ void k_chan_insert(const double *__restrict__ freq, int64_t n, int max_chan,
                              unsigned long long *__restrict__ keys, unsigned mask, int32_t *__restrict__ count) {
  unsigned long long last = kNoKey;
  for (int64_t r = kChanFirst + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long k = chan_key(freq[r]);
    if (k != last && !chan_add(k, max_chan, keys, mask, count)) return;
    last = k;
  }
}

__global__ void k_chan_rank(const unsigned long long *__restrict__ keys, int cap, int32_t *__restrict__ rank) {
  __shared__ unsigned long long s_key[256];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned long long k = i < cap ? keys[i] : 0;
  int less = 0;
  for (int t0 = 0; t0 < cap; t0 += 256) {
    __syncthreads();
    s_key[threadIdx.x] = t0 + threadIdx.x < cap ? keys[t0 + threadIdx.x] : kNoKey;
    __syncthreads();
    for (int t = 0; t < 256; ++t) less += s_key[t] < k;
  }
  if (i < cap) rank[i] = less;
}

__global__ void k_chan_rows(const double *__restrict__ freq, int64_t n, const unsigned long long *__restrict__ keys,
                            const int32_t *__restrict__ rank, unsigned mask, int32_t *__restrict__ row_chan) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long k = chan_key(freq[r]);
    unsigned h = chan_hash(k) & mask;
    for (unsigned probe = 0; probe < mask && keys[h] != k; ++probe) h = (h + 1) & mask;
    row_chan[r] = rank[h];
  }
}

// k_chan_rank compares every pair of slots; beyond this many channels a sort is
// the better method and the caller's.
constexpr int32_t kMaxChan = 1 << 14;

static int chan_cap(int32_t max_chan) {
  int cap = 256;
  while (cap < 2 * ((int64_t)max_chan + 1)) cap <<= 1;
  return cap;
}

// image[k, p] += Re sum_r conj(phasor_rk) x[r, p]: one warp per component,
// lanes over rows, shuffle reduction.
template <typename R, int NPOL>
__global__ void __launch_bounds__(256)
k_dft_adjoint(const double *__restrict__ uvw, int64_t nvis, const double *__restrict__ lmn, int ncomp,
              const typename Cplx<R>::T *__restrict__ x, double *__restrict__ image) {
  const int lane = threadIdx.x & 31;
  const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= ncomp) return;
  const double l = lmn[3 * k], m = lmn[3 * k + 1], n = lmn[3 * k + 2];
  double acc[NPOL];
#pragma unroll
  for (int p = 0; p < NPOL; ++p) acc[p] = 0.0;
  for (int64_t r = lane; r < nvis; r += 32) {
    const double turns = fma(uvw[3 * r], l, fma(uvw[3 * r + 1], m, uvw[3 * r + 2] * n));
    R cs, sn;
    Phasor<R>::at(turns, &cs, &sn);
#pragma unroll
    for (int p = 0; p < NPOL; ++p) {
      const typename Cplx<R>::T xv = x[r * NPOL + p];
      acc[p] += (double)(cs * xv.x + sn * xv.y);  // Re(conj(c + i s) x)
    }
  }
#pragma unroll
  for (int p = 0; p < NPOL; ++p) {
    double s = acc[p];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) image[k * NPOL + p] += s;
  }
}

// Two rows a thread share the component's words and halve the blocks' set-up;
// one where that would leave SMs without a block (2 x 152 blocks of 512 rows).
// Fluxes are staged, as many components at a time as fit, where a component has at
// most half as many channels as a block has rows; more are read from global memory,
// where a block converts the ones its rows ask for.  Staged / read, us, 20 components,
// one polarisation: 3,000 rows of 128 channels 10.4 / 11.2, of 512 12.6 / 11.5, of
// 1,500 23.2 / 11.7; 200,000 rows x 4 of 256 channels 31.6 / 40.5, of 512 47.9 / 41.9.
template <int NPOL>
static void launch_predict32(const double *uvw, const int32_t *chan, int64_t nvis, const double *lmn,
                             const double *flux, int ncomp, int nchan, void *vis, cudaStream_t st) {
  float2 *o = static_cast<float2 *>(vis);
  const bool two = nvis >= 2 * 152 * 512;
  const int tile = nchan <= (two ? 256 : 128) ? std::min(kFluxWords / (nchan * NPOL), kTile) : 0;
  if (two)
    k_dft_predict32<NPOL, 2><<<(unsigned)((nvis + 511) / 512), 256, 0, st>>>(uvw, chan, nvis, lmn, flux, ncomp, nchan,
                                                                             tile, o);
  else
    k_dft_predict32<NPOL, 1><<<(unsigned)((nvis + 255) / 256), 256, 0, st>>>(uvw, chan, nvis, lmn, flux, ncomp, nchan,
                                                                             tile, o);
}

template <typename R>
static int launch_predict(const double *uvw, const int32_t *chan, int64_t nvis, const double *lmn,
                          const double *flux, int ncomp, int nchan, int npol, void *vis, cudaStream_t st) {
  const int blocks = (int)((nvis + 255) / 256);
  if constexpr (sizeof(R) == 4) {
    switch (npol) {
      case 1: launch_predict32<1>(uvw, chan, nvis, lmn, flux, ncomp, nchan, vis, st); break;
      case 2: launch_predict32<2>(uvw, chan, nvis, lmn, flux, ncomp, nchan, vis, st); break;
      case 4: launch_predict32<4>(uvw, chan, nvis, lmn, flux, ncomp, nchan, vis, st); break;
      default: return fail(ARLGPU_ERR_UNSUPPORTED, "npol must be 1, 2 or 4");
    }
  } else {
    double2 *o = static_cast<double2 *>(vis);
    switch (npol) {
      case 1: k_dft_predict<R, 1><<<blocks, 256, 0, st>>>(uvw, chan, nvis, lmn, flux, ncomp, nchan, o); break;
      case 2: k_dft_predict<R, 2><<<blocks, 256, 0, st>>>(uvw, chan, nvis, lmn, flux, ncomp, nchan, o); break;
      case 4: k_dft_predict<R, 4><<<blocks, 256, 0, st>>>(uvw, chan, nvis, lmn, flux, ncomp, nchan, o); break;
      default: return fail(ARLGPU_ERR_UNSUPPORTED, "npol must be 1, 2 or 4");
    }
  }
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

template <typename R>
static int launch_adjoint(const double *uvw, int64_t nvis, const double *lmn, int ncomp, int npol, const void *x,
                          double *image, cudaStream_t st) {
  const int64_t threads = (int64_t)ncomp * 32;
  const int blocks = (int)((threads + 255) / 256);
  using CT = typename Cplx<R>::T;
  const CT *xi = static_cast<const CT *>(x);
  switch (npol) {
    case 1: k_dft_adjoint<R, 1><<<blocks, 256, 0, st>>>(uvw, nvis, lmn, ncomp, xi, image); break;
    case 2: k_dft_adjoint<R, 2><<<blocks, 256, 0, st>>>(uvw, nvis, lmn, ncomp, xi, image); break;
    case 4: k_dft_adjoint<R, 4><<<blocks, 256, 0, st>>>(uvw, nvis, lmn, ncomp, xi, image); break;
    default: return fail(ARLGPU_ERR_UNSUPPORTED, "npol must be 1, 2 or 4");
  }
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

}  // namespace arlgpu

using namespace arlgpu;

extern "C" int arlgpu_dft_predict(const double *uvw, const int32_t *row_chan, int64_t nvis, const double *lmn,
                                  const double *flux, int32_t ncomp, int32_t nchan, int32_t npol, int precision,
                                  void *vis, void *stream) {
  if (precision != ARLGPU_FP32C && precision != ARLGPU_FP64) return fail(ARLGPU_ERR_INVALID, "bad precision");
  if (nvis < 0 || ncomp < 0 || nchan < 1) return fail(ARLGPU_ERR_INVALID, "bad sizes");
  if (nvis == 0 || ncomp == 0) return ARLGPU_OK;
  if (!uvw || !lmn || !flux || !vis) return fail(ARLGPU_ERR_INVALID, "null array argument");
  if (nchan > 1 && !row_chan) return fail(ARLGPU_ERR_INVALID, "row_chan is required when nchan > 1");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == ARLGPU_FP64) return launch_predict<double>(uvw, row_chan, nvis, lmn, flux, ncomp, nchan, npol, vis, st);
  return launch_predict<float>(uvw, row_chan, nvis, lmn, flux, ncomp, nchan, npol, vis, st);
}

extern "C" int arlgpu_dft_adjoint(const double *uvw, int64_t nvis, const double *lmn, int32_t ncomp, int32_t npol,
                                  int precision, const void *x, double *image, void *stream) {
  if (precision != ARLGPU_FP32C && precision != ARLGPU_FP64) return fail(ARLGPU_ERR_INVALID, "bad precision");
  if (nvis < 0 || ncomp < 0) return fail(ARLGPU_ERR_INVALID, "bad sizes");
  if (nvis == 0 || ncomp == 0) return ARLGPU_OK;
  if (!uvw || !lmn || !x || !image) return fail(ARLGPU_ERR_INVALID, "null array argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == ARLGPU_FP64) return launch_adjoint<double>(uvw, nvis, lmn, ncomp, npol, x, image, st);
  return launch_adjoint<float>(uvw, nvis, lmn, ncomp, npol, x, image, st);
}

extern "C" int arlgpu_row_channels_bytes(int32_t max_chan, size_t *bytes_host) {
  if (max_chan < 0 || max_chan > kMaxChan || !bytes_host) return fail(ARLGPU_ERR_INVALID, "bad channel count");
  *bytes_host = (size_t)chan_cap(max_chan) * (sizeof(unsigned long long) + sizeof(int32_t));
  return ARLGPU_OK;
}

extern "C" int arlgpu_row_channels(const double *frequency, int64_t nvis, int32_t max_chan, int32_t *row_chan,
                                   int32_t *nchan_dev, void *workspace, size_t workspace_bytes, void *stream) {
  if (nvis < 0 || max_chan < 0 || max_chan > kMaxChan) return fail(ARLGPU_ERR_INVALID, "bad sizes");
  if (!nchan_dev || !workspace || (nvis > 0 && (!frequency || !row_chan)))
    return fail(ARLGPU_ERR_INVALID, "null array argument");
  if ((uintptr_t)workspace & 7) return fail(ARLGPU_ERR_INVALID, "workspace must be 8-byte aligned");
  const int cap = chan_cap(max_chan);
  if (workspace_bytes < (size_t)cap * (sizeof(unsigned long long) + sizeof(int32_t)))
    return fail(ARLGPU_ERR_WORKSPACE, "workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned long long *keys = static_cast<unsigned long long *>(workspace);
  int32_t *rank = reinterpret_cast<int32_t *>(keys + cap);
  k_chan_first<<<1, 1024, 0, st>>>(frequency, nvis, max_chan, keys, cap, nchan_dev);
  count_launch(1);
  ARL_LAUNCH_CHECK();
  if (nvis == 0) return ARLGPU_OK;
  const int64_t want = (nvis + 255) / 256;
  const int blocks = (int)(want < 152 * 8 ? want : 152 * 8);
  if (nvis > kChanFirst) {
    k_chan_insert<<<blocks, 256, 0, st>>>(frequency, nvis, max_chan, keys, (unsigned)cap - 1, nchan_dev);
    ARL_LAUNCH_CHECK();
    count_launch(1);
  }
  k_chan_rank<<<(cap + 255) / 256, 256, 0, st>>>(keys, cap, rank);
  ARL_LAUNCH_CHECK();
  k_chan_rows<<<blocks, 256, 0, st>>>(frequency, nvis, keys, rank, (unsigned)cap - 1, row_chan);
  ARL_LAUNCH_CHECK();
  count_launch(2);
  return ARLGPU_OK;
}
