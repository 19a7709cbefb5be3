// Double-single inverse 2-D FFT for the FP32C path (K5 / K9 transforms).
//
// Reference behaviour:
//   ifft (centred inverse transform)  processing_library/fourier_transforms/fft_support.py:41-89
//   fft_griddata_to_image             processing_components/griddata/gridding.py:270-289
//   w-stack slice sum                 processing_components/imaging/wstack_single.py:26-60 with
//                                     workflows/serial/imaging/imaging_serial.py:186-197
//
// The grid correction multiplies transform rounding by up to max(gcf)/min(gcf)
// (~6e4 at the edge of a PSWF-corrected field), so the inverse transform must
// be much more accurate than FP32.  GB300 runs FP64 at 1/64 of its FP32 rate,
// which makes cuFFT's FP64 transform of an 8192^2 plane compute-bound at
// ~14 ms.  Here every complex value is a pair of double-single numbers (~48-bit
// significands) and all arithmetic runs on the FP32 pipes.
//
// Layout: a plane of ny x nx points, row-major, a point as float4 (re.hi, im.hi,
// re.lo, im.lo).  Three passes per plane:
//   rows   one CTA per 4096 points (4096 / nx rows, or half of an
//          8192-point row): FP32 grid (w-planes summed, chk sign) -> row
//          DFTs -> DS buffer
//   cols1  ny = N1 * N2: DFTs of length N1 over rows n2 + N2 n1 of 32 or more
//          adjacent columns, times exp(2 pi i n2 k1 / ny), in place
//   cols2  DFTs of length N2 over rows N2 k1 + n2 -> row k1 + N1 k2, with the
//          epilogue fused: image write (invert_2d) or the w-screen product
//          summed over the slices of the group (w-stacking)
// What bounds them is the FP32 pipe, about 790 operations a point of 8192^2 (1.4 ms a
// plane) against 4.5 GB of traffic (0.7 ms), so the passes spend their issue slots
// on those operations:
//   * a thread transforms 16 points in registers (radix 16, or 16 / R of radix R), so
//     that a DFT of up to 4096 points crosses shared memory twice and one of up to
//     128 once; the lengths are compile-time constants, and the first pass reads
//     global memory into registers (16 loads in flight), the last writes the
//     epilogue;
//   * real and imaginary parts are adjacent, so that sums are packed FP32 pairs:
//     the same lane rate as single ones, for half the issue slots.
// Radix-4 passes of run-time length, one butterfly a thread through shared
// memory, were at 3.15 ms a plane of 8192^2 (w-stack, 32 planes: rows 1.20, cols1
// 0.74, cols2 1.20 ms); now 1.80 ms (0.62, 0.54, 0.63).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "dsmath.cuh"

namespace arlgpu {

void count_launch(unsigned n);

constexpr int kLog2Tw = 14;
constexpr int kTw = 1 << kLog2Tw;
// exp(+2 pi i m / 16384) as (cos hi, sin hi, cos lo, sin lo), for the twiddles between the column passes
__device__ float4 g_tw[kTw];
// exp(+2 pi i m k / (16 M)) at [k][m], for the passes with M points left: the lanes of a warp take adjacent m
__device__ float4 g_tw256[16 * 256];
__device__ float4 g_tw16[16 * 16];

__global__ void k_tw_init() {
  auto at = [](int m, int n) {  // exp(2 pi i m / n)
    double s, c;
    sincospi(2.0 * (double)(m % n) / (double)n, &s, &c);
    const dsf cc = ds_from_double(c), ss = ds_from_double(s);
    return make_float4(cc.hi, ss.hi, cc.lo, ss.lo);
  };
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kTw; i += gridDim.x * blockDim.x) {
    g_tw[i] = at(i, kTw);
    if (i < 16 * 256) g_tw256[i] = at((i >> 8) * (i & 255), 4096);
    if (i < 16 * 16) g_tw16[i] = at((i >> 4) * (i & 15), 256);
  }
}

static std::atomic<unsigned> g_tw_ready{0};

// The tables are filled once per device on a stream that is not capturing
// (synchronised so that every later stream sees them); under capture the fill
// is recorded into the graph instead, every time, so a graph never relies on
// a fill that did not run.
static int ensure_twiddles(cudaStream_t st) {
  int dev = 0;
  ARL_CUDA(cudaGetDevice(&dev));
  const unsigned bit = 1u << (dev & 31);
  if (g_tw_ready.load() & bit) return ARLGPU_OK;
  k_tw_init<<<64, 256, 0, st>>>();
  ARL_LAUNCH_CHECK();
  count_launch(1);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  ARL_CUDA(cudaStreamIsCapturing(st, &cs));
  if (cs == cudaStreamCaptureStatusNone) {
    ARL_CUDA(cudaStreamSynchronize(st));
    g_tw_ready.fetch_or(bit);
  }
  return ARLGPU_OK;
}

// ---------------------------------------------------------------------------
// Packed FP32 pairs and complex double-single values.  h = (re.hi, im.hi), l = the
// low parts.  Sums are left unnormalised (hi + lo still equals the value; the
// next error-free sum or twiddle product absorbs it), which NumPy float32 emulation
// shows costs nothing measurable (7.9e-15 against 7.4e-15 of the scale at 8192 points).
// ---------------------------------------------------------------------------
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 un(f2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f2 swp(f2 a) {
  const float2 v = un(a);
  return pk(v.y, v.x);
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

struct cds {
  f2 h, l;
};
__device__ __forceinline__ cds c_from(float4 v) { return {pk(v.x, v.y), pk(v.z, v.w)}; }
__device__ __forceinline__ float4 c_to(cds a) {
  const float2 h = un(a.h), l = un(a.l);
  return make_float4(h.x, h.y, l.x, l.y);
}

// a + b, a - b: error-free sums of the high parts, low parts and errors added.
__device__ __forceinline__ cds c_add(cds a, cds b) {
  const f2 s = add2(a.h, b.h), v = sub2(s, a.h), e = add2(sub2(a.h, sub2(s, v)), sub2(b.h, v));
  return {s, add2(e, add2(a.l, b.l))};
}
__device__ __forceinline__ cds c_sub(cds a, cds b) {
  const f2 s = sub2(a.h, b.h), v = sub2(s, a.h), e = sub2(sub2(a.h, sub2(s, v)), add2(b.h, v));
  return {s, add2(e, sub2(a.l, b.l))};
}
// a + i b (SIGN > 0) or a - i b: b's parts change places, and products with +-1 in the fused operations (exact) give
// their signs.
template <int SIGN>
__device__ __forceinline__ cds c_addi(cds a, cds b) {
  const f2 j = SIGN > 0 ? pk(-1.f, 1.f) : pk(1.f, -1.f);
  const f2 bh = swp(b.h), s = fma2(bh, j, a.h), v = sub2(a.h, s);  // v = -(s - a)
  const f2 e = add2(sub2(a.h, add2(s, v)), fma2(bh, j, v));
  return {s, add2(e, fma2(swp(b.l), j, a.l))};
}

// a * w: the four products error-free through FMAs, part by part (their operands need no re-pairing), the rest packed.
__device__ __forceinline__ cds c_mul(cds a, float4 w) {
  const float2 ah = un(a.h), al = un(a.l);
  const float p1 = __fmul_rn(ah.x, w.x), p2 = __fmul_rn(-ah.y, w.y), p3 = __fmul_rn(ah.x, w.y), p4 = __fmul_rn(ah.y, w.x);
  const float e1 = __fmaf_rn(ah.x, w.x, -p1), e2 = __fmaf_rn(-ah.y, w.y, -p2), e3 = __fmaf_rn(ah.x, w.y, -p3),
              e4 = __fmaf_rn(ah.y, w.x, -p4);
  const f2 p = pk(p1, p3), q = pk(p2, p4);
  const f2 s = add2(p, q), v = sub2(s, p), t = add2(sub2(p, sub2(s, v)), sub2(q, v));
  const float2 c = un(add2(t, add2(pk(e1, e3), pk(e2, e4))));
  const float r = __fmaf_rn(-al.y, w.y, __fmaf_rn(-ah.y, w.w, __fmaf_rn(al.x, w.x, __fmaf_rn(ah.x, w.z, c.x))));
  const float i = __fmaf_rn(al.y, w.x, __fmaf_rn(ah.y, w.z, __fmaf_rn(al.x, w.y, __fmaf_rn(ah.x, w.w, c.y))));
  const f2 lo = pk(r, i), h = add2(s, lo);
  return {h, sub2(lo, sub2(h, s))};
}

// a * c for a real double-single constant.
__device__ __forceinline__ cds c_scale(cds a, float ch, float cl) {
  const f2 c = pk(ch, ch), d = pk(cl, cl);
  const f2 p = mul2(a.h, c), m = pk(-1.f, -1.f);
  const f2 e = fma2(a.l, c, fma2(a.h, d, fma2(a.h, c, mul2(p, m))));
  const f2 h = add2(p, e);
  return {h, sub2(e, sub2(h, p))};
}
constexpr float kR2h = 0.707106769f, kR2l = 1.21016175e-08f;  // sqrt(1/2)
__device__ __forceinline__ cds c_w8(cds a) { return c_scale(c_addi<1>(a, a), kR2h, kR2l); }     // a exp(2 pi i / 8)
__device__ __forceinline__ cds c_w8c(cds a) { return c_scale(c_addi<-1>(a, a), -kR2h, -kR2l); }  // a exp(2 pi i 3 / 8)

// Inverse DFTs of 2, 4, 8 and 16 points in registers, natural order in and out.
// DFT4 of (x0, x1, x2, x3); I2: of (x0, x1, i x2, x3).
template <bool I2 = false>
__device__ __forceinline__ void dft4(cds &x0, cds &x1, cds &x2, cds &x3) {
  const cds a = I2 ? c_addi<1>(x0, x2) : c_add(x0, x2), b = I2 ? c_addi<-1>(x0, x2) : c_sub(x0, x2);
  const cds c = c_add(x1, x3), d = c_sub(x1, x3);
  x0 = c_add(a, c);
  x1 = c_addi<1>(b, d);
  x2 = c_sub(a, c);
  x3 = c_addi<-1>(b, d);
}

template <int R> struct Dft;
template <> struct Dft<2> {
  __device__ static __forceinline__ void run(cds *x) {
    const cds a = c_add(x[0], x[1]);
    x[1] = c_sub(x[0], x[1]);
    x[0] = a;
  }
};
template <> struct Dft<4> {
  __device__ static __forceinline__ void run(cds *x) { dft4(x[0], x[1], x[2], x[3]); }
};
template <> struct Dft<8> {
  __device__ static __forceinline__ void run(cds *x) {
    cds s[4], d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[j] = c_add(x[j], x[j + 4]);
      d[j] = c_sub(x[j], x[j + 4]);
    }
    d[1] = c_w8(d[1]);
    d[3] = c_w8c(d[3]);
    dft4(s[0], s[1], s[2], s[3]);
    dft4<true>(d[0], d[1], d[2], d[3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      x[2 * j] = s[j];
      x[2 * j + 1] = d[j];
    }
  }
};
template <> struct Dft<16> {
  __device__ static __forceinline__ void run(cds *x) {
#pragma unroll
    for (int j = 0; j < 4; ++j) dft4(x[j], x[j + 4], x[j + 8], x[j + 12]);  // x[j + 4 k1]
    // times exp(2 pi i j k1 / 16); j k1 = 4 is a factor i, taken by the next DFT4.  cos, sin of pi / 8:
    constexpr float ch = 0.923879504f, cl = 2.83074897e-08f, sh = 0.382683426f, sl = 6.22335072e-09f;
    x[5] = c_mul(x[5], make_float4(ch, sh, cl, sl));
    x[9] = c_w8(x[9]);
    x[13] = c_mul(x[13], make_float4(sh, ch, sl, cl));
    x[6] = c_w8(x[6]);
    x[14] = c_w8c(x[14]);
    x[7] = c_mul(x[7], make_float4(sh, ch, sl, cl));
    x[11] = c_w8c(x[11]);
    x[15] = c_mul(x[15], make_float4(-ch, -sh, -cl, -sl));
    dft4(x[0], x[1], x[2], x[3]);
    dft4(x[4], x[5], x[6], x[7]);
    dft4<true>(x[8], x[9], x[10], x[11]);
    dft4(x[12], x[13], x[14], x[15]);
#pragma unroll
    for (int k = 0; k < 4; ++k)  // x[4 k1 + k2] holds X[k1 + 4 k2]: transpose
#pragma unroll
      for (int j = 0; j < k; ++j) {
        const cds t = x[4 * k + j];
        x[4 * k + j] = x[4 * j + k];
        x[4 * j + k] = t;
      }
  }
};

// ---------------------------------------------------------------------------
// Pass 1: row transforms of length L = 2^LX over CTAs of 4096 points (S = 4096 / L
// rows, 256 threads).  L = R0 M0: radix R0 on points n = n1 M0 + m, times
// exp(2 pi i m k1 / L); then radix 16 on what is left (M0 = 256: twice; M0 = 16:
// once).  The point with digit k1 done and n left lies at k1 M0 + n, one slot of
// padding every M0: the last pass's lanes run over k1.  Output k = k1 + R0 k2 +
// 16 R0 k3.
//
// Logical plane q of the input is the sum over z < nsum of grid[q * qstride +
// z * plane]; rows of planes [q0, q0 + np) go to buf[(q - q0) * plane + y * nx + x]
// with the chk sign applied on input.
//
// SPLIT: rows of 8192 points as two 4096-point halves on two CTAs: the first
// decimation-in-frequency stage, span 4096, is done while loading, half 0 taking
// x[n] + x[n + 4096] (whose DFT is X[2k]) and half 1 taking (x[n] - x[n + 4096])
// exp(2 pi i n / 8192) (DFT X[2k + 1]).  Half h's output k goes to slot
// h 4096 + k of the row (whole lines; the last column pass takes the columns in
// pairs from the halves).
// ---------------------------------------------------------------------------
constexpr int kRowT = 256, kRowPts = 4096;
template <int LX> struct RowGeom {
  static constexpr int L = 1 << LX, R0 = LX >= 9 ? L / 256 : L / 16, M0 = L / R0, S = kRowPts / L,
                       LP = L + R0, SMEM = S * LP * 16, LOG2M0 = LX >= 9 ? 8 : 4;
};

template <int LX, bool SPLIT>
__global__ void __launch_bounds__(kRowT, 2)
k_dsfft_rows(const float2 *__restrict__ grid, int64_t qstride, int nsum, int64_t q0, int np, int log2ny,
             float4 *__restrict__ buf) {
  using G = RowGeom<LX>;
  extern __shared__ float4 sm[];
  constexpr int R0 = G::R0, M0 = G::M0, S = G::S, IT = 16 / R0, LROW = SPLIT ? LX + 1 : LX;
  const int ny = 1 << log2ny, half = SPLIT ? blockIdx.x & 1 : 0;
  const int64_t plane = (int64_t)ny << LROW, nrows = (int64_t)np << log2ny;
  const int64_t row0 = SPLIT ? blockIdx.x >> 1 : (int64_t)blockIdx.x * S;
  // Points [j0, j0 + W) of plane z, signed; SPLIT: with the other half's added or subtracted.  All loads are in
  // flight before any is used.
  cds x[16];
  auto points = [&](auto j0_c, auto w_c, int z) {
    constexpr int J0 = decltype(j0_c)::value, W = decltype(w_c)::value;
    float2 ga[W], gb[SPLIT ? W : 1];
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int j = J0 + i, item = threadIdx.x + (j / R0) * kRowT, m = item & (M0 - 1), q = item >> G::LOG2M0;
      const int64_t R = row0 + q;
      const float2 *src = grid + (q0 + (R >> log2ny)) * qstride + z * plane + ((R & (ny - 1)) << LROW) + (j % R0) * M0 + m;
      ga[i] = R < nrows ? src[0] : make_float2(0.f, 0.f);
      if (SPLIT) gb[SPLIT ? i : 0] = src[1 << LX];
    }
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int j = J0 + i, item = threadIdx.x + (j / R0) * kRowT, m = item & (M0 - 1), q = item >> G::LOG2M0;
      const float sg = ((m + (int)(row0 + q)) & 1) ? -1.f : 1.f;  // M0, ny and 4096 are even
      const cds v{mul2(pk(ga[i].x, ga[i].y), pk(sg, sg)), 0};
      x[j] = z ? c_add(x[j], v) : v;
      if (SPLIT) {
        const float2 b = gb[SPLIT ? i : 0];
        const cds y{mul2(pk(b.x, b.y), pk(sg, sg)), 0};
        x[j] = half ? c_sub(x[j], y) : c_add(x[j], y);
      }
    }
  };
  points(std::integral_constant<int, 0>(), std::integral_constant<int, 16>(), 0);
  // Further w-planes four points at a time (the sums take the other loads' registers).  Point by point, plane after
  // plane, three planes of 8192^2 took 4.35 ms, now 2.62.
#pragma unroll 1
  for (int z = 1; z < nsum; ++z) {
    points(std::integral_constant<int, 0>(), std::integral_constant<int, 4>(), z);
    points(std::integral_constant<int, 4>(), std::integral_constant<int, 4>(), z);
    points(std::integral_constant<int, 8>(), std::integral_constant<int, 4>(), z);
    points(std::integral_constant<int, 12>(), std::integral_constant<int, 4>(), z);
  }
  // Rows (or the half's sums) that are all zero, common in w-stack slices, transform to zero.
  bool nz = false;
#pragma unroll
  for (int j = 0; j < 16; ++j) nz = nz || ((x[j].h | x[j].l) & 0x7fffffff7fffffffull) != 0;  // w-planes may cancel in h
  if (!__syncthreads_or(nz)) {
    for (int t = threadIdx.x; t < kRowPts; t += kRowT) {
      const int64_t R = row0 + (t >> LX);
      if (R < nrows)
        buf[(R << LROW) + (half << LX) + (t & (G::L - 1))] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  if (SPLIT && half) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = c_mul(x[j], __ldg(&g_tw[(j * M0 + threadIdx.x) << (kLog2Tw - LROW)]));
  }
#pragma unroll
  for (int j = 0; j < IT; ++j) {
    const int item = threadIdx.x + j * kRowT, m = item & (M0 - 1), q = item >> G::LOG2M0;
    Dft<R0>::run(x + j * R0);
    float4 *o = sm + q * G::LP + m;
#pragma unroll
    for (int k = 0; k < R0; ++k) {
      const float4 *tw = M0 == 256 ? g_tw256 : g_tw16;
      if (k) x[j * R0 + k] = c_mul(x[j * R0 + k], __ldg(&tw[k * (16 / R0) * M0 + m]));
      o[k * (M0 + 1)] = c_to(x[j * R0 + k]);
    }
  }
  __syncthreads();
  if (M0 == 256) {  // radix 16 on n = n2 16 + m2, in place
    const int m = threadIdx.x & 15, k1 = (threadIdx.x >> 4) % R0, q = (threadIdx.x >> 4) / R0;
    float4 *o = sm + q * G::LP + k1 * (M0 + 1) + m;
#pragma unroll
    for (int n = 0; n < 16; ++n) x[n] = c_from(o[n * 16]);
    Dft<16>::run(x);
#pragma unroll
    for (int k = 0; k < 16; ++k) o[k * 16] = c_to(k ? c_mul(x[k], __ldg(&g_tw16[k * 16 + m])) : x[k]);
    __syncthreads();
  }
  constexpr int KS = G::L / 16;  // outputs with the last digit 0
  const int kk = threadIdx.x & (KS - 1), q = threadIdx.x / KS, k1 = kk % R0, k2 = kk / R0;
  const float4 *o = sm + q * G::LP + k1 * (M0 + 1) + k2 * 16;
#pragma unroll
  for (int n = 0; n < 16; ++n) x[n] = c_from(o[n]);
  Dft<16>::run(x);
  const int64_t R = row0 + q;
  if (R >= nrows) return;
  float4 *out = buf + (R << LROW) + (half << LX) + kk;
#pragma unroll
  for (int k = 0; k < 16; ++k) out[k * KS] = c_to(x[k]);
}

// ---------------------------------------------------------------------------
// Column DFTs of length N = 2^LN over CTA tiles of PTS = N S points (S sequences, T =
// PTS / 16 threads): N <= 16 in registers; else radix R0 = N / 16 on n = n1 16 + m,
// through shared memory at [k1 16 + m][q], then radix 16.  Lanes run over the
// sequences (adjacent columns), so no access conflicts and the twiddles are one
// per warp.  load(n, q) gives a point, out(i, k, q, v) takes output k (i = 0..15
// numbers the thread's outputs); `sm` is free again after the last read's barrier,
// which the caller places.
// ---------------------------------------------------------------------------
// HALVES: the exchange goes in two steps, high parts, then low parts, through half the
// shared memory.
template <int LN, int LOG2PTS, bool HALVES = false, typename Load, typename Out>
__device__ __forceinline__ void col_dft(float4 *sm, Load load, Out out) {
  constexpr int N = 1 << LN, LS = LOG2PTS - LN, S = 1 << LS, T = 1 << (LOG2PTS - 4);
  cds x[16];
  if constexpr (N <= 16) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = load(j % N, (int)threadIdx.x + (j / N) * T);
#pragma unroll
    for (int j = 0; j < 16 / N; ++j) {
      Dft<N>::run(x + j * N);
#pragma unroll
      for (int k = 0; k < N; ++k) out(j * N + k, k, (int)threadIdx.x + j * T, x[j * N + k]);
    }
  } else {
    constexpr int R0 = N / 16;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int item = threadIdx.x + (j / R0) * T;
      x[j] = load((j % R0) * 16 + (item >> LS), item & (S - 1));
    }
#pragma unroll
    for (int j = 0; j < 16 / R0; ++j) {
      const int item = threadIdx.x + j * T, m = item >> LS, q = item & (S - 1);
      Dft<R0>::run(x + j * R0);
#pragma unroll
      for (int k = 0; k < R0; ++k) {
        if (k && m) x[j * R0 + k] = c_mul(x[j * R0 + k], __ldg(&g_tw16[k * (16 / R0) * 16 + m]));
        if (HALVES)
          reinterpret_cast<f2 *>(sm)[((k * 16 + m) << LS) + q] = x[j * R0 + k].h;
        else
          sm[((k * 16 + m) << LS) + q] = c_to(x[j * R0 + k]);
      }
    }
    __syncthreads();
    const int q = threadIdx.x & (S - 1), k1 = threadIdx.x >> LS;
    if (HALVES) {
      f2 *sh = reinterpret_cast<f2 *>(sm);
      f2 h[16];
#pragma unroll
      for (int n = 0; n < 16; ++n) h[n] = sh[((k1 * 16 + n) << LS) + q];
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int item = threadIdx.x + (j / R0) * T;
        sh[(((j % R0) * 16 + (item >> LS)) << LS) + (item & (S - 1))] = x[j].l;
      }
      __syncthreads();
#pragma unroll
      for (int n = 0; n < 16; ++n) x[n] = {h[n], sh[((k1 * 16 + n) << LS) + q]};
    } else {
#pragma unroll
      for (int n = 0; n < 16; ++n) x[n] = c_from(sm[((k1 * 16 + n) << LS) + q]);
    }
    Dft<16>::run(x);
#pragma unroll
    for (int k = 0; k < 16; ++k) out(k, k1 + R0 * k, q, x[k]);
  }
}

// Column decomposition ny = N1 N2 (N1 <= N2 <= 128) and the CTA tiles.
struct ColGeom {
  int log2N1, log2N2;
  int log2G1, log2WC1;  // cols1: n2 values x columns per 4096 points (the 2048-point tiles: half the columns)
  int log2G2, log2WC2;  // cols2: k1 values x columns, likewise
};

static bool col_geom(int log2ny, int log2nx, ColGeom *c) {
  c->log2N1 = log2ny / 2;
  c->log2N2 = log2ny - c->log2N1;
  if (c->log2N2 > 7 || c->log2N1 < 3) return false;
  const int lp = 12;  // log2 of the points per column CTA
  c->log2G1 = std::min(7 - c->log2N1, c->log2N2);
  c->log2WC1 = lp - c->log2N1 - c->log2G1;
  c->log2G2 = std::min(7 - c->log2N2, c->log2N1);
  c->log2WC2 = lp - c->log2N2 - c->log2G2;
  return c->log2WC1 <= log2nx && c->log2WC2 <= log2nx && c->log2WC1 >= 5 && c->log2WC2 >= 5;
}

constexpr int kColPts = 4096, kColT = 256, kWsPts = 2048, kWsT = 128;

// Slot within a row of image column x: 8192-point rows come as two halves.
__device__ __forceinline__ int col_slot(int x, int log2nx) {
  return log2nx == 13 ? ((x & 1) << 12) + (x >> 1) : x;
}

// Pass 2: length-N1 DFTs over rows n2 + N2 n1, twiddled, in place.  Tiles of 2048
// points on 128 threads, four CTAs an SM (this pass moves 32 bytes a point for some
// 180 operations, near the machine's balance; it waits on its loads a third of the
// time).  32 planes of 8192^2: 17.4 ms; the same with five CTAs, 18.0 with two of
// 256 threads, 22.5 with resident CTAs that copy their next tile into shared memory
// under the arithmetic.
template <int LN>
__global__ void __launch_bounds__(kWsT, 4)
k_dsfft_cols1(float4 *__restrict__ buf, int log2ny, int log2nx, ColGeom cg, int64_t ntile_pl) {
  extern __shared__ float4 sm[];
  const int64_t pl = blockIdx.x / ntile_pl;
  const int64_t t0 = blockIdx.x - pl * ntile_pl;
  const int lwc = cg.log2WC1 - 1, ntx = 1 << (log2nx - lwc);
  const int n2_0 = (int)(t0 / ntx) << cg.log2G1, x0 = (int)(t0 % ntx) << lwc;
  float4 *p = buf + (pl << (log2ny + log2nx)) + x0;
  const int WC1 = (1 << lwc) - 1;
  auto addr = [&](int n1, int q) {
    const int n2 = n2_0 + (q >> lwc);
    return ((int64_t)(n2 + (n1 << cg.log2N2)) << log2nx) + (q & WC1);
  };
  col_dft<LN, 11>(
      sm, [&](int n, int q) { return c_from(p[addr(n, q)]); },
      [&](int, int k, int q, cds v) {
        const int e = (n2_0 + (q >> lwc)) * k;
        p[addr(k, q)] = c_to(e ? c_mul(v, __ldg(&g_tw[e << (kLog2Tw - log2ny)])) : v);
      });
}

// Pass 3 for invert_2d: length-N2 DFTs over rows N2 k1 + n2 -> row k1 + N1 k2;
// image = part(v * chk * s0) * gcf [/ sumwt].  Plane pl is image b = b0 + pl.
template <int LN>
__global__ void __launch_bounds__(kColT, 2)
k_dsfft_cols2_image(const float4 *__restrict__ buf, int log2ny, int log2nx, ColGeom cg, int64_t ntile_pl, int64_t b0,
                    float s0, const double *__restrict__ gcf, const double *__restrict__ sumwt,
                    double *__restrict__ im_re, double *__restrict__ im_im) {
  extern __shared__ float4 sm[];
  const int64_t pl = blockIdx.x / ntile_pl;
  const int64_t t0 = blockIdx.x - pl * ntile_pl;
  const int ntx = 1 << (log2nx - cg.log2WC2);
  const int k1_0 = (int)(t0 / ntx) << cg.log2G2, x0 = (int)(t0 % ntx) << cg.log2WC2;
  const float4 *p = buf + (pl << (log2ny + log2nx));
  const int WC2 = (1 << cg.log2WC2) - 1;
  const int64_t b = b0 + pl;
  const int64_t obase = b << (log2ny + log2nx);
  double inv = 1.0;
  bool zero = false;
  if (sumwt) {
    const double w = sumwt[b];
    zero = !(w > 0.0);
    inv = zero ? 0.0 : 1.0 / w;
  }
  col_dft<LN, 12>(
      sm,
      [&](int n, int q) {
        const int k1 = k1_0 + (q >> cg.log2WC2);
        return c_from(p[((int64_t)((k1 << cg.log2N2) + n) << log2nx) + col_slot(x0 + (q & WC2), log2nx)]);
      },
      [&](int, int k2, int q, cds c) {
        const float4 v = c_to(c);
        const int k = k1_0 + (q >> cg.log2WC2) + (k2 << cg.log2N1), x = x0 + (q & WC2);
        const int64_t o = obase + ((int64_t)k << log2nx) + x;
        const double f = (double)((((x + k) & 1) ? -1.f : 1.f) * s0) * gcf[o];
        double re = ds_to_double({v.x, v.z}) * f, im = ds_to_double({v.y, v.w}) * f;
        if (sumwt) {
          re = zero ? 0.0 : re * inv;
          im = zero ? 0.0 : im * inv;
        }
        im_re[o] = re;
        if (im_im) im_im[o] = im;
      });
}

// Re(exp(-2 pi i w nterm) v) as a double-single number; nt.hi < 0 marks pixels beyond the horizon (0).
__device__ __forceinline__ dsf wscreen_re(float2 nt, dsf w, cds c) {
  const dsf t = ds_mul(w, {nt.x, nt.y});
  // turns reduced to [-1/2, 1/2], then the quadrant: roundings through the 1.5 2^23 shift
  const float big = 12582912.f;
  const float r = fabsf(t.hi) < 4.0e6f ? __fsub_rn(__fadd_rn(t.hi, big), big) : rintf(t.hi);
  const float f = __fadd_rn(__fsub_rn(t.hi, r), t.lo);
  const float q4 = __fmaf_rn(f, 4.f, big);
  float cs, sn;
  sincos_quadrant(__fmaf_rn(__fsub_rn(q4, big), -2.f, 8.f * f), __float_as_uint(q4) & 3u, &cs, &sn);
  // cos re + sin im
  const float4 v = c_to(c);
  const dsf p = two_prod(v.x, cs), q = two_prod(v.y, sn), s = two_sum(p.hi, q.hi);
  const float e = __fmaf_rn(v.w, sn, __fmaf_rn(v.z, cs, __fadd_rn(s.lo, __fadd_rn(p.lo, q.lo))));
  return nt.x < 0.f ? dsf{0.f, 0.f} : dsf{s.hi, e};
}

// Pass 3 for w-stacking: planes [p0, p1) of the flattened (image b, slice s)
// order, buf holding them from p0.  Each CTA sums Re(wb_s v) over the slices
// of its tile into double-single accumulators and adds them to the image's DS
// slots (image memory viewed as float2; the group holding slice 0 of image b
// writes them).  Tiles of 2048 points on 128 threads, and four CTAs share an SM,
// one's loads under the others' arithmetic; the sums and the w-screen terms wait in
// shared memory, each in its thread's own slots (in registers the sums spilled), and
// the exchange takes half a tile at a time to leave them the room: 20.1 ms for 32
// planes of 8192^2 against 23.3 ms with a whole tile and three CTAs.
template <int LN>
__global__ void __launch_bounds__(kWsT, 4)
k_dsfft_cols2_wstack(const float4 *__restrict__ buf, int log2ny, int log2nx, ColGeom cg, int64_t p0, int64_t p1,
                     int K, double fov, const double *__restrict__ wmean, float2 *__restrict__ slots) {
  extern __shared__ float4 sm[];
  constexpr int TILE = (1 << LN) > 16 ? kWsPts / 2 : 0;
  float2 *snt = reinterpret_cast<float2 *>(sm + TILE);  // per-pixel w-screen terms, [i][thread]
  const int lwc = cg.log2WC2 - 1, ntx = 1 << (log2nx - lwc);
  const int k1_0 = (int)(blockIdx.x / ntx) << cg.log2G2, x0 = (int)(blockIdx.x % ntx) << lwc;
  const int WC = (1 << lwc) - 1, n = 1 << log2nx;
  const dsf c2 = ds_from_double(fov * fov / ((double)n * n));
  float2 *sacc = snt + kWsPts;  // and the sums
  // the image pixel of the thread's output i
  auto pixel = [&](int i, int *k, int *x) {
    constexpr int N = 1 << LN, LS = 11 - LN, S = 1 << LS;
    const int q = N <= 16 ? (int)threadIdx.x + (i / N) * kWsT : threadIdx.x & (S - 1);
    const int k2 = N <= 16 ? i % N : (int)(threadIdx.x >> LS) + (N / 16) * i;
    *k = k1_0 + (q >> lwc) + (k2 << cg.log2N1);
    *x = x0 + (q & WC);
  };
#pragma unroll 1
  for (int i = 0; i < 16; ++i) {
    int k, x;
    pixel(i, &k, &x);
    const DsPix px = ds_wpix(k, x, n, c2);
    // nterm, or hi = -1 where r^2 >= 1
    snt[i * kWsT + threadIdx.x] = px.state == 2 ? make_float2(-1.f, 0.f) : make_float2(px.nterm.hi, px.nterm.lo);
    sacc[i * kWsT + threadIdx.x] = make_float2(0.f, 0.f);
  }
  for (int64_t pp = p0; pp < p1; ++pp) {
    const int64_t b = pp / K;
    const dsf w = ds_from_double(wmean[pp - b * K]);
    const float4 *p = buf + ((pp - p0) << (log2ny + log2nx));
    col_dft<LN, 11, true>(
        sm,
        [&](int n2, int q) {
          const int k1 = k1_0 + (q >> lwc);
          return c_from(p[((int64_t)((k1 << cg.log2N2) + n2) << log2nx) + col_slot(x0 + (q & WC), log2nx)]);
        },
        [&](int i, int, int, cds v) {
          float2 &sum = sacc[i * kWsT + threadIdx.x];
          const dsf a = ds_add({sum.x, sum.y}, wscreen_re(snt[i * kWsT + threadIdx.x], w, v));
          sum = make_float2(a.hi, a.lo);
        });
    if (pp + 1 == p1 || (pp + 1) / K != b) {
      const bool first = p0 <= b * K;
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        int k, x;
        pixel(i, &k, &x);
        float2 *o = slots + (b << (log2ny + log2nx)) + ((int64_t)k << log2nx) + x;
        float2 &sum = sacc[i * kWsT + threadIdx.x];
        dsf a{sum.x, sum.y};
        if (!first) {
          const float2 old = *o;
          a = ds_add(a, {old.x, old.y});
        }
        *o = make_float2(a.hi, a.lo);
        sum = make_float2(0.f, 0.f);
      }
    }
    __syncthreads();  // the exchange area is free for the next plane
  }
}

// image[b, y, x] = DS slot * chk * s0 * gcf / sumwt[b] (0 where sumwt <= 0), in
// place over the slots.
// An FP64 division a pixel and conversions bound it to 1.84 ms for 8192^2: 1.26 ms with the rounded quotient and
// integer conversions.
__global__ void k_ds_wstack_finish(double *image, int log2ny, int log2nx, float s0, const double *__restrict__ gcf,
                                   const double *__restrict__ sumwt) {
  const int64_t plane = (int64_t)1 << (log2ny + log2nx), base = blockIdx.y * plane;
  const int nx1 = (1 << log2nx) - 1;
  const double w = sumwt[blockIdx.y], rcp = w > 0.0 ? __drcp_rn(w) : 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < plane; i += (int64_t)gridDim.x * blockDim.x) {
    const int y = (int)(i >> log2nx), x = (int)(i & nx1);
    const float2 sl = reinterpret_cast<const float2 *>(image)[base + i];
    const float sg = (((x + y) & 1) ? -1.f : 1.f) * s0;
    const double v = (widen(sl.x * sg) + widen(sl.y * sg)) * gcf[base + i];
    image[base + i] = w > 0.0 ? rounded_quotient(v, w, rcp) : 0.0;
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static int ilog2_exact(int n) {
  if (n <= 0 || (n & (n - 1))) return -1;
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}

bool dsfft_supported(int ny, int nx) {
  const int ly = ilog2_exact(ny), lx = ilog2_exact(nx);
  if (ly < 6 || lx < 6 || lx > 13 || ly > 14) return false;
  ColGeom cg;
  return col_geom(ly, lx, &cg);
}

// Shared memory of the column kernels: the exchange tile where N > 16; the w-screen terms and sums.
static size_t col_smem(int log2N, bool wstack) {
  if (wstack) return (log2N > 4 ? kWsPts * 8 : 0) + kWsPts * 16;
  return log2N > 4 ? kColPts * 16 : 0;
}

// Calls f(std::integral_constant<int, V>) for the V of [LO, HI] that equals v.
template <int LO, int HI, typename F>
static void with_const(int v, F f) {
  if constexpr (LO <= HI) {
    if (v == LO)
      f(std::integral_constant<int, LO>());
    else
      with_const<LO + 1, HI>(v, f);
  }
}

// Function attributes belong to each device's context: set once per device.
static int set_smem() {
  static std::atomic<unsigned> done{0};
  int dev = 0;
  ARL_CUDA(cudaGetDevice(&dev));
  const unsigned bit = 1u << (dev & 31);
  if (done.load() & bit) return ARLGPU_OK;
  cudaError_t e = cudaSuccess;
  auto set = [&](const void *f, size_t bytes) {
    const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r != cudaSuccess) e = r;
  };
  for (int l = 6; l <= 12; ++l)
    with_const<6, 12>(l, [&](auto c) { set((const void *)k_dsfft_rows<c.value, false>, RowGeom<c.value>::SMEM); });
  set((const void *)k_dsfft_rows<12, true>, RowGeom<12>::SMEM);
  for (int l = 3; l <= 7; ++l)
    with_const<3, 7>(l, [&](auto c) {
      set((const void *)k_dsfft_cols1<c.value>, col_smem(l, false));
      set((const void *)k_dsfft_cols2_image<c.value>, col_smem(l, false));
      set((const void *)k_dsfft_cols2_wstack<c.value>, col_smem(l, true));
    });
  ARL_CUDA(e);
  done.fetch_or(bit);
  return ARLGPU_OK;
}

// Rows and first column pass of logical planes [q0, q0 + np) into buf.
static int rows_cols1(const float2 *grid, int64_t qstride, int nsum, int64_t q0, int64_t np, int ly, int lx,
                      const ColGeom &cg, float4 *buf, cudaStream_t st) {
  const int64_t nrows = np << ly;
  if (lx == 13) {
    k_dsfft_rows<12, true><<<(unsigned)(2 * nrows), kRowT, RowGeom<12>::SMEM, st>>>(grid, qstride, nsum, q0, (int)np,
                                                                                   ly, buf);
  } else {
    const int log2S = 12 - lx;
    const int64_t rblocks = (nrows + ((int64_t)1 << log2S) - 1) >> log2S;
    with_const<6, 12>(lx, [&](auto c) {
      k_dsfft_rows<c.value, false><<<(unsigned)rblocks, kRowT, RowGeom<c.value>::SMEM, st>>>(grid, qstride, nsum, q0,
                                                                                            (int)np, ly, buf);
    });
  }
  ARL_LAUNCH_CHECK();
  const int64_t ntile = ((int64_t)1 << (cg.log2N2 - cg.log2G1)) << (lx - cg.log2WC1 + 1);
  with_const<3, 7>(cg.log2N1, [&](auto c) {
    k_dsfft_cols1<c.value><<<(unsigned)(np * ntile), kWsT, col_smem(cg.log2N1, false) / 2, st>>>(buf, ly, lx, cg, ntile);
  });
  ARL_LAUNCH_CHECK();
  count_launch(2);
  return ARLGPU_OK;
}

// invert_2d: grid [nb][nw][ny][nx] FP32 complex -> image (real part, and the
// imaginary part when im_im is set); buf holds nb planes of float4.
int dsfft_g2i_2d(const float2 *grid, int nb, int nw, int ny, int nx, const double *gcf, const double *sumwt,
                 double *im_re, double *im_im, void *buf, cudaStream_t st) {
  const int ly = ilog2_exact(ny), lx = ilog2_exact(nx);
  ColGeom cg;
  if (!dsfft_supported(ny, nx) || !col_geom(ly, lx, &cg)) return fail(ARLGPU_ERR_UNSUPPORTED, "dsfft size");
  ARL_TRY(ensure_twiddles(st));
  ARL_TRY(set_smem());
  const int64_t plane = (int64_t)ny * nx;
  float4 *b4 = static_cast<float4 *>(buf);
  ARL_TRY(rows_cols1(grid, plane * nw, nw, 0, nb, ly, lx, cg, b4, st));
  const int64_t ntile = ((int64_t)1 << (cg.log2N1 - cg.log2G2)) << (lx - cg.log2WC2);
  const float s0 = (((nx / 2) + (ny / 2)) & 1) ? -1.f : 1.f;
  with_const<3, 7>(cg.log2N2, [&](auto c) {
    k_dsfft_cols2_image<c.value><<<(unsigned)(nb * ntile), kColT, col_smem(cg.log2N2, false), st>>>(
        b4, ly, lx, cg, ntile, 0, s0, gcf, sumwt, im_re, im_im);
  });
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

// w-stacking: grid [nb][K][ny][nx] FP32 complex; planes go through buf
// (room for G planes of float4) a group at a time; the image accumulates in
// double-single slots and is finished in place.
int dsfft_g2i_wstack(const float2 *grid, int nb, int K, int ny, int nx, double fov, const double *wmean,
                     const double *gcf, const double *sumwt, double *image, void *buf, int64_t G, cudaStream_t st) {
  const int ly = ilog2_exact(ny), lx = ilog2_exact(nx);
  ColGeom cg;
  if (!dsfft_supported(ny, nx) || !col_geom(ly, lx, &cg)) return fail(ARLGPU_ERR_UNSUPPORTED, "dsfft size");
  if (G < 1) return fail(ARLGPU_ERR_INVALID, "empty FFT group");
  ARL_TRY(ensure_twiddles(st));
  ARL_TRY(set_smem());
  const int64_t plane = (int64_t)ny * nx, nplanes = (int64_t)nb * K;
  float4 *b4 = static_cast<float4 *>(buf);
  const int64_t ntile = ((int64_t)1 << (cg.log2N1 - cg.log2G2)) << (lx - cg.log2WC2 + 1);
  for (int64_t p0 = 0; p0 < nplanes; p0 += G) {
    const int64_t np = std::min(G, nplanes - p0);
    ARL_TRY(rows_cols1(grid, plane, 1, p0, np, ly, lx, cg, b4, st));
    with_const<3, 7>(cg.log2N2, [&](auto c) {
      k_dsfft_cols2_wstack<c.value><<<(unsigned)ntile, kWsT, col_smem(cg.log2N2, true), st>>>(
          b4, ly, lx, cg, p0, p0 + np, K, fov, wmean, reinterpret_cast<float2 *>(image));
    });
    ARL_LAUNCH_CHECK();
    count_launch(1);
  }
  const float s0 = (((nx / 2) + (ny / 2)) & 1) ? -1.f : 1.f;
  for (int64_t b = 0; b < nb; b += 65535) {  // images along the grid's y
    const dim3 blocks((unsigned)std::min<int64_t>((plane + 255) / 256, 152 * 32), (unsigned)std::min<int64_t>(nb - b, 65535));
    k_ds_wstack_finish<<<blocks, 256, 0, st>>>(image + b * plane, ly, lx, s0, gcf + b * plane, sumwt + b);
    ARL_LAUNCH_CHECK();
  }
  ARL_LAUNCH_CHECK();
  count_launch(1);
  return ARLGPU_OK;
}

}  // namespace arlgpu
