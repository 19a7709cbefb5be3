// Double-single ("float-float") arithmetic: a value is the unevaluated sum
// hi + lo of two FP32 numbers with |lo| <= ulp(hi) / 2, about 48 significant
// bits.  GB300 runs FP32 at 64x its FP64 rate, so the FP32C path's transforms
// and w-screens use these instead of FP64.
//
// Published algorithms, written out here from the mathematics:
//   two_sum       Knuth, TAOCP vol. 2, 4.2.2 (error-free sum, 6 operations)
//   quick_two_sum Dekker 1971, "A floating-point technique for extending the
//                 available precision" (|a| >= |b|, 3 operations)
//   two_prod      the error-free product through one FMA
//   ds_sqrt       one Newton step on an FP32 root (Karp and Markstein, 1997)
//   ds_div        one correction step on an FP32 quotient
// Every FP32 operation is an explicit round-to-nearest intrinsic so the
// compiler cannot contract or reorder the error terms away.
#pragma once
#include <cuda_runtime.h>

namespace arlgpu {

struct dsf {
  float hi, lo;
};

__device__ __forceinline__ dsf two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float v = __fsub_rn(s, a);
  const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(b, v));
  return {s, e};
}

__device__ __forceinline__ dsf quick_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ dsf two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ dsf ds_add(dsf a, dsf b) {
  const dsf s = two_sum(a.hi, b.hi);
  return quick_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}

__device__ __forceinline__ dsf ds_neg(dsf a) { return {-a.hi, -a.lo}; }

__device__ __forceinline__ dsf ds_sub(dsf a, dsf b) { return ds_add(a, ds_neg(b)); }

__device__ __forceinline__ dsf ds_mul(dsf a, dsf b) {
  const dsf p = two_prod(a.hi, b.hi);
  const float e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
  return quick_two_sum(p.hi, e);
}

__device__ __forceinline__ dsf ds_mul_f(dsf a, float b) {
  const dsf p = two_prod(a.hi, b);
  return quick_two_sum(p.hi, __fmaf_rn(a.lo, b, p.lo));
}

// sqrt(a), a > 0: s0 = sqrtf(a.hi), s = s0 + (a - s0^2) / (2 s0).
__device__ __forceinline__ dsf ds_sqrt(dsf a) {
  if (!(a.hi > 0.f)) return {0.f, 0.f};
  const float s0 = sqrtf(a.hi);
  const dsf sq = two_prod(s0, s0);
  const float r = __fadd_rn(__fsub_rn(__fsub_rn(a.hi, sq.hi), sq.lo), a.lo);
  return quick_two_sum(s0, __fdiv_rn(r, __fmul_rn(2.f, s0)));
}

// a / b: q0 = a.hi / b.hi, q = q0 + (a - q0 b) / b.hi.
__device__ __forceinline__ dsf ds_div(dsf a, dsf b) {
  const float q0 = __fdiv_rn(a.hi, b.hi);
  const dsf qb = ds_mul_f(b, q0);
  const dsf r = ds_sub(a, qb);
  return quick_two_sum(q0, __fdiv_rn(r.hi, b.hi));
}

// Exact split of an integer |n| < 2^48.
__device__ __forceinline__ dsf ds_from_i64(long long n) {
  const float hi = (float)n;  // round to nearest
  return {hi, (float)(n - (long long)hi)};
}

__device__ __forceinline__ dsf ds_from_double(double x) {
  const float hi = __double2float_rn(x);
  return {hi, __double2float_rn(x - (double)hi)};
}

__device__ __forceinline__ double ds_to_double(dsf a) { return (double)a.hi + (double)a.lo; }

// cos and sin of (q + y / 2) quarter turns, |y| <= 1: y is the offset from
// quadrant q's centre in eighths of a turn.  Least-maximum fits of sin(pi y / 4) / y
// (degree 3 in y^2) and cos(pi y / 4) (degree 4), made for these intervals; pi / 4 is
// split so that its rounding does not scale the sine.  With the coefficients rounded
// to FP32 they are off by 3.6e-9 and 6.7e-9 at most, a ninth of FP32's half ulp at 1.
__device__ __forceinline__ void sincos_quadrant(float y, unsigned q, float *c, float *s) {
  const float z = y * y;
  float a = fmaf(z, -3.59545078e-05f, 2.49000713e-03f);
  a = fmaf(a, z, -8.07454348e-02f);
  a = fmaf(a, z, -2.4e-08f);  // pi / 4 = 0.78539818525 - 2.19e-8, less the fit's -2.1e-9
  const float sn = fmaf(y, 0.78539818525f, y * a);
  float b = fmaf(z, 3.52981134e-06f, -3.25938614e-04f);
  b = fmaf(b, z, 1.58543252e-02f);
  b = fmaf(b, z, -3.08425135e-01f);
  const float cs = fmaf(b, z, 1.f);
  const float cc = (q & 1) ? sn : cs, ss = (q & 1) ? cs : sn;
  *c = __int_as_float(__float_as_int(cc) ^ (((q + 1) & 2) << 30));
  *s = __int_as_float(__float_as_int(ss) ^ ((q & 2) << 30));
}

// w-screen phase of create_w_term_like at one pixel, in double-single:
// nterm = 1 - sqrt(1 - r^2), r^2 = c2 ((y - n/2)^2 + (x - n/2)^2) with
// c2 = fov^2 / n^2 (split from FP64).  The subtraction loses relative accuracy
// only where nterm is small, and there the phase w nterm is small too: its
// absolute error stays ~1e-14 w.
// state 0: r^2 == 0 (screen 1), 1: inside, 2: r^2 >= 1 (screen 0).
struct DsPix {
  dsf nterm;
  int state;
};
__device__ __forceinline__ DsPix ds_wpix(int y, int x, int n, dsf c2) {
  const long long dy = y - n / 2, dx = x - n / 2;
  const long long R = dy * dy + dx * dx;
  DsPix p;
  p.nterm = {0.f, 0.f};
  if (R == 0) {
    p.state = 0;
    return p;
  }
  const dsf r2 = ds_mul(c2, ds_from_i64(R));
  if (r2.hi > 1.f || (r2.hi == 1.f && r2.lo >= 0.f)) {
    p.state = 2;
    return p;
  }
  p.nterm = ds_sub({1.f, 0.f}, ds_sqrt(ds_sub({1.f, 0.f}, r2)));
  p.state = 1;
  return p;
}

// exp(-2 pi i w nterm) with the phase in turns reduced in double-single
// before an FP32 sincospi: the phase error is FP32 rounding of the reduced
// argument (< 1e-7 rad) for any w.
__device__ __forceinline__ float2 ds_wbeam(const DsPix &p, dsf w) {
  if (p.state == 0) return make_float2(1.f, 0.f);
  if (p.state == 2) return make_float2(0.f, 0.f);
  const dsf t = ds_mul(w, p.nterm);
  const float f = __fadd_rn(__fsub_rn(t.hi, rintf(t.hi)), t.lo);
  float s, c;
  sincospif(-2.f * f, &s, &c);
  return make_float2(c, s);
}

// Conversions through integer registers: GB300's FP64 unit retires 2
// conversions a clock and SM, its integer units 64 operations or more.  Both give
// the hardware conversion's value (to FP32: round to nearest, ties to even) and
// leave zeros, denormals, infinities and NaNs to it.
__device__ __forceinline__ double widen(double x) { return x; }
__device__ __forceinline__ double widen(float x) {
  const unsigned b = __float_as_uint(x), m = b & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u) return (double)x;
  return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __forceinline__ void narrow(double x, double *o) { *o = x; }
__device__ __forceinline__ void narrow(double x, float *o) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), m = hi & 0x7fffffffu;
  if (m - 0x38100000u >= 0x47e00000u - 0x38100000u) {  // outside [2^-126, 2^127)
    *o = (float)x;
    return;
  }
  unsigned f = ((m - 0x38000000u) << 3) | (lo >> 29);
  const unsigned rest = lo << 3;  // the 29 bits below, at the top of the word
  f += rest > 0x80000000u || (rest == 0x80000000u && (f & 1));
  *o = __uint_as_float((hi & 0x80000000u) | f);
}

// a / b for y = 1 / b rounded to nearest: after a correction step the quotient is
// within an ulp, and after a second one it is the rounded quotient (Markstein, IBM
// J. Res. Dev. 34, 1990, pp. 111-119).  Five operations
// instead of the division's 9 (throughput) and shorter dependence.  Outside the range
// where no step under- or overflows, the division itself.
__device__ __forceinline__ double rounded_quotient(double a, double b, double y) {
  const int ea = (__double2hiint(a) >> 20) & 0x7ff, eb = (__double2hiint(b) >> 20) & 0x7ff;
  if (ea < 1023 - 800 || ea > 1023 + 800 || eb < 1023 - 100 || eb > 1023 + 100) return __ddiv_rn(a, b);
  double q = __dmul_rn(a, y);
  q = fma(fma(-b, q, a), y, q);
  return fma(fma(-b, q, a), y, q);
}

}  // namespace arlgpu
