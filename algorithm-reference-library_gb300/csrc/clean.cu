// Hogbom CLEAN on the GPU.
//
// Reference behaviour:
//   hogbom, overlapIndices    processing_library/arrays/cleaners.py:12-69, :134-154
//   hogbom_complex            processing_library/arrays/cleaners.py:72-131
//   deconvolve_cube('hogbom') processing_components/image/deconvolution.py:43-300
//
// The real minor cycle is one cooperative launch (k_hogbom below); the complex
// and multi-scale ones are two launches per iteration on one stream, with no
// host round trip:
//   k_*_find  argmax over the image, first index on ties as numpy.argmax; the
//             last block to finish (counted with an atomic, no waiting) reduces
//             the per-block maxima and forms the component;
//   k_*_sub   the PSF patch subtracted, and the stopping test on the peak.
// A set stop flag turns the remaining launches into no-ops; the host reads
// the flag every kCheck iterations to stop launching.  All arithmetic is FP64
// with each operation rounded on its own (no FMA contraction), in the
// reference's order, so the result equals NumPy's bit for bit.
#include <algorithm>

#include "common.cuh"
#include "dsmath.cuh"

namespace arlgpu {

void count_launch(unsigned n);

struct Best {
  double v;
  long long i;
};

__device__ __forceinline__ Best better(Best a, Best b) {
  // larger value wins; on equal values the smaller index (numpy.argmax)
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

constexpr int kFindThreads = 256;

// ---------------------------------------------------------------------------
// Hogbom minor cycle, all iterations in one cooperative launch.
//
// As two launches per iteration (a search over the whole image, a subtraction)
// an iteration on 1024^2 with a 512^2 PSF took 22 us of GPU time and 30 us in
// all: the search alone spends three FP64 operations a pixel at 2 a clock and
// SM, and a launch costs more than the subtraction.  Here
//   * the image is cut into segments of 256 pixels of one row, dealt to the CTAs
//     in turn (an odd number of CTAs, so that a patch narrower than the image
//     still meets all of them); the residual stays in shared memory for the
//     whole cycle where it fits (about 2048^2), else in its global array;
//   * each segment's best pixel is kept, and only the segments that the PSF patch
//     touched are searched again, while they are updated.  |res * window| is
//     compared as integers, and a window of 0 or 1 (2-bit codes) takes no product;
//   * an iteration has one exchange: every CTA publishes its best pixel in a
//     16-byte slot and reads all the others', so all know the peak and need no
//     second barrier.  Both words of a slot carry their own generation mark (two
//     buffers in turn: nobody can be two iterations ahead), so that they need no
//     fence.  The wait is bounded; when it runs out the cycle ends with an error.
// What is left is the exchange (two L2 trips), one division and two FP64
// operations per pixel of the patch: 5.7 us an iteration (3.8 on 128^2).
// ---------------------------------------------------------------------------
constexpr int kHogThreads = 512, kHogSeg = 256, kHogPx = kHogSeg / 32;
constexpr unsigned long long kAbsMask = 0x7fffffffffffffffull;

// Copies of the slots, each polled by every kHogCopies-th CTA: with one, the
// 19 cache lines were read by all SMs at once and an iteration took 6.4 us on the
// smallest image.
constexpr int kHogCopies = 16;
constexpr int kHogPoll = 5;         // slots a polling lane reads: up to 160 CTAs
constexpr int kHogTries = 1 << 20;  // rounds of polling (about a microsecond each) before a CTA gives up

__device__ __forceinline__ void hog_put(unsigned long long *p, unsigned long long a, unsigned long long b) {
  asm volatile("st.volatile.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void hog_get(const unsigned long long *p, unsigned long long *a, unsigned long long *b) {
  asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(*a), "=l"(*b) : "l"(p) : "memory");
}

struct HogStatus {
  int iters, stop, error;
};

struct HogArgs {
  const double *src, *psf, *window;
  double *comps, *res;
  long long nx, ny, pnx, pny;
  double gain, pmax, stop_level;
  int niter, width, nloc;       // iterations of this launch, pixels per segment, segments per CTA (at most)
  unsigned long long *slots;    // [2][kHogCopies][gridDim.x][2]
  unsigned char *bests;         // the segments' bests of all CTAs where they do not fit shared memory, else null
  double *lookup;               // [2][gridDim.x]: the residual at a slot's pixel where |res| is not the slot's value
  HogStatus *status;
};

// A candidate: |res * window| as its bit pattern, and the pixel; first index on
// ties.  Where nothing qualifies (every value a NaN) the pixel stays kNoPixel.
constexpr int kNoPixel = 0x7fffffff;
__device__ __forceinline__ void hog_take(unsigned long long v, int i, unsigned long long *bv, int *bi) {
  if (v > *bv || (v == *bv && i < *bi)) {
    *bv = v;
    *bi = i;
  }
}

// The lane whose (v, key) is best: largest v, then smallest key.  Warp-wide
// 32-bit maxima and minima, a word at a time.
__device__ __forceinline__ bool hog_largest(unsigned long long v) {
  const unsigned all = 0xffffffffu, vh = (unsigned)(v >> 32), vl = (unsigned)v;
  const bool in = vh == __reduce_max_sync(all, vh);
  return (__reduce_max_sync(all, in ? vl : 0u) == vl) && in;
}
__device__ __forceinline__ int hog_best_lane(unsigned long long v, unsigned key) {
  const unsigned all = 0xffffffffu;
  const bool in = hog_largest(v);
  const unsigned k = __reduce_min_sync(all, in ? key : all);
  return __ffs(__ballot_sync(all, in && key == k)) - 1;
}
__device__ __forceinline__ int hog_best_lane(unsigned long long v, unsigned long long key) {
  const unsigned all = 0xffffffffu, kh = (unsigned)(key >> 32), kl = (unsigned)key;
  bool in = hog_largest(v);
  const unsigned h = __reduce_min_sync(all, in ? kh : all);
  in = in && kh == h;
  const unsigned l = __reduce_min_sync(all, in ? kl : all);
  return __ffs(__ballot_sync(all, in && kl == l)) - 1;
}

// |res * window| of one pixel; NaN results never qualify (marked all ones).
__device__ __forceinline__ unsigned long long hog_value(double r, int code, const double *win) {
  unsigned long long a = (unsigned long long)__double_as_longlong(r) & kAbsMask;
  if (code == 2) a = (unsigned long long)__double_as_longlong(__dmul_rn(r, *win)) & kAbsMask;
  if (code == 0) a = a >= 0x7ff0000000000000ull ? ~0ull : 0;
  return a > 0x7ff0000000000000ull ? ~0ull : a;
}

__device__ __forceinline__ int hog_code(double window) {
  const unsigned long long w = (unsigned long long)__double_as_longlong(window);
  return w == 0x3ff0000000000000ull ? 1 : ((w & kAbsMask) == 0 ? 0 : 2);
}

template <bool SMEM> struct HogPx { using T = int; };
template <> struct HogPx<true> { using T = unsigned short; };

template <bool SMEM>
__global__ void __launch_bounds__(kHogThreads, 1)
k_hogbom(HogArgs a) {
  extern __shared__ double s_dyn[];
  __shared__ unsigned long long s_bits, s_key;  // the iteration's peak
  __shared__ unsigned s_word;
  __shared__ double s_mval;
  __shared__ int s_stop, s_end;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, G = gridDim.x, cta = blockIdx.x;
  const int width = SMEM ? kHogSeg : a.width;
  // segments per row, in all (32-bit divisions below: the host keeps nseg below 2^31)
  const unsigned spr = (unsigned)((a.ny + width - 1) / width), nseg = (unsigned)a.nx * spr;
  // shared memory: [nloc][256] residual, [nloc][32] window codes (SMEM), then the segments' bests
  double *s_res = s_dyn;
  unsigned short *s_code = reinterpret_cast<unsigned short *>(s_dyn + (SMEM ? (size_t)a.nloc * kHogSeg : 0));
  unsigned long long *s_segv =
      reinterpret_cast<unsigned long long *>(s_dyn + (SMEM ? (size_t)a.nloc * (kHogSeg + 8) : 0));
  if (!SMEM && a.bests) s_segv = reinterpret_cast<unsigned long long *>(a.bests + (size_t)cta * a.nloc * 16);
  using Px = typename HogPx<SMEM>::T;
  constexpr Px kNone = (Px)kNoPixel;
  Px *s_segi = reinterpret_cast<Px *>(s_segv + a.nloc);

  // Local pixel p of segment i: offset p in [0, width) of segment cta + i G.
  // A segment's row: seg and spr stay below 2^15 where the residual is in shared memory, so that a high word does it.
  const unsigned inv = SMEM && spr > 1 ? 0xffffffffu / spr + 1 : 0;
  auto seg_div = [&](unsigned s) { return SMEM ? (spr > 1 ? __umulhi(s, inv) : s) : s / spr; };
  auto seg_row = [&](int i, long long *col) {
    const unsigned s = (unsigned)cta + (unsigned)i * G, row = seg_div(s);
    *col = (long long)(s - row * spr) * width;
    return (long long)row;
  };
  // Best pixel of segment i after subtracting mval * psf over columns [c0, c1) with the PSF pixel of column c at
  // prow[c] (null: no subtraction).  pre: the warp's PSF values when they are already in registers.
  auto scan = [&](int i, long long row, long long col, const double *prow, long long c0, long long c1, double mval,
                  const double *pre) {
    unsigned long long bv = 0;
    int bi = kNoPixel;
    const unsigned codes = SMEM && a.window ? s_code[i * 32 + lane] : 0x5555u;
    auto one = [&](int j, double r, double win) {
      const int p = lane + 32 * j;
      const long long c = col + p, px = row * a.ny + c;
      if (c >= a.ny) return;
      if (prow && c >= c0 && c < c1) {
        r = __dsub_rn(r, __dmul_rn(pre ? pre[j] : prow[c], mval));
        if (SMEM)
          s_res[i * kHogSeg + p] = r;
        else
          a.res[px] = r;
      }
      const int code = SMEM ? (codes >> (2 * j)) & 3 : hog_code(win);
      const unsigned long long v = hog_value(r, code, SMEM ? a.window + px : &win);
      if (v != ~0ull) hog_take(v, p, &bv, &bi);
    };
    if (SMEM) {
#pragma unroll
      for (int j = 0; j < kHogPx; ++j) one(j, s_res[i * kHogSeg + lane + 32 * j], 0.0);
    } else {  // eight pixels a lane at a time from global memory; the first search copies the image
      const double *from = prow ? a.res : a.src;
      for (int j0 = 0; j0 < width / 32; j0 += kHogPx) {
        double r[kHogPx], win[kHogPx];
#pragma unroll
        for (int j = 0; j < kHogPx; ++j) {
          const long long c = col + lane + 32 * (j0 + j);
          r[j] = c < a.ny ? from[row * a.ny + c] : 0.0;
          win[j] = a.window && c < a.ny ? a.window[row * a.ny + c] : 1.0;
        }
#pragma unroll
        for (int j = 0; j < kHogPx; ++j) {
          const long long c = col + lane + 32 * (j0 + j);
          if (from != a.res && c < a.ny) a.res[row * a.ny + c] = r[j];
          one(j0 + j, r[j], win[j]);
        }
      }
    }
    if (lane == hog_best_lane(bv, (unsigned)bi)) {
      s_segv[i] = bv;
      s_segi[i] = (Px)bi;
    }
  };

  const int mine = (unsigned)cta < nseg ? (int)((nseg - 1 - cta) / G) + 1 : 0;
  for (int i = warp; i < mine; i += kHogThreads / 32) {
    long long col;
    const long long row = seg_row(i, &col);
    if (SMEM) {
      unsigned codes = 0;
#pragma unroll
      for (int j = 0; j < kHogPx; ++j) {
        const long long c = col + lane + 32 * j;
        const bool in = c < a.ny;
        s_res[i * kHogSeg + lane + 32 * j] = in ? a.src[row * a.ny + c] : 0.0;
        codes |= (in && a.window ? hog_code(a.window[row * a.ny + c]) : 1) << (2 * j);
      }
      s_code[i * 32 + lane] = (unsigned short)codes;
    }
    scan(i, row, col, nullptr, 0, 0, 0.0, nullptr);
  }
  const long long wx = a.pnx / 2, wy = a.pny / 2;
  const double centre = a.psf[wx * a.pny + wy], rcp = __drcp_rn(a.pmax);
  __syncthreads();

  int it = 0;
  bool stop = false, dead = false;
  while (it < a.niter && !stop) {
    const int buf = it & 1;
    unsigned long long *slot = a.slots + 2ull * G * kHogCopies * buf;
    const unsigned long long mark = (unsigned long long)((it >> 1) & 1) << 63;
    if (warp == 0) {
      // This CTA's best pixel; its segments lie in the image's order.
      unsigned long long bv = 0;
      int bi = kNoPixel;
      for (int i = lane; i < mine; i += 32)
        if (s_segi[i] != kNone) hog_take(s_segv[i], i, &bv, &bi);
      int leader = hog_best_lane(bv, (unsigned)bi);
      unsigned long long w1 = 0;
      if (lane == leader) {
        unsigned word = 0x80000000u;  // bit 31: no pixel, bit 30: the residual is in lookup, bit 29: it is negative
        if (bi != kNoPixel) {
          const int p = s_segi[bi];
          double r;
          if (SMEM) {
            r = s_res[bi * kHogSeg + p];
          } else {
            long long col;
            const long long row = seg_row(bi, &col);
            r = a.res[row * a.ny + col + p];
          }
          const unsigned long long rb = (unsigned long long)__double_as_longlong(r);
          word = (unsigned)p;  // below 2^29
          if ((rb & kAbsMask) != bv) {
            word |= 0x40000000u;
            *(volatile double *)&a.lookup[(size_t)buf * G + cta] = r;
            __threadfence();
          } else if (rb >> 63) {
            word |= 0x20000000u;
          }
        }
        // word 0: value, mark; word 1: generation (8 bits; the slot's last one is it - 2), segment (24), word (32)
        w1 = (unsigned long long)((unsigned)(it & 0xff) << 24 | ((unsigned)bi & 0xffffffu)) << 32 | word;
      }
      bv = __shfl_sync(0xffffffffu, bv, leader);
      w1 = __shfl_sync(0xffffffffu, w1, leader);
      __syncwarp();  // orders the leader's lookup value and its fence before the other lanes' slots
      if (lane < kHogCopies) hog_put(slot + 2 * ((size_t)lane * G + cta), bv | mark, w1);
      // Everybody's best pixel, kHogPoll slots a lane, all loads of a round in flight together; the key (segment,
      // pixel in it) orders pixels as the image does.
      const unsigned long long *from = slot + 2 * (size_t)(cta % kHogCopies) * G;
      unsigned long long v = 0, key = ~0ull, w0[kHogPoll], w2[kHogPoll];
      unsigned word = 0x80000000u, todo = 0;
#pragma unroll
      for (int k = 0; k < kHogPoll; ++k) todo |= (lane + 32 * k < G ? 1u : 0u) << k;
      for (int tries = 0; __any_sync(0xffffffffu, todo) && tries < kHogTries; ++tries) {
#pragma unroll
        for (int k = 0; k < kHogPoll; ++k)
          if ((todo >> k) & 1) hog_get(from + 2 * (lane + 32 * k), &w0[k], &w2[k]);
#pragma unroll
        for (int k = 0; k < kHogPoll; ++k)
          if (((todo >> k) & 1) && (w0[k] & ~kAbsMask) == mark && (unsigned)(w2[k] >> 56) == (unsigned)(it & 0xff)) {
            todo &= ~(1u << k);
            const unsigned long long t = w0[k] & kAbsMask;
            const unsigned long long at =
                (unsigned long long)(lane + 32 * k + ((unsigned)(w2[k] >> 32) & 0xffffffu) * G) << 32 |
                ((unsigned)w2[k] & 0x1fffffffu);
            if (!((unsigned)w2[k] >> 31) && (t > v || (t == v && at < key))) {
              v = t;
              key = at;
              word = (unsigned)w2[k];
            }
          }
      }
      const bool late = __any_sync(0xffffffffu, todo);
      leader = hog_best_lane(v, key);
      if (lane == leader) {
        s_bits = v;
        s_key = key;
        s_word = word;
        s_end = late ? 2 : (int)(word >> 31);  // 1: no pixel qualifies
      }
    }
    __syncthreads();
    if (s_end) {
      dead = s_end == 2;
      break;
    }
    const unsigned long long key = s_key;
    const unsigned seg = (unsigned)(key >> 32);
    const unsigned mrow = seg_div(seg);
    const long long mx = mrow, my = (long long)(seg - mrow * spr) * width + (unsigned)key;
    if (threadIdx.x == 0) {
      const unsigned word = s_word;
      double r = __longlong_as_double((long long)(s_bits | ((unsigned long long)((word >> 29) & 1) << 63)));
      if ((word >> 30) & 1) {
        __threadfence();
        r = *(volatile double *)&a.lookup[(size_t)buf * G + seg % G];
      }
      s_mval = rounded_quotient(__dmul_rn(r, a.gain), a.pmax, rcp);
    }
    // The patch (overlapIndices of the reference): rows [r0, r1), columns [c0, c1), PSF pixel (x - mx + wx, y - my + wy).
    const long long r0 = max(0ll, mx - wx), r1 = min(a.nx, mx + wx);
    const long long c0 = max(0ll, my - wy), c1 = min(my + wy, a.ny);
    const int first = (int)r0 * (int)spr - cta, last = (int)r1 * (int)spr - cta;  // i G in [first, last)
    const int i0 = first > 0 ? (int)((unsigned)(first + G - 1) / G) : 0;
    const int i1 = last > 0 ? (int)((unsigned)(last + G - 1) / G) : 0;
    const int start = i0 + warp;
    double pre[kHogPx];
    if (SMEM && start < i1) {  // the first segment's PSF values come in while thread 0 divides
      long long col;
      const long long row = seg_row(start, &col);
      const double *prow = a.psf + (row - mx + wx) * a.pny + (wy - my);
#pragma unroll
      for (int j = 0; j < kHogPx; ++j) {
        const long long c = col + lane + 32 * j;
        pre[j] = c >= c0 && c < c1 ? prow[c] : 0.0;
      }
    }
    __syncthreads();
    const double mval = s_mval;
    if (threadIdx.x == kHogThreads - 1) {
      // the last warp, which has a segment least often: the component, and the stopping test on the updated peak
      const unsigned word = s_word;
      double r = __longlong_as_double((long long)(s_bits | ((unsigned long long)((word >> 29) & 1) << 63)));
      if ((word >> 30) & 1) r = *(volatile double *)&a.lookup[(size_t)buf * G + seg % G];
      s_stop = fabs(__dsub_rn(r, __dmul_rn(centre, mval))) < a.stop_level;
      if (seg % G == (unsigned)cta) a.comps[mx * a.ny + my] = __dadd_rn(a.comps[mx * a.ny + my], mval);
    }
    for (int i = start; i < i1; i += kHogThreads / 32) {
      long long col;
      const long long row = seg_row(i, &col);
      if (col >= c1 || col + width <= c0) continue;
      scan(i, row, col, a.psf + (row - mx + wx) * a.pny + (wy - my), c0, c1, mval, SMEM && i == start ? pre : nullptr);
    }
    ++it;
    __syncthreads();
    stop = s_stop;
  }
  if (SMEM)
    for (int i = warp; i < mine; i += kHogThreads / 32) {
      long long col;
      const long long row = seg_row(i, &col);
      for (int p = lane; p < kHogSeg && col + p < a.ny; p += 32) a.res[row * a.ny + col + p] = s_res[i * kHogSeg + p];
    }
  if (cta == 0 && threadIdx.x == 0) {
    a.status->iters = it;
    a.status->stop = stop || it < a.niter;
  }
  if (dead && threadIdx.x == 0) a.status->error = 1;
}

// ---------------------------------------------------------------------------
// Complex Hogbom CLEAN of Q + iU (processing_library/arrays/cleaners.py:72-131):
// the same two launches per iteration on a residual held as two planes
// (real, imaginary).  The peak is the first largest |res * window| (or |res|)
// with |.| the hypotenuse of the two parts, as numpy.absolute; the component
// res[peak] * gain / pmax and the PSF subtraction are taken part by part
// (the PSF is real), and the loop stops when |res[peak]| after the
// subtraction falls below the threshold itself (no 0.9 factor here).
// ---------------------------------------------------------------------------
struct HogCState {
  double mre, mim;
  long long peak;
  int stop;
  int iters;
  unsigned int counter;
};

__global__ void __launch_bounds__(kFindThreads)
k_hogc_find(const double *__restrict__ rre, const double *__restrict__ rim, const double *__restrict__ window,
            long long n, double gain, double pmax, double *__restrict__ cre, double *__restrict__ cim,
            Best *__restrict__ partial, HogCState *__restrict__ st) {
  if (st->stop) return;
  __shared__ Best s_best[kFindThreads / 32];
  __shared__ bool s_last;
  Best b{-1.0, 0x7fffffffffffffffll};
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double a = window ? hypot(__dmul_rn(rre[i], window[i]), __dmul_rn(rim[i], window[i])) : hypot(rre[i], rim[i]);
    b = better(b, Best{a, i});
  }
  for (int o = 16; o > 0; o >>= 1) {
    Best c;
    c.v = __shfl_xor_sync(0xffffffffu, b.v, o);
    c.i = __shfl_xor_sync(0xffffffffu, b.i, o);
    b = better(b, c);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_best[warp] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    Best t = s_best[0];
    for (int k = 1; k < kFindThreads / 32; ++k) t = better(t, s_best[k]);
    partial[blockIdx.x] = t;
    __threadfence();
    s_last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  Best t{-1.0, 0x7fffffffffffffffll};
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    Best q;
    q.v = __ldcg(&partial[k].v);
    q.i = __ldcg(&partial[k].i);
    t = better(t, q);
  }
  for (int o = 16; o > 0; o >>= 1) {
    Best c;
    c.v = __shfl_xor_sync(0xffffffffu, t.v, o);
    c.i = __shfl_xor_sync(0xffffffffu, t.i, o);
    t = better(t, c);
  }
  if (lane == 0) s_best[warp] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    Best f = s_best[0];
    for (int k = 1; k < kFindThreads / 32; ++k) f = better(f, s_best[k]);
    const double mre = __ddiv_rn(__dmul_rn(rre[f.i], gain), pmax);
    const double mim = __ddiv_rn(__dmul_rn(rim[f.i], gain), pmax);
    cre[f.i] = __dadd_rn(cre[f.i], mre);
    cim[f.i] = __dadd_rn(cim[f.i], mim);
    st->mre = mre;
    st->mim = mim;
    st->peak = f.i;
    st->counter = 0;
  }
}

__global__ void k_hogc_sub(double *__restrict__ rre, double *__restrict__ rim, int nx, int ny,
                           const double *__restrict__ psf, int pnx, int pny, double stop_level,
                           HogCState *__restrict__ st) {
  if (st->stop) return;
  const long long peak = st->peak;
  const int mx = (int)(peak / ny), my = (int)(peak - (long long)mx * ny);
  const double mre = st->mre, mim = st->mim;
  const int wx = pnx / 2, wy = pny / 2;
  const int r0 = max(0, mx - wx), r1 = min(nx, mx + wx);
  const int c0 = max(0, my - wy), c1 = min(my + wy, ny);
  const int p0 = max(0, wx + (r0 - mx)), q0 = max(0, wy + (c0 - my));
  const int p1 = min(pnx, wx + (r1 - mx)), q1 = min(wy + (c1 - my), pny);
  const int h = min(r1 - r0, p1 - p0), w = min(c1 - c0, q1 - q0);
  const long long total = (long long)h * w;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / w), j = (int)(k - (long long)i * w);
    const long long ri = (long long)(r0 + i) * ny + (c0 + j);
    const double pv = psf[(long long)(p0 + i) * pny + (q0 + j)];
    const double nre = __dsub_rn(rre[ri], __dmul_rn(pv, mre));
    const double nim = __dsub_rn(rim[ri], __dmul_rn(pv, mim));
    rre[ri] = nre;
    rim[ri] = nim;
    if (ri == peak) {
      st->iters += 1;
      if (hypot(nre, nim) < stop_level) st->stop = 1;
    }
  }
}

// ---------------------------------------------------------------------------
// Multi-scale multi-frequency CLEAN minor cycle (processing_library/arrays/
// cleaners.py:469-600 with find_global_optimum :601-634,
// update_scale_moment_residual :636-646, update_moment_model :648-661,
// calculate_scale_moment_principal_solution :722-735 and
// find_optimum_scale_zero_moment :738-767).  Inputs from the set-up: the
// scale-moment residual smres [ns][nm][n0][n1], the scale-scale-moment-moment
// PSF ssm [ns][ns][nm][nm][p0][p1], the PSF-sized scale images pscale
// [ns][p0][p1], an optional window stack [ns][n0][n1] and the moment-moment
// Hessian and its inverse [ns][nm][nm].  Per iteration:
//   k_mfs_find  for each scale, the principal solution
//               smpsol[s][n] = sum_m ih[s][m][n] smres[s][m] at every pixel and
//               the search image (ARL: smpsol[s][0] smres[s][0]; Algorithm1:
//               smpsol[s][0]; CASA: the chi^2 change); the scale whose search
//               image has the largest |. * window| (first scale on ties, 0 if
//               none exceeds 0) wins, at the first largest signed (unwindowed)
//               search value -- the reference's argmax; the last block forms
//               mval = smpsol[scale][:, peak] and stops the loop when
//               max |mval| falls below the threshold;
//   k_mfs_sub   smres[:, :, lhs] -= gain * sum_q ssm[scale, :, :, q, rhs] mval[q]
//               and model[t, lhs] += pscale[scale, rhs] * gain * mval[t].
// FP64 with each operation rounded on its own, in the reference's order.
// ---------------------------------------------------------------------------
constexpr int kMfsMaxScales = 16, kMfsMaxMoments = 8;

struct MfsState {
  double mval[kMfsMaxMoments];
  long long peak;
  int scale;
  int stop;
  int iters;
  unsigned int counter;
};

struct MfsBest {
  double absmax;  // largest |search * window| (value only)
  Best vmax;      // first largest signed search value
};

__device__ __forceinline__ void mfs_solution(const double *__restrict__ smres, const double *__restrict__ ihess,
                                             int s, int nm, long long plane, long long i, double *sol) {
  // einsum("smn,smxy->snxy"): sum over m in order
  for (int n = 0; n < nm; ++n) {
    double acc = 0.0;
    for (int m = 0; m < nm; ++m)
      acc = __dadd_rn(acc, __dmul_rn(ihess[(s * nm + m) * nm + n], smres[((long long)s * nm + m) * plane + i]));
    sol[n] = acc;
  }
}

__device__ __forceinline__ double mfs_search(const double *__restrict__ smres, const double *__restrict__ hess,
                                             const double *sol, int s, int nm, long long plane, long long i,
                                             int findpeak) {
  if (findpeak == 1) return sol[0];  // Algorithm1
  if (findpeak == 2) {               // CASA: dchisq
    double d = 0.0;
    for (int m1 = 0; m1 < nm; ++m1) {
      d = __dadd_rn(d, __dmul_rn(__dmul_rn(2.0, sol[m1]), smres[((long long)s * nm + m1) * plane + i]));
      for (int m2 = 0; m2 < nm; ++m2)
        d = __dsub_rn(d, __dmul_rn(__dmul_rn(hess[(s * nm + m1) * nm + m2], sol[m1]), sol[m2]));
    }
    return d;
  }
  return __dmul_rn(sol[0], smres[(long long)s * nm * plane + i]);  // ARL
}

__global__ void __launch_bounds__(kFindThreads)
k_mfs_find(const double *__restrict__ smres, const double *__restrict__ windowstack, const double *__restrict__ hess,
           const double *__restrict__ ihess, int ns, int nm, long long plane, int findpeak, double absthresh,
           MfsBest *__restrict__ partial, MfsState *__restrict__ st) {
  if (st->stop) return;
  __shared__ double s_abs[kFindThreads / 32];
  __shared__ Best s_best[kFindThreads / 32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double sol[kMfsMaxMoments];
  for (int s = 0; s < ns; ++s) {
    double am = 0.0;
    Best b{-INFINITY, 0x7fffffffffffffffll};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < plane;
         i += (long long)gridDim.x * blockDim.x) {
      mfs_solution(smres, ihess, s, nm, plane, i, sol);
      const double v = mfs_search(smres, hess, sol, s, nm, plane, i, findpeak);
      const double vw = windowstack ? __dmul_rn(v, windowstack[(long long)s * plane + i]) : v;
      am = fmax(am, fabs(vw));
      b = better(b, Best{v, i});
    }
    for (int o = 16; o > 0; o >>= 1) {
      am = fmax(am, __shfl_xor_sync(0xffffffffu, am, o));
      Best c;
      c.v = __shfl_xor_sync(0xffffffffu, b.v, o);
      c.i = __shfl_xor_sync(0xffffffffu, b.i, o);
      b = better(b, c);
    }
    if (lane == 0) {
      s_abs[warp] = am;
      s_best[warp] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      MfsBest t{s_abs[0], s_best[0]};
      for (int k = 1; k < kFindThreads / 32; ++k) {
        t.absmax = fmax(t.absmax, s_abs[k]);
        t.vmax = better(t.vmax, s_best[k]);
      }
      partial[(long long)blockIdx.x * ns + s] = t;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x != 0) return;
  // Last block, one thread: per scale the reduction over blocks, then the
  // scale search of find_optimum_scale_zero_moment.
  __threadfence();
  double optimum = 0.0;
  int sscale = 0;
  long long sidx = 0;
  for (int s = 0; s < ns; ++s) {
    double am = 0.0;
    Best b{-INFINITY, 0x7fffffffffffffffll};
    for (int k = 0; k < (int)gridDim.x; ++k) {
      const MfsBest *q = &partial[(long long)k * ns + s];
      am = fmax(am, __ldcg(&q->absmax));
      b = better(b, Best{__ldcg(&q->vmax.v), __ldcg(&q->vmax.i)});
    }
    if (am > optimum) {
      optimum = am;
      sscale = s;
      sidx = b.i;
    }
  }
  mfs_solution(smres, ihess, sscale, nm, plane, sidx, sol);
  double peak = 0.0;
  for (int n = 0; n < nm; ++n) {
    st->mval[n] = sol[n];
    peak = fmax(peak, fabs(sol[n]));
  }
  st->scale = sscale;
  st->peak = sidx;
  st->counter = 0;
  st->iters += 1;
  if (peak < absthresh) st->stop = 2;  // stop before this iteration's update
}

__global__ void k_mfs_sub(double *__restrict__ smres, double *__restrict__ model, const double *__restrict__ ssm,
                          const double *__restrict__ pscale, int ns, int nm, int n0, int n1, int p0n, int p1n,
                          double gain, MfsState *__restrict__ st) {
  if (st->stop) return;
  const long long peak = st->peak;
  const int mx = (int)(peak / n1), my = (int)(peak - (long long)mx * n1);
  const int ms = st->scale;
  const int wx = p0n / 2, wy = p1n / 2;
  const int r0 = max(0, mx - wx), r1 = min(n0, mx + wx);
  const int c0 = max(0, my - wy), c1 = min(my + wy, n1);
  const int q0 = max(0, wx + (r0 - mx)), s0 = max(0, wy + (c0 - my));
  const int q1 = min(p0n, wx + (r1 - mx)), s1 = min(wy + (c1 - my), p1n);
  const int h = min(r1 - r0, q1 - q0), w = min(c1 - c0, s1 - s0);
  const long long plane = (long long)n0 * n1, pplane = (long long)p0n * p1n;
  const long long total = (long long)h * w;
  double mv[kMfsMaxMoments];
  for (int t = 0; t < nm; ++t) mv[t] = st->mval[t];
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / w), j = (int)(k - (long long)i * w);
    const long long ri = (long long)(r0 + i) * n1 + (c0 + j);
    const long long pi = (long long)(q0 + i) * p1n + (s0 + j);
    for (int s = 0; s < ns; ++s)
      for (int t = 0; t < nm; ++t) {
        double acc = 0.0;  // einsum("stqxy,q->stxy"): sum over q in order
        for (int q = 0; q < nm; ++q)
          acc = __dadd_rn(acc, __dmul_rn(ssm[((((long long)ms * ns + s) * nm + t) * nm + q) * pplane + pi], mv[q]));
        double *r = smres + ((long long)s * nm + t) * plane + ri;
        *r = __dsub_rn(*r, __dmul_rn(gain, acc));
      }
    const double ps = pscale[(long long)ms * pplane + pi];
    for (int t = 0; t < nm; ++t) {
      double *m = model + (long long)t * plane + ri;
      *m = __dadd_rn(*m, __dmul_rn(__dmul_rn(ps, gain), mv[t]));
    }
  }
}

// ---------------------------------------------------------------------------
// Multiscale CLEAN (processing_library/arrays/cleaners.py:165-280): the
// minor-cycle loop over the scale stack.  The scale images, the twice-
// convolved PSF stack and the coupling matrix come from the caller (the
// reference forms them with NumPy FFTs).  Per iteration:
//   k_ms_find  argmax over scales and pixels of |stack_s * window_s / c_ss|,
//              ties to the lower scale, then the lower index (the reference
//              scans scales in order and keeps a strictly larger value); the
//              last block applies the stopping tests (|stack[peak]| below
//              0.9 * threshold, or a zero component) and forms mval;
//   k_ms_sub   stack_s[overlap] -= psf_ss[s, mscale][overlap] * gain * mval for
//              every scale, comps[overlap] += pscale[mscale][overlap] * gain * mval.
// ---------------------------------------------------------------------------
struct MsState {
  double mval;
  long long peak;  // flat pixel index
  int mscale;
  int stop;
  int iters;
  unsigned int counter;
};

struct BestS {
  double v;
  long long key;  // scale * npix + pixel: lower key wins ties
};

__device__ __forceinline__ BestS better_s(BestS a, BestS b) {
  if (b.v > a.v || (b.v == a.v && b.key < a.key)) return b;
  return a;
}

__global__ void __launch_bounds__(kFindThreads)
k_ms_find(const double *__restrict__ stack, const double *__restrict__ wstack, const double *__restrict__ coupling,
          int ns, long long npix, double stop_level, BestS *__restrict__ partial, MsState *__restrict__ st) {
  if (st->stop) return;
  __shared__ BestS s_best[kFindThreads / 32];
  __shared__ bool s_last;
  BestS b{-1.0, 0x7fffffffffffffffll};
  const long long total = (long long)ns * npix;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += (long long)gridDim.x * blockDim.x) {
    const int sc = (int)(k / npix);
    const double c = coupling[sc * ns + sc];
    const double v = wstack ? __dmul_rn(stack[k], wstack[k]) : stack[k];
    b = better_s(b, BestS{fabs(__ddiv_rn(v, c)), k});
  }
  for (int o = 16; o > 0; o >>= 1) {
    BestS c;
    c.v = __shfl_xor_sync(0xffffffffu, b.v, o);
    c.key = __shfl_xor_sync(0xffffffffu, b.key, o);
    b = better_s(b, c);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_best[warp] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    BestS t = s_best[0];
    for (int k = 1; k < kFindThreads / 32; ++k) t = better_s(t, s_best[k]);
    partial[blockIdx.x] = t;
    __threadfence();
    s_last = atomicAdd(&st->counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  BestS t{-1.0, 0x7fffffffffffffffll};
  for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
    BestS q;  // other blocks' results: read past L1
    q.v = __ldcg(&partial[k].v);
    q.key = __ldcg(&partial[k].key);
    t = better_s(t, q);
  }
  for (int o = 16; o > 0; o >>= 1) {
    BestS c;
    c.v = __shfl_xor_sync(0xffffffffu, t.v, o);
    c.key = __shfl_xor_sync(0xffffffffu, t.key, o);
    t = better_s(t, c);
  }
  if (lane == 0) s_best[warp] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    BestS f = s_best[0];
    for (int k = 1; k < kFindThreads / 32; ++k) f = better_s(f, s_best[k]);
    const int sc = (int)(f.key / npix);
    const double r = stack[f.key];
    const double mval = __ddiv_rn(r, coupling[sc * ns + sc]);
    st->counter = 0;
    st->iters += 1;
    if (fabs(r) < stop_level || !(fabs(mval) > 0.0)) {
      st->stop = 1;
      return;
    }
    st->mval = mval;
    st->mscale = sc;
    st->peak = f.key - (long long)sc * npix;
  }
}

__global__ void k_ms_sub(double *__restrict__ stack, double *__restrict__ comps, int ns, int nx, int ny,
                         const double *__restrict__ psf_ss, const double *__restrict__ pscale, int pnx, int pny,
                         double gain, MsState *__restrict__ st) {
  if (st->stop) return;
  const long long peak = st->peak;
  const int mscale = st->mscale;
  const int mx = (int)(peak / ny), my = (int)(peak - (long long)mx * ny);
  const double mval = st->mval;
  const int wx = pnx / 2, wy = pny / 2;
  const int r0 = max(0, mx - wx), r1 = min(nx, mx + wx);
  const int c0 = max(0, my - wy), c1 = min(my + wy, ny);
  const int p0 = max(0, wx + (r0 - mx)), q0 = max(0, wy + (c0 - my));
  const int p1 = min(pnx, wx + (r1 - mx)), q1 = min(wy + (c1 - my), pny);
  const int h = min(r1 - r0, p1 - p0), w = min(c1 - c0, q1 - q0);
  const long long patch = (long long)h * w, total = patch * (ns + 1);
  const long long npix = (long long)nx * ny, ppix = (long long)pnx * pny;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
       k += (long long)gridDim.x * blockDim.x) {
    const int slot = (int)(k / patch);
    const long long e = k - (long long)slot * patch;
    const int i = (int)(e / w), j = (int)(e - (long long)i * w);
    const long long ri = (long long)(r0 + i) * ny + (c0 + j);
    const long long pi = (long long)(p0 + i) * pny + (q0 + j);
    if (slot < ns) {
      const double d = __dmul_rn(__dmul_rn(psf_ss[((long long)slot * ns + mscale) * ppix + pi], gain), mval);
      stack[slot * npix + ri] = __dsub_rn(stack[slot * npix + ri], d);
    } else {
      const double d = __dmul_rn(__dmul_rn(pscale[(long long)mscale * ppix + pi], gain), mval);
      comps[ri] = __dadd_rn(comps[ri], d);
    }
  }
}

static int nblk(long long n, int cap) {
  long long b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace arlgpu

using namespace arlgpu;

extern "C" int arlgpu_hogbom(const double *dirty, const double *psf, const double *window, int32_t nx, int32_t ny,
                             int32_t psf_nx, int32_t psf_ny, double gain, double thresh, int32_t niter,
                             double fracthresh, double dirty_absmax, double psf_max, double *comps, double *res,
                             int32_t *iterations, void *stream) {
  if (!dirty || !psf || !comps || !res || !iterations) return fail(ARLGPU_ERR_INVALID, "null array argument");
  if (nx < 1 || ny < 1 || psf_nx < 2 || psf_ny < 2) return fail(ARLGPU_ERR_INVALID, "bad image or psf shape");
  if (!(gain > 0.0 && gain < 2.0)) return fail(ARLGPU_ERR_INVALID, "gain must be in (0, 2)");
  if (niter < 1) return fail(ARLGPU_ERR_INVALID, "niter must be > 0");
  if (!(psf_max > 0.0)) return fail(ARLGPU_ERR_INVALID, "psf maximum must be > 0");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long n = (long long)nx * ny;
  const double absthresh = fmax(thresh, fracthresh * dirty_absmax);
  HogArgs args{};
  args.psf = psf;
  args.window = window;
  args.comps = comps;
  args.res = res;
  args.nx = nx;
  args.ny = ny;
  args.pnx = psf_nx;
  args.pny = psf_ny;
  args.gain = gain;
  args.pmax = psf_max;
  args.stop_level = 0.9 * absthresh;
  int dev = 0, sms = 0, smem_max = 0;
  ARL_CUDA(cudaGetDevice(&dev));
  ARL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ARL_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const long long odd = std::min((sms - 1) | 1, 32 * kHogPoll - 1);
  // The residual in shared memory where it fits, in 256-pixel segments; else in
  // global memory, in segments wide enough for 8192 to serve a CTA.
  auto segments = [&](long long width) { return (long long)nx * ((ny + width - 1) / width); };
  long long width = kHogSeg, ctas = std::min(odd, segments(width));
  long long nloc = (segments(width) + ctas - 1) / ctas;
  const size_t statics = 1024;  // at least the kernel's static shared memory
  size_t smem = (size_t)nloc * (kHogSeg * 8 + 64 + 10);
  const bool in_smem = smem + statics <= (size_t)smem_max;
  if (!in_smem) {
    while ((segments(width) + odd - 1) / odd > 8192 && width < ny) width <<= 1;
    ctas = std::min(odd, segments(width));
    nloc = (segments(width) + ctas - 1) / ctas;
    smem = (size_t)nloc * 12;
    if (smem + statics > (size_t)smem_max) smem = 0;  // a tall, narrow image: the bests in global memory
  }
  args.width = (int)width;
  args.nloc = (int)nloc;
  const void *kern = in_smem ? (const void *)k_hogbom<true> : (const void *)k_hogbom<false>;
  ARL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - (int)statics));
  // status, then the slots and the lookup values
  const size_t slot_bytes = (size_t)ctas * kHogCopies * 2 * 2 * sizeof(unsigned long long);
  const size_t bests = smem ? 0 : (size_t)ctas * nloc * 16;
  const size_t bytes = 16 + slot_bytes + (size_t)ctas * 2 * sizeof(double) + bests;
  char *ws = nullptr;
  ARL_CUDA(cudaMallocAsync(&ws, bytes, st));
  args.status = reinterpret_cast<HogStatus *>(ws);
  args.slots = reinterpret_cast<unsigned long long *>(ws + 16);
  args.lookup = reinterpret_cast<double *>(ws + 16 + slot_bytes);
  args.bests = bests ? reinterpret_cast<unsigned char *>(args.lookup + 2 * ctas) : nullptr;
  int rc = ARLGPU_OK, done = 0;
  HogStatus hs{};
  if (cudaMemsetAsync(comps, 0, sizeof(double) * n, st) != cudaSuccess) rc = fail(ARLGPU_ERR_CUDA, "hogbom set-up failed");
  args.src = dirty;
  constexpr int kBatch = 20000;  // iterations per launch: some tens of milliseconds
  while (rc == ARLGPU_OK && done < niter && !hs.stop) {
    args.niter = std::min(niter - done, kBatch);
    void *params[] = {&args};
    if (cudaMemsetAsync(args.status, 0, sizeof(HogStatus), st) != cudaSuccess ||
        cudaMemsetAsync(args.slots, 0xff, slot_bytes, st) != cudaSuccess ||
        cudaLaunchCooperativeKernel(kern, dim3((unsigned)ctas), dim3(kHogThreads), params, smem, st) != cudaSuccess) {
      rc = fail(ARLGPU_ERR_CUDA, "hogbom launch failed: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    count_launch(1);
    if (cudaMemcpyAsync(&hs, args.status, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      rc = fail(ARLGPU_ERR_CUDA, "hogbom state read failed");
    else if (hs.error)
      rc = fail(ARLGPU_ERR_CUDA, "hogbom: a CTA waited too long for the others");
    done += hs.iters;
    args.src = res;
  }
  *iterations = done;
  cudaFreeAsync(ws, st);
  return rc;
}

extern "C" int arlgpu_hogbom_complex(const double *dirty_q, const double *dirty_u, const double *psf,
                                     const double *window, int32_t nx, int32_t ny, int32_t psf_nx, int32_t psf_ny,
                                     double gain, double thresh, int32_t niter, double fracthresh,
                                     double dirty_absmax, double psf_max, double *comps_q, double *comps_u,
                                     double *res_q, double *res_u, int32_t *iterations, void *stream) {
  if (!dirty_q || !dirty_u || !psf || !comps_q || !comps_u || !res_q || !res_u || !iterations)
    return fail(ARLGPU_ERR_INVALID, "null array argument");
  if (nx < 1 || ny < 1 || psf_nx < 2 || psf_ny < 2) return fail(ARLGPU_ERR_INVALID, "bad image or psf shape");
  if (!(gain > 0.0 && gain < 2.0)) return fail(ARLGPU_ERR_INVALID, "gain must be in (0, 2)");
  if (niter < 1) return fail(ARLGPU_ERR_INVALID, "niter must be > 0");
  if (!(psf_max > 0.0)) return fail(ARLGPU_ERR_INVALID, "psf maximum must be > 0");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long n = (long long)nx * ny;
  const int fblocks = nblk(n, 152 * 4);
  const int sblocks = nblk((long long)psf_nx * psf_ny, 152 * 8);
  HogCState *state = nullptr;
  Best *partial = nullptr;
  ARL_CUDA(cudaMallocAsync(&state, sizeof(HogCState), st));
  int rc = ARLGPU_OK;
  if (cudaMallocAsync(&partial, sizeof(Best) * fblocks, st) != cudaSuccess) {
    cudaFreeAsync(state, st);
    return fail(ARLGPU_ERR_CUDA, "cudaMallocAsync failed");
  }
  const double absthresh = fmax(thresh, fracthresh * dirty_absmax);
  constexpr int kCheck = 64;
  int it = 0;
  HogCState hs{};
  do {
    if (cudaMemsetAsync(state, 0, sizeof(HogCState), st) != cudaSuccess ||
        cudaMemcpyAsync(res_q, dirty_q, sizeof(double) * n, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(res_u, dirty_u, sizeof(double) * n, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
        cudaMemsetAsync(comps_q, 0, sizeof(double) * n, st) != cudaSuccess ||
        cudaMemsetAsync(comps_u, 0, sizeof(double) * n, st) != cudaSuccess) {
      rc = fail(ARLGPU_ERR_CUDA, "hogbom_complex set-up failed");
      break;
    }
    while (it < niter) {
      const int batch = niter - it < kCheck ? niter - it : kCheck;
      for (int k = 0; k < batch; ++k) {
        k_hogc_find<<<fblocks, kFindThreads, 0, st>>>(res_q, res_u, window, n, gain, psf_max, comps_q, comps_u,
                                                       partial, state);
        k_hogc_sub<<<sblocks, 256, 0, st>>>(res_q, res_u, nx, ny, psf, psf_nx, psf_ny, absthresh, state);
      }
      count_launch(2 * batch);
      it += batch;
      if (cudaGetLastError() != cudaSuccess) {
        rc = fail(ARLGPU_ERR_CUDA, "hogbom_complex launch failed");
        break;
      }
      if (cudaMemcpyAsync(&hs, state, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess) {
        rc = fail(ARLGPU_ERR_CUDA, "hogbom_complex state read failed");
        break;
      }
      if (hs.stop) break;
    }
  } while (false);
  *iterations = hs.iters;
  cudaFreeAsync(partial, st);
  cudaFreeAsync(state, st);
  return rc;
}

extern "C" int arlgpu_msmfsclean(double *smres, const double *ssm, const double *pscale, const double *windowstack,
                                 const double *hess, const double *ihess, int32_t nscales, int32_t nmoment,
                                 int32_t n0, int32_t n1, int32_t psf_n0, int32_t psf_n1, double gain, double absthresh,
                                 int32_t niter, int32_t findpeak, double *model, int32_t *iterations, void *stream) {
  if (!smres || !ssm || !pscale || !hess || !ihess || !model || !iterations)
    return fail(ARLGPU_ERR_INVALID, "null array argument");
  if (nscales < 1 || nscales > kMfsMaxScales || nmoment < 1 || nmoment > kMfsMaxMoments)
    return fail(ARLGPU_ERR_UNSUPPORTED, "msmfsclean takes 1..%d scales and 1..%d moments", kMfsMaxScales,
                kMfsMaxMoments);
  if (n0 < 1 || n1 < 1 || psf_n0 < 2 || psf_n1 < 2) return fail(ARLGPU_ERR_INVALID, "bad image or psf shape");
  if (!(gain > 0.0 && gain < 2.0)) return fail(ARLGPU_ERR_INVALID, "gain must be in (0, 2)");
  if (niter < 1) return fail(ARLGPU_ERR_INVALID, "niter must be > 0");
  if (findpeak < 0 || findpeak > 2) return fail(ARLGPU_ERR_INVALID, "findpeak must be 0 (ARL), 1 (Algorithm1), 2 (CASA)");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long plane = (long long)n0 * n1;
  const int fblocks = nblk(plane, 152 * 2);
  const int sblocks = nblk((long long)psf_n0 * psf_n1, 152 * 8);
  MfsState *state = nullptr;
  MfsBest *partial = nullptr;
  ARL_CUDA(cudaMallocAsync(&state, sizeof(MfsState), st));
  int rc = ARLGPU_OK;
  if (cudaMallocAsync(&partial, sizeof(MfsBest) * fblocks * nscales, st) != cudaSuccess) {
    cudaFreeAsync(state, st);
    return fail(ARLGPU_ERR_CUDA, "cudaMallocAsync failed");
  }
  constexpr int kCheck = 32;
  int it = 0;
  MfsState hs{};
  do {
    if (cudaMemsetAsync(state, 0, sizeof(MfsState), st) != cudaSuccess ||
        cudaMemsetAsync(model, 0, sizeof(double) * plane * nmoment, st) != cudaSuccess) {
      rc = fail(ARLGPU_ERR_CUDA, "msmfsclean set-up failed");
      break;
    }
    while (it < niter) {
      const int batch = niter - it < kCheck ? niter - it : kCheck;
      for (int k = 0; k < batch; ++k) {
        k_mfs_find<<<fblocks, kFindThreads, 0, st>>>(smres, windowstack, hess, ihess, nscales, nmoment, plane,
                                                      findpeak, absthresh, partial, state);
        k_mfs_sub<<<sblocks, 256, 0, st>>>(smres, model, ssm, pscale, nscales, nmoment, n0, n1, psf_n0, psf_n1,
                                           gain, state);
      }
      count_launch(2 * batch);
      it += batch;
      if (cudaGetLastError() != cudaSuccess) {
        rc = fail(ARLGPU_ERR_CUDA, "msmfsclean launch failed");
        break;
      }
      if (cudaMemcpyAsync(&hs, state, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
          cudaStreamSynchronize(st) != cudaSuccess) {
        rc = fail(ARLGPU_ERR_CUDA, "msmfsclean state read failed");
        break;
      }
      if (hs.stop) break;
    }
  } while (false);
  *iterations = hs.iters;
  cudaFreeAsync(partial, st);
  cudaFreeAsync(state, st);
  return rc;
}

extern "C" int arlgpu_msclean(double *stack, const double *psf_ss, const double *pscale, const double *windowstack,
                              const double *coupling, int32_t nscales, int32_t nx, int32_t ny, int32_t psf_nx,
                              int32_t psf_ny, double gain, double absthresh, int32_t niter, double *comps,
                              int32_t *iterations, void *stream) {
  if (!stack || !psf_ss || !pscale || !coupling || !comps || !iterations)
    return fail(ARLGPU_ERR_INVALID, "null array argument");
  if (nscales < 1 || nx < 1 || ny < 1 || psf_nx < 2 || psf_ny < 2) return fail(ARLGPU_ERR_INVALID, "bad shapes");
  if (!(gain > 0.0 && gain < 2.0)) return fail(ARLGPU_ERR_INVALID, "gain must be in (0, 2)");
  if (niter < 1) return fail(ARLGPU_ERR_INVALID, "niter must be > 0");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long npix = (long long)nx * ny;
  const int fblocks = nblk((long long)nscales * npix, 152 * 4);
  const int sblocks = nblk((long long)psf_nx * psf_ny * (nscales + 1), 152 * 8);
  MsState *state = nullptr;
  BestS *partial = nullptr;
  ARL_CUDA(cudaMallocAsync(&state, sizeof(MsState), st));
  if (cudaMallocAsync(&partial, sizeof(BestS) * fblocks, st) != cudaSuccess) {
    cudaFreeAsync(state, st);
    return fail(ARLGPU_ERR_CUDA, "cudaMallocAsync failed");
  }
  const double stop_level = 0.9 * absthresh;
  constexpr int kCheck = 64;
  int rc = ARLGPU_OK;
  MsState hs{};
  if (cudaMemsetAsync(state, 0, sizeof(MsState), st) != cudaSuccess ||
      cudaMemsetAsync(comps, 0, sizeof(double) * npix, st) != cudaSuccess) {
    rc = fail(ARLGPU_ERR_CUDA, "msclean set-up failed");
  }
  for (int it = 0; rc == ARLGPU_OK && it < niter;) {
    const int batch = niter - it < kCheck ? niter - it : kCheck;
    for (int k = 0; k < batch; ++k) {
      k_ms_find<<<fblocks, kFindThreads, 0, st>>>(stack, windowstack, coupling, nscales, npix, stop_level, partial,
                                                  state);
      k_ms_sub<<<sblocks, 256, 0, st>>>(stack, comps, nscales, nx, ny, psf_ss, pscale, psf_nx, psf_ny, gain, state);
    }
    count_launch(2 * batch);
    it += batch;
    if (cudaGetLastError() != cudaSuccess) {
      rc = fail(ARLGPU_ERR_CUDA, "msclean launch failed");
      break;
    }
    if (cudaMemcpyAsync(&hs, state, sizeof hs, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = fail(ARLGPU_ERR_CUDA, "msclean state read failed");
      break;
    }
    if (hs.stop) break;
  }
  *iterations = hs.iters;
  cudaFreeAsync(partial, st);
  cudaFreeAsync(state, st);
  return rc;
}
