// compat.cu -- the reference library's arithmetic on the GB300 pipeline.
//
// Compiled with --use_fast_math, the flag the reference builds with
// (Makefile:26), so expf/powf/sqrtf/division in the filter coefficients map to
// the same hardware approximations and the per-tap weights agree with the
// reference's GPU build bit for bit; only the summation order differs.
//
// Pipeline per call (all on the caller's stream, no host synchronisation;
// dependent launches from the scatter pass on):
//   k_bin_count / k_scan_tiles / k_bin_scatter  samples -> tile-sorted records
//   k_grid_compat     one CTA per (tile, resample): taps accumulated in shared
//                     memory in fixed point, flushed once with f_hat[c].x += acc[c]
//   FFT               in-place inverse FFT of ng points with the reference's
//                     deconvolution fused into the last pass
//                     (single CTA for ng <= 2^14 (f32) / 2^13 (f64), four-step
//                     otherwise; non power-of-two ng falls back to cuFFT +
//                     k_compat_normalize)
#include <cufft.h>
#include <limits.h>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <algorithm>
#include "binning.cuh"
#include "fft.cuh"
#include "fftpass_core.cuh"
#include "rng.cuh"
#include "runtime.h"

namespace cuna {
namespace {

#define CUNA_PI 3.14159265358979323846

template <typename T> struct FpOf;
template <> struct FpOf<float> { typedef cuna2_filter_properties_f32 type; };
template <> struct FpOf<double> { typedef cuna2_filter_properties_f64 type; };

constexpr int kCompatLogTL = 12;  // 4096-cell tiles
constexpr int kCompatMaxRf = 64;  // shared E3 table size

// ---------------------------------------------------------------------------
// filter precompute: set_gpu_filter_properties, src/gaussian_filter.cu:204-228
// ---------------------------------------------------------------------------
// Filter origin u = (int)(ng x - R_f) of src/gaussian_filter.cu:213, in the
// sample's own precision (nvcc contracts the product and the difference into
// one fused multiply-add, here as in the reference's build).
__device__ __forceinline__ int compat_origin(float x, int ng, int rf) { return (int)(ng * x - rf); }
__device__ __forceinline__ int compat_origin(double x, int ng, int rf) { return (int)(ng * x - rf); }

// kFilterItems samples per thread, their loads in flight together (the kernel
// streams 12 bytes per float sample through short dependent chains: 1e6 samples
// 9.8 us with one per thread)
constexpr int kFilterItems = 4, kFilterThreads = 256;

__global__ void __launch_bounds__(kFilterThreads) k_compat_filter_f32(cuna2_filter_properties_f32 *f, const float *x,
                                                                      int ng, int n) {
  const int i0 = blockIdx.x * (kFilterThreads * kFilterItems) + threadIdx.x;
  float xv[kFilterItems];
#pragma unroll
  for (int k = 0; k < kFilterItems; ++k) {
    const int i = i0 + k * kFilterThreads;
    xv[k] = i < n ? x[i] : 0.f;
  }
  const float b = f->b;
  const int rf = f->filter_radius;
  float *E1 = f->E1, *E2 = f->E2;
#pragma unroll
  for (int k = 0; k < kFilterItems; ++k) {
    const int i = i0 + k * kFilterThreads;
    if (i < n) {
      int u = compat_origin(xv[k], ng, rf);
      float eps = ng * xv[k] - u;
      float eps2 = eps / b;
      E1[i] = expf(-eps * eps2) / sqrtf(CUNA_PI * b);
      E2[i] = expf(2 * eps2);
    } else if (i < n + rf) {
      int m = i - n;
      f->E3[m] = expf(-m * m / b);
    }
  }
}

// a / b from r, the reciprocal of b: one correction of the quotient by its exact
// remainder (Markstein 1990), the correctly rounded quotient for ordinary
// values; b is infinite (r = 0) on grids of n / 2 cells
__device__ __forceinline__ double div_by(double a, double b, double r) {
  const double q = a * r;
  return r == 0.0 ? q : fma(fma(-q, b, a), r, q);
}
// The FP64 pipe bounds this kernel: the square root and the two reciprocals that
// all samples share are one warp's work (1e5 samples: 15.8 us, 13.3 here).
__global__ void __launch_bounds__(kFilterThreads) k_compat_filter_f64(cuna2_filter_properties_f64 *f, const double *x,
                                                                      int ng, int n) {
  __shared__ double s[3];  // 1 / b, sqrt(pi b), 1 / sqrt(pi b)
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const double xi = i < n ? x[i] : 0.0, b = f->b;
  if (threadIdx.x < 32) {
    const double w = sqrt(CUNA_PI * b);
    s[0] = 1.0 / b;
    s[1] = w;
    s[2] = 1.0 / w;
  }
  __syncthreads();
  if (i < n) {
    int u = compat_origin(xi, ng, f->filter_radius);
    double eps = ng * xi - u;
    double eps2 = div_by(eps, b, s[0]);
    f->E1[i] = div_by(exp(-eps * eps2), s[1], s[2]);
    f->E2[i] = exp(2 * eps2);
  } else if (i < n + f->filter_radius) {
    int m = i - n;
    f->E3[m] = exp(-m * m / b);
  }
}

// ---------------------------------------------------------------------------
// deconvolution factor of normalize / normalize_bootstrap,
// src/gaussian_filter.cu:278-302
// ---------------------------------------------------------------------------
__device__ __forceinline__ float compat_fac(int k, int ng, float b, float normfac) {
  float K = ((float)k) / ((float)ng);
  return normfac * expf(K * K * b * 0.25);
}
__device__ __forceinline__ double compat_fac(int k, int ng, double b, double normfac) {
  double K = ((double)k) / ((double)ng);
  return normfac * exp(K * K * b * 0.25);
}

// fac(k0 + r stride), r = 0..R-1, of one radix-R butterfly's outputs (R = 16,
// or the only stage's radix).  Float evaluates each (one approximate exp).
// Double takes an exp at every fourth output only and forms the three between
// by exp(c (k + d)^2) = exp(c k^2) exp(2 c k d) exp(c d^2), c = b / (4 ng^2):
// five FP64 exps per butterfly instead of sixteen, at most four roundings each
// (the FP64 pipe bounds the double row pass).  hs: exp(c j d^2)
// for the butterfly's output stride d and j = 1, 4, 9, 8 (the last: the growth
// of exp(2 c k d) from one anchor to the next), per CTA.
__device__ __forceinline__ void compat_fac_steps(int stride, int ng, double b, double *hs) {
  if (threadIdx.x < 4) {
    const double D = (double)stride / (double)ng;
    const int j = threadIdx.x;
    hs[j] = exp(b * 0.25 * D * D * (double)(j == 0 ? 1 : (j == 1 ? 4 : (j == 2 ? 9 : 8))));
  }
}
__device__ __forceinline__ void compat_fac_steps(int, int, float, float *) {}
template <int R>
__device__ __forceinline__ void compat_facs(int k0, int stride, int ng, float b, float normfac, const float *,
                                            float *f) {
#pragma unroll
  for (int r = 0; r < R; ++r) f[r] = compat_fac(k0 + r * stride, ng, b, normfac);
}
template <int R>
__device__ __forceinline__ void compat_facs(int k0, int stride, int ng, double b, double normfac, const double *hs,
                                            double *f) {
  if constexpr (R < 16) {
#pragma unroll
    for (int r = 0; r < R; ++r) f[r] = compat_fac(k0 + r * stride, ng, b, normfac);
  } else {
    const double inv = 1.0 / (double)ng, D = (double)stride * inv, c = b * 0.25;
    const double h1 = hs[0], h2 = hs[1], h3 = hs[2], g4 = hs[3];
    double g = exp(2.0 * c * ((double)k0 * inv) * D);  // exp(2 c k d) at the anchor
#pragma unroll
    for (int a = 0; a < R; a += 4) {
      const double K = (double)(k0 + a * stride) * inv;
      const double e = normfac * exp(K * K * c);
      const double g2 = g * g;
      f[a] = e;
      f[a + 1] = e * (g * h1);
      f[a + 2] = e * (g2 * h2);
      f[a + 3] = e * (g2 * g * h3);
      g *= g4;
    }
  }
}

__device__ __forceinline__ float cpow(float a, int m) { return powf(a, m); }

// Reference cell j = (int)((x + 0.5) * (ng - 1)), in double arithmetic
// (src/gridding.cu:43,93).
__device__ __forceinline__ int compat_cell(double x, int ng) { return (int)((x + 0.5) * (ng - 1)); }
// The same for a float sample without the FP64 pipe (four operations of it per
// sample in each binning pass; 1e6 samples, ng = 2^22: with the dependent
// launches and the filter pass 118 -> 97 us per call): in units of 2^-40, x is an integer
// when 2^-16 <= |x| <= 1/2 (or 0), x + 1/2 and its product with ng - 1 < 2^23
// are exact in 64 bits, and the double product, rounded to 53 of its at most 63
// bits, truncates to another integer only if the fraction is within 2^-31 of 1.
// Everything else takes the double expression.
__device__ __forceinline__ int compat_cell(float x, int ng) {
  const unsigned u = __float_as_uint(x), ex = (u >> 23) & 0xff;
  if (ex >= 111 && fabsf(x) <= 0.5f && ng <= (1 << 23)) {
    const long long m = (long long)((u & 0x7fffffu) | 0x800000u) << (ex - 110);
    const unsigned long long p = (unsigned long long)((1ll << 39) + ((int)u < 0 ? -m : m)) * (unsigned)(ng - 1);
    if ((p & ((1ull << 40) - 1)) < (1ull << 40) - 1024) return (int)(p >> 40);
  }
  return compat_cell((double)x, ng);
}

// The cell and the tap bounds of src/gridding.cu:53-58.  Returns false when the
// tap range is empty.  |j| beyond 2^30 is treated as empty: the reference's
// int arithmetic overflows there and writes out of bounds.
template <typename T>
__device__ __forceinline__ bool compat_taps(T x, int ng, int rf, bool clamp, int &j, int &ms, int &me) {
  j = compat_cell(x, ng);
  if (clamp) {
    if (j >= ng) j = ng - 1;
    if (j < 0) j = 0;
  }
  if (j > (1 << 30) || j < -(1 << 30)) return false;
  ms = -rf + 1;
  me = rf;
  if (j + ms < 0) ms = -j;
  if (j + me > ng) me = ng - j;
  return ms < me;
}

// ---------------------------------------------------------------------------
// samplers for the binning kernels
// ---------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ void set_val(RecF &r, float v) { r.p = __float_as_int(v); }
template <typename T> __device__ __forceinline__ void set_val(RecD &r, double v) { r.v = v; }

template <typename T, bool BOOT> struct SampCompat {
  typedef typename RecOf<T>::type Rec;
  typedef typename FpOf<T>::type FP;
  struct Raw {
    T x, y, E1, E2;
  };
  const T *x;
  const T *y;
  const FP *fp;
  int64_t n;
  int ng;
  __device__ __forceinline__ Raw load(int64_t i, bool with_value) const {
    Raw r;
    r.x = x[i];
    if (!BOOT && with_value) {
      r.y = y ? y[i] : (T)1.0;
      r.E1 = fp->E1[i];
      r.E2 = fp->E2[i];
    }
    return r;
  }
  __device__ __forceinline__ void prep(int64_t i, const Raw &r, Prep<Rec> &p) const {
    int j, ms, me;
    p.nt = 0;
    if (!compat_taps(r.x, ng, fp->filter_radius, !BOOT, j, ms, me)) return;
    const int t0 = (j + ms) >> kCompatLogTL, t1 = (j + me - 1) >> kCompatLogTL;
    p.t[0] = t0;
    p.t[1] = t1;
    p.nt = t0 == t1 ? 1 : 2;
    p.rec.cell = j;
    if (BOOT) {
      p.rec.p = (int)i;
    } else {
      p.rec.a = r.E1;
      p.rec.b = r.E2;
      set_val<T>(p.rec, r.y);
    }
  }
};

__device__ __forceinline__ float rec_val(const RecF &r) { return __int_as_float(r.p); }
__device__ __forceinline__ double rec_val(const RecD &r) { return r.v; }

// ---------------------------------------------------------------------------
// tiled gridding: fast_gridding / fast_gridding_bootstrap,
// src/gridding.cu:36-65,86-117.  Every tap weight is the reference's own
// expression val * (E1 * pow(E2, m) * E3[|m|]) (filter(),
// src/gaussian_filter.cu:264-273); only the summation differs: instead of
// float atomics into f_hat (order-dependent) each CTA sums its tile in
// fixed point with native shared integer atomics and adds the tile to f_hat
// once.  The tile's scale comes from a bound on every cell's sum: |val| <=
// Ymax over the tile's records, a weight is at most 1 / sqrt(pi b), and at
// most 2 hmax records reach one cell (hmax: the most records in a bucket of
// >= 2 rf cells).  The quantum is 2^-30 (float) / 2^-62 (double) of that
// bound, and the sums no longer depend on the order of the atomics.
// ---------------------------------------------------------------------------
template <typename T, bool BOOT>
__device__ __forceinline__ void compat_coefs(const typename RecOf<T>::type &rc, const T *E1g, const T *E2g,
                                             const T *y, int n, unsigned seed, int slab, T &E1, T &E2, T &val) {
  if (BOOT) {
    const int i = slab * n + rc.p;
    int d = rc.p;
    val = (T)1.0;
    if (y) {
      d = (int)boot_draw(seed, (unsigned)i, (unsigned)n);
      val = y[d];
    }
    E1 = E1g[d];
    E2 = E2g[d];
  } else {
    E1 = rc.a;
    E2 = rc.b;
    val = rec_val(rc);
  }
}

// All taps of one record into the tile: cell m0 + m for m in [lo, hi), scaled
// by sc.  Float: powf of the fast-math build per tap, two approximate
// instructions, the reference's own bits.
template <typename A>
__device__ __forceinline__ void compat_record(A *acc, int m0, int lo, int hi, int rf, float E1, float E2, float val,
                                              float sc, const float *e3, const float *E3g) {
  for (int m = lo; m < hi; ++m) {
    const int mp = m < 0 ? -m : m;
    const float e3m = mp < kCompatMaxRf ? e3[mp] : E3g[mp];
    const float w = val * (E1 * cpow(E2, m) * e3m);
    FixAccWide<float>::add(acc + m0 + m, FixAccWide<float>::to_fix(w * sc));
  }
}
// Double: E2^m by a running product up and down from m = 0, kept as an
// unevaluated sum (p + pl) with FMA-exact products, so each power is the
// correctly rounded one to a few 2^-100 before it enters the tap; seven FP64
// operations per tap where pow() takes over a hundred.  The FP64 pipe (two
// FMA per clock and SM) bounds this kernel (1e5 samples on 2^19 cells: the
// whole transform 746 us with pow(), 588 of them here, and an exp per output;
// 193 us now).  The two chains are independent, which hides half of the FP64
// latency.
template <typename A>
__device__ __forceinline__ void compat_record(A *acc, int m0, int lo, int hi, int rf, double E1, double E2,
                                              double val, double sc, const double *e3, const double *E3g) {
  const double vs = val * sc;
  if (lo <= 0 && 0 < hi) FixAccWide<double>::add(acc + m0, FixAccWide<double>::to_fix(vs * (E1 * e3[0])));
  const double q = 1.0 / E2, ql = fma(-q, E2, 1.0) * q;  // 1/E2 = q + ql
  double p = 1.0, pl = 0.0, r = 1.0, rl = 0.0;
#pragma unroll 2
  for (int k = 1; k < rf; ++k) {
    const double t = E1 * (k < kCompatMaxRf ? e3[k] : E3g[k]);
    const double p1 = p * E2, r1 = r * q;
    pl = fma(pl, E2, fma(p, E2, -p1));
    rl = fma(rl, q, fma(r, ql, fma(r, q, -r1)));
    p = p1;
    r = r1;
    if (lo <= k && k < hi) FixAccWide<double>::add(acc + m0 + k, FixAccWide<double>::to_fix(vs * fma(t, pl, t * p)));
    if (lo <= -k && -k < hi)
      FixAccWide<double>::add(acc + m0 - k, FixAccWide<double>::to_fix(vs * fma(t, rl, t * r)));
  }
}

// Threads per tile: 256, or 1024 where the tiles and resamples of the call do
// not fill the SMs twice (a tile's records are then the serial chain: 128
// tiles of 780 records each for 1e5 samples on 2^19 cells).
constexpr int kCompatThreads = 256;
constexpr int kCompatThreadsFew = 1024;

template <typename T, bool BOOT, int NT>
__global__ void __launch_bounds__(NT) k_grid_compat(const typename RecOf<T>::type *rec_ptr, const int *off,
                                                    typename CxOf<T>::type *f_hat, int ng,
                                                    const typename FpOf<T>::type *fp, const T *__restrict__ y, int n,
                                                    unsigned seed) {
  typedef typename RecOf<T>::type Rec;
  const CgSrc<Rec> recs{rec_ptr};
  typedef FixAccWide<T> FA;
  typedef typename FA::type A;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  A *acc = reinterpret_cast<A *>(smem_raw);
  T *e3 = reinterpret_cast<T *>(acc + (1 << kCompatLogTL));
  int *hist = reinterpret_cast<int *>(e3 + kCompatMaxRf);
  __shared__ float red[NT / 32];
  __shared__ int redi[NT / 32];
  __shared__ T scale_s;
  pdl_trigger();
  const int tile = blockIdx.x, slab = blockIdx.y;
  const int base = tile << kCompatLogTL;
  const int tl = min(1 << kCompatLogTL, ng - base);
  const int rf = fp->filter_radius;
  const T *E3g = fp->E3, *E1g = fp->E1, *E2g = fp->E2;
  // buckets of >= 2 rf cells: the records reaching one cell lie in two buckets
  int logBS = 4;
  while ((1 << logBS) < 2 * rf) ++logBS;
  const int NB = ((tl + 2 * rf) >> logBS) + 1;
  for (int c = threadIdx.x; c < tl; c += NT) acc[c] = 0;
  for (int m = threadIdx.x; m < rf && m < kCompatMaxRf; m += NT) e3[m] = E3g[m];
  for (int q = threadIdx.x; q < NB; q += NT) hist[q] = 0;
  __syncthreads();
  pdl_wait();  // records and offsets come from the binning
  const int r0 = __ldcg(off + tile), r1 = __ldcg(off + tile + 1);
  // bound pass: records per bucket and the largest |value| (NaN if any is not finite)
  float ym = 0.f;
  // a thread's first records stay in registers for the taps
  constexpr int KEEP = sizeof(T) == 4 ? 2 : 1;
  const int cnt = r1 - r0;
  Rec keep[KEEP];
#pragma unroll
  for (int k = 0; k < KEEP; ++k)
    if (threadIdx.x + k * NT < cnt) keep[k] = recs[r0 + threadIdx.x + k * NT];
  Rec nx = keep[0];
#pragma unroll 1
  for (int i = threadIdx.x; i < cnt; i += NT) {
    const Rec rc = nx;
    nx = keep[KEEP - 1];
    if (i >= (KEEP - 1) * NT && i + NT < cnt) nx = recs[r0 + i + NT];
    atomicAdd(&hist[(rc.cell - base + rf) >> logBS], 1);
    T E1, E2, val;
    compat_coefs<T, BOOT>(rc, E1g, E2g, y, n, seed, slab, E1, E2, val);
    ym = isfinite(val) && !isnan(ym) ? fmaxf(ym, (float)fabs(val)) : __int_as_float(0x7fffffff);
  }
  __syncthreads();
  int hmax = 0;
  for (int q = threadIdx.x; q < NB; q += NT) hmax = max(hmax, hist[q]);
  for (int o = 16; o > 0; o >>= 1) {
    hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
    const float u = __shfl_xor_sync(0xffffffffu, ym, o);
    ym = (isnan(u) || isnan(ym)) ? __int_as_float(0x7fffffff) : fmaxf(ym, u);
  }
  if ((threadIdx.x & 31) == 0) {
    redi[threadIdx.x >> 5] = hmax;
    red[threadIdx.x >> 5] = ym;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int h = 0;
    float v = 0.f;
    bool bad = false;
    for (int w = 0; w < NT / 32; ++w) {
      h = max(h, redi[w]);
      bad |= isnan(red[w]);
      v = fmaxf(v, red[w]);
    }
    // a tap weight E1 E2^m E3[|m|] = exp(-(eps - m)^2 / b) / sqrt(pi b) is at
    // most 1 / sqrt(pi b); 1% margin for the approximate exp and pow
    const T wmax = (T)1.01 / sqrt((T)CUNA_PI * fp->b);
    const T B = (T)v * wmax * (T)(2 * h);
    T sc = B > (T)0 ? FA::range / B : (T)0;
    if (isinf(sc)) sc = (T)0;
    scale_s = bad ? (T)NAN : sc;
  }
  __syncthreads();
  const T sc = scale_s;
  if (sc > (T)0) {
    nx = keep[0];
#pragma unroll 1
    for (int i = threadIdx.x; i < cnt; i += NT) {
      const Rec rc = nx;
      nx = keep[KEEP - 1];
      if (i >= (KEEP - 1) * NT && i + NT < cnt) nx = recs[r0 + i + NT];
      const int j = rc.cell;
      int ms = -rf + 1, me = rf;
      if (j + ms < 0) ms = -j;
      if (j + me > ng) me = ng - j;
      T E1, E2, val;
      compat_coefs<T, BOOT>(rc, E1g, E2g, y, n, seed, slab, E1, E2, val);
      const int lo = max(ms, base - j), hi = min(me, base + tl - j);
      compat_record(acc, j - base, lo, hi, rf, E1, E2, val, sc, e3, E3g);
    }
  }
  __syncthreads();
  typename CxOf<T>::type *out = f_hat + (int64_t)slab * ng + base;
  if (isnan(sc)) {  // a non-finite value: the tile is NaN, as the float sums would spread it
    for (int c = threadIdx.x; c < tl; c += NT) out[c].x += (T)NAN;
    return;
  }
  const T inv = sc > (T)0 ? (T)1 / sc : (T)0;
  // f_hat's cells as whole 16-byte words, FB of them in flight per thread (one
  // at a time, and records read twice: 1e6 samples on 2^22 cells 27 us, 22 here)
  typedef typename std::conditional<sizeof(T) == 4, float4, double2>::type V;
  constexpr int CPV = sizeof(T) == 4 ? 2 : 1, FB = 4;
  int c0 = 0;
  if (((uintptr_t)out & 15) == 0) {
    V *ov = reinterpret_cast<V *>(out);
    const int nv = tl / CPV;
    for (int i = threadIdx.x; i < nv; i += FB * NT) {
      V v[FB];
#pragma unroll
      for (int k = 0; k < FB; ++k)
        if (i + k * NT < nv) v[k] = ov[i + k * NT];
#pragma unroll
      for (int k = 0; k < FB; ++k) {
        if (i + k * NT >= nv) continue;
        const int c = (i + k * NT) * CPV;
        const A a = acc[c];
        if (a != 0) v[k].x += (T)a * inv;
        if constexpr (CPV == 2) {
          const A b = acc[c + 1];
          if (b != 0) v[k].z += (T)b * inv;
        }
        ov[i + k * NT] = v[k];
      }
    }
    c0 = nv * CPV;
  }
  for (int c = c0 + threadIdx.x; c < tl; c += NT) {
    const A v = acc[c];
    if (v != 0) out[c].x += (T)v * inv;
  }
}

template <typename T> constexpr size_t compat_grid_smem() {
  // accumulators, E3 table, bucket counts (buckets of >= 16 cells)
  return sizeof(typename FixAcc<T>::type) * (1 << kCompatLogTL) + sizeof(T) * kCompatMaxRf +
         sizeof(int) * (((1 << kCompatLogTL) + 2 * kCompatMaxRf) / 16 + 1);
}

// ---------------------------------------------------------------------------
// FFT with the reference deconvolution fused in
// ---------------------------------------------------------------------------
template <typename T> struct FacDst {
  typename CxOf<T>::type *p;
  int ng, logL1, r0, norm;
  T b, nf;
  __device__ __forceinline__ void store(int seq, int k2, typename CxOf<T>::type v) const {
    const int k = r0 + seq + (k2 << logL1);
    p[k] = norm ? cscale(v, compat_fac(k, ng, b, nf)) : v;
  }
};
template <typename T> struct RowSrc {
  const typename CxOf<T>::type *p;
  int logL2;
  __device__ __forceinline__ typename CxOf<T>::type load(int seq, int i) const {
    return p[((int64_t)seq << logL2) + i];
  }
};

template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512) k_fft_single_compat(typename CxOf<T>::type *data, FftDev<T> f,
                                                            const typename FpOf<T>::type *fp, int norm) {
  typedef typename CxOf<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int L = 1 << f.logL;
  C *d = data + (int64_t)blockIdx.x * L;
  // in place: every read of d precedes the first barrier, every write follows it
  RowSrc<T> src{d, 0};
  FacDst<T> dst{d, L, 0, 0, norm, fp->b, fp->normfac};
  fft_fused<T, true, false, false>(s, 0, f.logL, 0, f.tw1, src, dst);
}

template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256) k_fft_rowpass_compat(const typename CxOf<T>::type *in,
                                                            typename CxOf<T>::type *out, FftDev<T> f,
                                                            const typename FpOf<T>::type *fp,
                                                            int64_t slab_stride, int norm) {
  typedef typename CxOf<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int logB = ilog2i((int64_t)blockDim.x * kFftE) - f.logL2;
  const int B = 1 << logB;
  const int pitch = fft_pitch(1 << f.logL2, B);
  const int r0 = blockIdx.x * B;
  RowSrc<T> src{in + blockIdx.y * slab_stride + ((int64_t)r0 << f.logL2), f.logL2};
  FacDst<T> dst{out + blockIdx.y * slab_stride, 1 << f.logL, f.logL1, r0, norm, fp->b, fp->normfac};
  // rows are read point-fastest (contiguous), outputs written row-fastest
  fft_fused<T, true, false, true>(s, pitch, f.logL2, logB, f.tw2, src, dst);
}

// Compile-time four-step passes of the compat transform: column pass from
// f_hat into scratch (twiddled), row pass from scratch back into f_hat in
// natural order with the reference normalisation fused in.
template <typename T, int LOGL, int LOGE>
__global__ void __launch_bounds__(1 << (LOGE - 4)) k_ct_colpass_oop(const typename CxOf<T>::type *in,
                                                                    typename CxOf<T>::type *out, FftDev<T> f,
                                                                    int64_t slab_stride) {
  ct_colpass_body<T, LOGL, LOGE>(in + blockIdx.y * slab_stride, out + blockIdx.y * slab_stride, f, blockIdx.x);
}

template <typename T, int LOG2> struct CtRowSrc {
  const typename CxOf<T>::type *p;  // first row of the block
  __device__ __forceinline__ typename CxOf<T>::type load(int seq, int j, int dr) const {
    return __ldcg(p + (seq << LOG2) + j + dr);  // through L2: the column pass may still be writing
  }
};

template <typename T, int LOG1> struct CtFacDst {
  typename CxOf<T>::type *p;  // slab
  int ng, r0, norm;
  T b, nf;
  const T *hs;  // compat_fac_steps
  template <int R, int LOGNS>
  __device__ __forceinline__ void store(int seq, int idxD, typename CxOf<T>::type *v) const {
    const int k0 = r0 + seq + (idxD << LOG1);
    constexpr int S = 1 << (LOGNS + LOG1);
    T fac[R];
    if (norm) compat_facs<R>(k0, S, ng, b, nf, hs, fac);
#pragma unroll
    for (int r = 0; r < R; ++r) p[k0 + r * S] = norm ? cscale(v[r], fac[r]) : v[r];
  }
};

template <typename T, int LOGL, int LOGE>
__global__ void __launch_bounds__(1 << (LOGE - 4)) k_ct_rowpass_compat(const typename CxOf<T>::type *in,
                                                                       typename CxOf<T>::type *out, FftDev<T> f,
                                                                       const typename FpOf<T>::type *fp,
                                                                       int64_t slab_stride, int norm) {
  typedef typename CxOf<T>::type C;
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2;
  constexpr int LOGB = LOGE - LOG2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int r0 = blockIdx.x << LOGB;
  CtRowSrc<T, LOG2> src{in + blockIdx.y * slab_stride + ((int64_t)r0 << LOG2)};
  __shared__ T hs[4];  // read by the storing stage, after at least one barrier
  static_assert(LOG2 > 4, "the row transform has more than one stage");
  pdl_trigger();
  compat_fac_steps(1 << (last_logns<LOG2>() + LOG1), 1 << LOGL, fp->b, hs);
  pdl_wait();  // the rows come from the column pass
  CtFacDst<T, LOG1> dst{out + blockIdx.y * slab_stride, 1 << LOGL, r0, norm, fp->b, fp->normfac, hs};
  // rows are read point-fastest (contiguous), outputs written row-fastest
  ct_fft<T, LOG2, LOGB, true, false, true>(s, f.tw2, src, dst);
}

// Dependent launch for the float kernels only.  The double ones are bound by
// the FP64 pipe: CTAs that become resident early crowd the SMs that happen to
// have room and then share their pipes (1e5 samples, ng = 2^19: 193 -> 276 us).
template <typename T, typename... KArgs, typename... Args>
cudaError_t launch_compat(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  if (sizeof(T) == 4) return launch_pdl(k, grid, block, smem, st, args...);
  k<<<grid, block, smem, st>>>(static_cast<KArgs>(args)...);
  return cudaGetLastError();
}

template <typename T, int LOGL, int LOGE>
int compat_ct_sized(typename CxOf<T>::type *f_hat, typename CxOf<T>::type *scratch, const FftDev<T> &f,
                    const typename FpOf<T>::type *dfp, int nbs, bool norm, cudaStream_t st) {
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2;
  constexpr int BA = 1 << (LOGE - LOG1), BB = 1 << (LOGE - LOG2), TH = 1 << (LOGE - 4);
  constexpr size_t smA = ct_colpass_smem<T, LOGL, LOGE>();
  constexpr size_t smB = sizeof(typename CxOf<T>::type) * (size_t)fft_pitch(1 << LOG2, BB) * BB;
  static SetupFlag attr;
  if (!setup_done(&attr)) {
    if (cudaFuncSetAttribute(k_ct_colpass_oop<T, LOGL, LOGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smA) ||
        cudaFuncSetAttribute(k_ct_rowpass_compat<T, LOGL, LOGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smB))
      return -1;
    mark_setup_done(&attr);
  }
  const int64_t L = (int64_t)1 << LOGL;
  typedef typename CxOf<T>::type C;
  if (launch_compat<T>(k_ct_colpass_oop<T, LOGL, LOGE>, dim3((1 << LOG2) / BA, nbs), dim3(TH), smA, st, (const C *)f_hat,
                 scratch, f, L) != cudaSuccess)
    return -1;
  if (launch_compat<T>(k_ct_rowpass_compat<T, LOGL, LOGE>, dim3((1 << LOG1) / BB, nbs), dim3(TH), smB, st, (const C *)scratch,
                 f_hat, f, dfp, L, norm ? 1 : 0) != cudaSuccess)
    return -1;
  return 1;
}
template <typename T, int LOGL>
int compat_ct_at(typename CxOf<T>::type *f_hat, typename CxOf<T>::type *scratch, const FftDev<T> &f,
                 const typename FpOf<T>::type *dfp, int nbs, bool norm, cudaStream_t st) {
  if constexpr (sizeof(T) == 4)
    if (pass_few<T>(LOGL, nbs, 4))
      return compat_ct_sized<T, LOGL, PassFew<T, LOGL>::LOGE>(f_hat, scratch, f, dfp, nbs, norm, st);
  return compat_ct_sized<T, LOGL, PassCfg<T>::LOGE>(f_hat, scratch, f, dfp, nbs, norm, st);
}

// 1: launched, 0: no compiled instance, -1: launch error
template <typename T>
int compat_ct(int logL, typename CxOf<T>::type *f_hat, typename CxOf<T>::type *scratch, const FftDev<T> &f,
              const typename FpOf<T>::type *dfp, int nbs, bool norm, cudaStream_t st) {
#define CUNA_CCT(LG) \
  case LG: return compat_ct_at<T, LG>(f_hat, scratch, f, dfp, nbs, norm, st);
  if constexpr (sizeof(T) == 4) {
    switch (logL) { CUNA_CCT(15) CUNA_CCT(16) CUNA_CCT(17) CUNA_CCT(18) CUNA_CCT(19) CUNA_CCT(20) CUNA_CCT(21) CUNA_CCT(22) CUNA_CCT(23) CUNA_CCT(24) CUNA_CCT(25) }
  } else {
    switch (logL) { CUNA_CCT(14) CUNA_CCT(15) CUNA_CCT(16) CUNA_CCT(17) CUNA_CCT(18) CUNA_CCT(19) CUNA_CCT(20) CUNA_CCT(21) CUNA_CCT(22) CUNA_CCT(23) }
  }
#undef CUNA_CCT
  return 0;
}

template <typename T>
__global__ void k_compat_normalize(typename CxOf<T>::type *f_hat, int ng, int64_t total,
                                   const typename FpOf<T>::type *fp) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) f_hat[i] = cscale(f_hat[i], compat_fac((int)(i % ng), ng, fp->b, fp->normfac));
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
template <typename T> FftDev<T> to_dev(const FftGeom &g) {
  typedef typename CxOf<T>::type C;
  FftDev<T> f;
  f.logL = g.logL;
  f.logL1 = g.logL1;
  f.logL2 = g.logL2;
  f.tw1 = (const C *)g.tw1;
  f.tw2 = (const C *)g.tw2;
  f.twlo = (const C *)g.twlo;
  f.twhi = (const C *)g.twhi;
  return f;
}

size_t align_up(size_t v) { return (v + 255) & ~(size_t)255; }

// cuFFT comparator plans for non power-of-two grids, cached per
// (device, stream, ng, batch, precision).
std::mutex g_cufft_mu;
std::map<std::tuple<int, cudaStream_t, int, int, int>, cufftHandle> *g_cufft =
    new std::map<std::tuple<int, cudaStream_t, int, int, int>, cufftHandle>();

template <typename T>
int cufft_inverse(typename CxOf<T>::type *data, int ng, int nbs, cudaStream_t st) {
  int dev = 0;
  CUNA_CK(cudaGetDevice(&dev));
  cufftHandle h;
  {
    std::lock_guard<std::mutex> lk(g_cufft_mu);
    auto key = std::make_tuple(dev, st, ng, nbs, (int)sizeof(T));
    auto it = g_cufft->find(key);
    if (it == g_cufft->end()) {
      int dims[1] = {ng};
      cufftResult r = cufftPlanMany(&h, 1, dims, nullptr, 1, ng, nullptr, 1, ng,
                                    sizeof(T) == 4 ? CUFFT_C2C : CUFFT_Z2Z, nbs);
      if (r != CUFFT_SUCCESS) return fail(CUNA2_ERROR_CUFFT, "cufftPlanMany failed (%d)", (int)r);
      if ((r = cufftSetStream(h, st)) != CUFFT_SUCCESS)
        return fail(CUNA2_ERROR_CUFFT, "cufftSetStream failed (%d)", (int)r);
      (*g_cufft)[key] = h;
    } else {
      h = it->second;
    }
  }
  cufftResult r;
  if (sizeof(T) == 4)
    r = cufftExecC2C(h, (cufftComplex *)data, (cufftComplex *)data, CUFFT_INVERSE);
  else
    r = cufftExecZ2Z(h, (cufftDoubleComplex *)data, (cufftDoubleComplex *)data, CUFFT_INVERSE);
  if (r != CUFFT_SUCCESS) return fail(CUNA2_ERROR_CUFFT, "cufftExec failed (%d)", (int)r);
  return CUNA2_SUCCESS;
}

template <typename T>
int compat_normalize(typename CxOf<T>::type *f_hat, int ng, int nbs, const typename FpOf<T>::type *dfp,
                     cudaStream_t st) {
  const int64_t total = (int64_t)ng * nbs;
  if (total == 0) return CUNA2_SUCCESS;
  k_compat_normalize<T><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(f_hat, ng, total, dfp);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

// In-place inverse FFT of nbs slabs of ng points; `norm` fuses the reference
// deconvolution into the last pass.
template <typename T>
int compat_fft(typename CxOf<T>::type *f_hat, int ng, int nbs, const typename FpOf<T>::type *dfp,
               typename CxOf<T>::type *scratch, bool norm, cudaStream_t st) {
  typedef typename CxOf<T>::type C;
  const bool pow2 = (ng & (ng - 1)) == 0;
  const int logL = ilog2i(ng);
  // four-step limit: the column pass holds at least one column of L1 points
  const int max_log = sizeof(T) == 4 ? 26 : 24;
  if (!pow2 || logL > max_log) {
    CUNA_TRY(cufft_inverse<T>(f_hat, ng, nbs, st));
    return norm ? compat_normalize<T>(f_hat, ng, nbs, dfp, st) : CUNA2_SUCCESS;
  }
  FftGeom g;
  CUNA_TRY(fft_geometry(sizeof(T) == 8, logL, &g));
  FftDev<T> f = to_dev<T>(g);
  if (g.single) {
    const int L = 1 << logL;
    const int threads = max(32, L / kFftE);
    const size_t smem = sizeof(C) * (size_t)fft_pitch(L, 1);
    static SetupFlag attr;
    if (!setup_done(&attr)) {
      CUNA_CK(cudaFuncSetAttribute(k_fft_single_compat<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   200 * 1024));
      mark_setup_done(&attr);
    }
    k_fft_single_compat<T><<<nbs, threads, smem, st>>>(f_hat, f, dfp, norm ? 1 : 0);
    CUNA_CK(cudaGetLastError());
    return CUNA2_SUCCESS;
  }
  {
    const int h = compat_ct<T>(logL, f_hat, scratch, f, dfp, nbs, norm, st);
    if (h < 0) return fail_cuda(cudaGetLastError(), "FFT pass launch");
    if (h == 1) return CUNA2_SUCCESS;
  }
  const int elems = sizeof(T) == 4 ? kPassElemsF32 : kPassElemsF64;
  const int threads = elems / kFftE;
  const int L1 = 1 << g.logL1, L2 = 1 << g.logL2;
  const int BA = elems / L1, BB = elems / L2;
  const size_t smemA = sizeof(C) * (size_t)BA * fft_pitch(L1, BA);
  const size_t smemB = sizeof(C) * (size_t)BB * fft_pitch(L2, BB);
  static SetupFlag attr2;
  if (!setup_done(&attr2)) {
    CUNA_CK(cudaFuncSetAttribute(k_fft_colpass<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    CUNA_CK(cudaFuncSetAttribute(k_fft_rowpass_compat<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 200 * 1024));
    mark_setup_done(&attr2);
  }
  const int64_t L = (int64_t)ng;
  k_fft_colpass<T><<<dim3(L2 / BA, nbs), threads, smemA, st>>>(f_hat, scratch, f, L);
  CUNA_CK(cudaGetLastError());
  k_fft_rowpass_compat<T><<<dim3(L1 / BB, nbs), threads, smemB, st>>>(scratch, f_hat, f, dfp, L,
                                                                      norm ? 1 : 0);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

struct CompatWs {
  int *counts, *offsets, *cursor;
  int *resv;  // reservation table of the two-launch binning (up to kScanFuseTiles tiles)
  void *recs;
  void *scratch;
};

// blocks of the reserved binning for n samples on ntiles tiles (0: not used)
inline int compat_resv_blocks(int n, int ntiles) {
  if (n <= 0 || ntiles > kScanFuseTiles) return 0;
  const int64_t span = resv_span(n, ntiles, device_sm_count());
  return (int)((n + span - 1) / span);
}

template <typename T>
int compat_workspace(int n, int ng, int nbs, bool need_fft, cudaStream_t st, CompatWs *cw) {
  typedef typename CxOf<T>::type C;
  typedef typename RecOf<T>::type Rec;
  const int ntiles = (ng + (1 << kCompatLogTL) - 1) >> kCompatLogTL;
  const bool pow2 = (ng & (ng - 1)) == 0;
  const bool fourstep = need_fft && pow2 && ilog2i(ng) > (sizeof(T) == 4 ? kSingleLogF32 : kSingleLogF64) &&
                        ilog2i(ng) <= (sizeof(T) == 4 ? 26 : 24);
  const size_t o_off = align_up(sizeof(int) * ntiles), o_cur = o_off + align_up(sizeof(int) * (ntiles + 1));
  const size_t o_rsv = o_cur + align_up(sizeof(int) * ntiles);
  const size_t o_rec = o_rsv + align_up(sizeof(int) * (size_t)compat_resv_blocks(n, ntiles) * ntiles);
  const size_t o_fft = o_rec + align_up(sizeof(Rec) * 2 * (size_t)(n > 0 ? n : 1));
  const size_t bytes = o_fft + (fourstep ? sizeof(C) * (size_t)ng * nbs : 0);
  void *ws = nullptr;
  CUNA_TRY(stream_workspace(st, bytes, &ws));
  char *w = (char *)ws;
  cw->counts = (int *)w;
  cw->offsets = (int *)(w + o_off);
  cw->cursor = (int *)(w + o_cur);
  cw->resv = (int *)(w + o_rsv);
  cw->recs = w + o_rec;
  cw->scratch = fourstep ? (void *)(w + o_fft) : nullptr;
  return CUNA2_SUCCESS;
}

int check_args(int n, int ng, int nbs, const void *x, const void *f_hat, const void *dfp) {
  if (n < 0 || ng < 1 || nbs < 1 || !f_hat || !dfp || (n > 0 && !x))
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid argument (n=%d ng=%d nbs=%d)", n, ng, nbs);
  if ((int64_t)n * nbs > INT_MAX || (int64_t)ng * nbs > ((int64_t)1 << 40))
    return fail(CUNA2_ERROR_UNSUPPORTED, "n*nbs exceeds the reference's int index range");
  if (nbs > 65535) return fail(CUNA2_ERROR_UNSUPPORTED, "more than 65535 resamples per call");
  return CUNA2_SUCCESS;
}

// Binning: the bucket sort of the samples into 4096-cell tiles (records
// in cw.recs, tile t's records at [cw.offsets[t], cw.offsets[t+1])).
template <typename T>
int compat_bin(const T *x, const T *y, int n, int ng, const typename FpOf<T>::type *dfp, bool boot,
               const CompatWs &cw, cudaStream_t st) {
  typedef typename RecOf<T>::type Rec;
  const int ntiles = (ng + (1 << kCompatLogTL) - 1) >> kCompatLogTL;
  Rec *recs = (Rec *)cw.recs;
  SampCompat<T, false> sp{x, y, dfp, n, ng};
  SampCompat<T, true> sb{x, y, dfp, n, ng};
  const int sms = device_sm_count();
  const size_t smc = ntiles <= kBinSmemTiles ? sizeof(int) * ntiles : 0;
  const int gcount = (int)std::min<int64_t>((n + 4095) / 4096, 4 * sms);
  const int gscat = (int)((n + 512 * kScatterItems - 1) / (512 * kScatterItems));
  const int nrb = compat_resv_blocks(n, ntiles);
  if (nrb <= 0) CUNA_CK(cudaMemsetAsync(cw.counts, 0, sizeof(int) * ntiles, st));
  if (nrb > 0) {
    // count + reserve, then scan + scatter without global atomics (binning.cuh)
    const int64_t span = resv_span(n, ntiles, device_sm_count());
    const size_t sms3 = sizeof(int) * (3 * (size_t)ntiles + 1);
    static SetupFlag attr;
    if (!setup_done(&attr)) {
      const int mx = (int)(sizeof(int) * (3 * kScanFuseTiles + 1));
      CUNA_CK(cudaFuncSetAttribute(k_bin_scatter_resv<SampCompat<T, false>>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
      CUNA_CK(cudaFuncSetAttribute(k_bin_scatter_resv<SampCompat<T, true>>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
      mark_setup_done(&attr);
    }
    if (sizeof(T) == 4) k_zero_counts<<<(ntiles + 255) / 256, 256, 0, st>>>(cw.counts, ntiles);
    else CUNA_CK(cudaMemsetAsync(cw.counts, 0, sizeof(int) * ntiles, st));  // plain launches follow
    CUNA_CK(cudaGetLastError());
    if (boot) {
      CUNA_CK(launch_compat<T>(k_bin_count_resv<SampCompat<T, true>>, dim3(nrb), dim3(512), sizeof(int) * ntiles, st, sb,
                               cw.counts, cw.resv, ntiles, span));
      CUNA_CK(launch_pdl(k_bin_scatter_resv<SampCompat<T, true>>, dim3(nrb), dim3(512), sms3, st, sb,
                         (const int *)cw.counts, (const int *)cw.resv, cw.offsets, recs, ntiles, span));
    } else {
      CUNA_CK(launch_compat<T>(k_bin_count_resv<SampCompat<T, false>>, dim3(nrb), dim3(512), sizeof(int) * ntiles, st, sp,
                               cw.counts, cw.resv, ntiles, span));
      CUNA_CK(launch_pdl(k_bin_scatter_resv<SampCompat<T, false>>, dim3(nrb), dim3(512), sms3, st, sp,
                         (const int *)cw.counts, (const int *)cw.resv, cw.offsets, recs, ntiles, span));
    }
    CUNA_CK(cudaGetLastError());
  } else {
    if (boot) k_bin_count<<<gcount, 512, smc, st>>>(sb, cw.counts, ntiles);
    else k_bin_count<<<gcount, 512, smc, st>>>(sp, cw.counts, ntiles);
    CUNA_CK(cudaGetLastError());
    k_scan_tiles<<<1, 1024, 0, st>>>(cw.counts, cw.offsets, cw.cursor, ntiles);
    CUNA_CK(cudaGetLastError());
    if (boot) k_bin_scatter<<<gscat, 512, 2 * smc, st>>>(sb, cw.offsets, cw.cursor, recs, ntiles);
    else k_bin_scatter<<<gscat, 512, 2 * smc, st>>>(sp, cw.offsets, cw.cursor, recs, ntiles);
    CUNA_CK(cudaGetLastError());
  }
  return CUNA2_SUCCESS;
}

// Gridding stage: binning + tiled gridding, accumulating into f_hat.
template <typename T>
int compat_grid(const T *x, const T *y, typename CxOf<T>::type *f_hat, int n, int ng, int nbs,
                const typename FpOf<T>::type *dfp, unsigned seed, bool boot, const CompatWs &cw,
                cudaStream_t st) {
  typedef typename RecOf<T>::type Rec;
  if (n == 0) return CUNA2_SUCCESS;
  const int ntiles = (ng + (1 << kCompatLogTL) - 1) >> kCompatLogTL;
  CUNA_TRY(compat_bin<T>(x, y, n, ng, dfp, boot, cw, st));
  Rec *recs = (Rec *)cw.recs;
  const size_t smg = compat_grid_smem<T>();
  const dim3 gg(ntiles, boot ? nbs : 1);
  constexpr int NF = kCompatThreadsFew, NM = kCompatThreads;
  const bool few = (int64_t)gg.x * gg.y < 2 * (int64_t)device_sm_count();
  auto k = boot ? (few ? k_grid_compat<T, true, NF> : k_grid_compat<T, true, NM>)
                : (few ? k_grid_compat<T, false, NF> : k_grid_compat<T, false, NM>);
  CUNA_CK(launch_compat<T>(k, gg, dim3(few ? NF : NM), smg, st, (const Rec *)recs, (const int *)cw.offsets, f_hat, ng, dfp, y,
                     n, seed));
  return CUNA2_SUCCESS;
}

template <typename T>
int compat_run(const T *x, const T *y, typename CxOf<T>::type *f_hat, int n, int ng, int nbs,
               const typename FpOf<T>::type *dfp, unsigned seed, bool boot, cudaStream_t st) {
  typedef typename CxOf<T>::type C;
  clear_error();
  CUNA_TRY(check_args(n, ng, boot ? nbs : 1, x, f_hat, dfp));
  if (!boot) nbs = 1;
  CompatWs cw;
  CUNA_TRY(compat_workspace<T>(n, ng, nbs, true, st, &cw));
  CUNA_TRY(compat_grid<T>(x, y, f_hat, n, ng, nbs, dfp, seed, boot, cw, st));
  return compat_fft<T>(f_hat, ng, nbs, dfp, (C *)cw.scratch, true, st);
}

template <typename T, typename FP>
int compat_filter(const T *x, int n, int ng, FP *h, FP *d, cudaStream_t st) {
  clear_error();
  if (n < 1 || ng < 1 || !h || !d || !x)
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid argument (n=%d ng=%d)", n, ng);
  const int rf = sizeof(T) == 4 ? 6 : 12;  // FILTER_RADIUS, src/gaussian_filter.cu:29-33
  // host part of generate_pinned_filter_properties, src/gaussian_filter.cu:54-57
  T R = ((T)ng) / n;
  h->b = 2 * R / (2 * R - 1) * (rf / CUNA_PI);
  h->filter_radius = rf;
  h->normfac = sqrt(2 * CUNA_PI);
  CUNA_CK(cudaMemcpyAsync(d, h, sizeof(FP), cudaMemcpyHostToDevice, st));
  const int per = kFilterThreads * (sizeof(T) == 4 ? kFilterItems : 1), nb = (int)(((int64_t)n + rf + per - 1) / per);
  if (sizeof(T) == 4)
    k_compat_filter_f32<<<nb, kFilterThreads, 0, st>>>((cuna2_filter_properties_f32 *)d, (const float *)x, ng, n);
  else
    k_compat_filter_f64<<<nb, kFilterThreads, 0, st>>>((cuna2_filter_properties_f64 *)d, (const double *)x, ng, n);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

}  // namespace
}  // namespace cuna

using namespace cuna;

extern "C" int cuna2_compat_filter_radius(int is_double) { return is_double ? 12 : 6; }

extern "C" int cuna2_compat_filter_f32(const float *x, int n, int ng, cuna2_filter_properties_f32 *h,
                                       cuna2_filter_properties_f32 *d, cudaStream_t st) {
  return compat_filter<float>(x, n, ng, h, d, st);
}
extern "C" int cuna2_compat_filter_f64(const double *x, int n, int ng, cuna2_filter_properties_f64 *h,
                                       cuna2_filter_properties_f64 *d, cudaStream_t st) {
  return compat_filter<double>(x, n, ng, h, d, st);
}
extern "C" int cuna2_compat_adjoint_f32(const float *x, const float *y, float2 *f_hat, int n, int ng,
                                        const cuna2_filter_properties_f32 *d, cudaStream_t st) {
  return compat_run<float>(x, y, f_hat, n, ng, 1, d, 0u, false, st);
}
extern "C" int cuna2_compat_adjoint_f64(const double *x, const double *y, double2 *f_hat, int n, int ng,
                                        const cuna2_filter_properties_f64 *d, cudaStream_t st) {
  return compat_run<double>(x, y, f_hat, n, ng, 1, d, 0u, false, st);
}
extern "C" int cuna2_compat_bootstrap_f32(const float *x, const float *y, float2 *f_hat, int n, int ng,
                                          int nbs, const cuna2_filter_properties_f32 *d, unsigned seed,
                                          cudaStream_t st) {
  return compat_run<float>(x, y, f_hat, n, ng, nbs, d, seed, true, st);
}
extern "C" int cuna2_compat_bootstrap_f64(const double *x, const double *y, double2 *f_hat, int n, int ng,
                                          int nbs, const cuna2_filter_properties_f64 *d, unsigned seed,
                                          cudaStream_t st) {
  return compat_run<double>(x, y, f_hat, n, ng, nbs, d, seed, true, st);
}

extern "C" int cuna2_compat_grid_f32(const float *x, const float *y, float2 *f_hat, int n, int ng,
                                     const cuna2_filter_properties_f32 *d, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(n, ng, 1, x, f_hat, d));
  CompatWs cw;
  CUNA_TRY(compat_workspace<float>(n, ng, 1, false, st, &cw));
  return compat_grid<float>(x, y, f_hat, n, ng, 1, d, 0u, false, cw, st);
}
extern "C" int cuna2_compat_grid_f64(const double *x, const double *y, double2 *f_hat, int n, int ng,
                                     const cuna2_filter_properties_f64 *d, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(n, ng, 1, x, f_hat, d));
  CompatWs cw;
  CUNA_TRY(compat_workspace<double>(n, ng, 1, false, st, &cw));
  return compat_grid<double>(x, y, f_hat, n, ng, 1, d, 0u, false, cw, st);
}
extern "C" int cuna2_compat_fft_f32(float2 *f_hat, int ng, int nbatch, const cuna2_filter_properties_f32 *d,
                                    int normalize, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(0, ng, nbatch, nullptr, f_hat, d));
  CompatWs cw;
  CUNA_TRY(compat_workspace<float>(0, ng, nbatch, true, st, &cw));
  return compat_fft<float>(f_hat, ng, nbatch, d, (float2 *)cw.scratch, normalize != 0, st);
}
extern "C" int cuna2_compat_fft_f64(double2 *f_hat, int ng, int nbatch, const cuna2_filter_properties_f64 *d,
                                    int normalize, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(0, ng, nbatch, nullptr, f_hat, d));
  CompatWs cw;
  CUNA_TRY(compat_workspace<double>(0, ng, nbatch, true, st, &cw));
  return compat_fft<double>(f_hat, ng, nbatch, d, (double2 *)cw.scratch, normalize != 0, st);
}
extern "C" int cuna2_compat_normalize_f32(float2 *f_hat, int ng, int nbatch,
                                          const cuna2_filter_properties_f32 *d, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(0, ng, nbatch, nullptr, f_hat, d));
  return compat_normalize<float>(f_hat, ng, nbatch, d, st);
}
extern "C" int cuna2_compat_normalize_f64(double2 *f_hat, int ng, int nbatch,
                                          const cuna2_filter_properties_f64 *d, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(0, ng, nbatch, nullptr, f_hat, d));
  return compat_normalize<double>(f_hat, ng, nbatch, d, st);
}

// ---------------------------------------------------------------------------
// Integer steps read back: per sample the cell j, the filter origin u and the
// tap range, the bootstrap draws, and the records of the binning, computed by
// the same device functions the transforms run (compat_taps, compat_origin,
// boot_draw, compat_bin).  Tests compare them with the oracle bit for bit;
// the transforms never call these.
// ---------------------------------------------------------------------------
namespace cuna {
namespace {

template <typename T>
__global__ void k_inspect_compat_taps(const T *x, int n, int ng, int rf, int clamp, int *cell, int *origin,
                                      int *tlo, int *thi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T xi = x[i];
  int j = 0, ms = 0, me = 0;
  const bool any = compat_taps(xi, ng, rf, clamp != 0, j, ms, me);
  if (cell) cell[i] = j;
  if (origin) origin[i] = compat_origin(xi, ng, rf);
  if (tlo) tlo[i] = any ? ms : 0;
  if (thi) thi[i] = any ? me : 0;
}

__global__ void k_inspect_draws(unsigned n, int64_t total, unsigned seed, int *d) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    d[i] = (int)boot_draw(seed, (unsigned)i, n);
}

template <typename T>
int inspect_compat_taps(const T *x, int n, int ng, int clamp, int *cell, int *origin, int *tlo, int *thi,
                        cudaStream_t st) {
  clear_error();
  if (n < 0 || ng < 1 || (n > 0 && !x))
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid argument (n=%d ng=%d)", n, ng);
  if (n == 0) return CUNA2_SUCCESS;
  const int rf = sizeof(T) == 4 ? 6 : 12;
  k_inspect_compat_taps<T><<<(n + 255) / 256, 256, 0, st>>>(x, n, ng, rf, clamp, cell, origin, tlo, thi);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

template <typename T>
int inspect_compat_bins(const T *x, const T *y, int n, int ng, const typename FpOf<T>::type *dfp, int boot,
                        int *offsets, void *records, int max_records, int *nrecords, cudaStream_t st) {
  typedef typename RecOf<T>::type Rec;
  clear_error();
  CUNA_TRY(check_args(n, ng, 1, x, offsets, dfp));
  if (max_records < 0 || (max_records > 0 && !records))
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid record buffer (max_records=%d)", max_records);
  const int ntiles = (ng + (1 << kCompatLogTL) - 1) >> kCompatLogTL;
  int total = 0;
  if (n == 0) {
    CUNA_CK(cudaMemsetAsync(offsets, 0, sizeof(int) * (ntiles + 1), st));
  } else {
    CompatWs cw;
    CUNA_TRY(compat_workspace<T>(n, ng, 1, false, st, &cw));
    CUNA_TRY(compat_bin<T>(x, y, n, ng, dfp, boot != 0, cw, st));
    CUNA_CK(cudaMemcpyAsync(offsets, cw.offsets, sizeof(int) * (ntiles + 1), cudaMemcpyDeviceToDevice, st));
    CUNA_CK(cudaMemcpyAsync(&total, cw.offsets + ntiles, sizeof(int), cudaMemcpyDeviceToHost, st));
    CUNA_CK(cudaStreamSynchronize(st));
    if (total > max_records) {
      if (nrecords) *nrecords = total;
      return fail(CUNA2_ERROR_INVALID_VALUE, "%d records do not fit in max_records = %d", total, max_records);
    }
    if (total > 0)
      CUNA_CK(cudaMemcpyAsync(records, cw.recs, sizeof(Rec) * (size_t)total, cudaMemcpyDeviceToDevice, st));
  }
  if (nrecords) *nrecords = total;
  return CUNA2_SUCCESS;
}

}  // namespace
}  // namespace cuna

extern "C" int cuna2_inspect_compat_taps_f32(const float *x, int n, int ng, int clamp, int *cell, int *origin,
                                             int *tap_lo, int *tap_hi, cudaStream_t st) {
  return inspect_compat_taps<float>(x, n, ng, clamp, cell, origin, tap_lo, tap_hi, st);
}
extern "C" int cuna2_inspect_compat_taps_f64(const double *x, int n, int ng, int clamp, int *cell, int *origin,
                                             int *tap_lo, int *tap_hi, cudaStream_t st) {
  return inspect_compat_taps<double>(x, n, ng, clamp, cell, origin, tap_lo, tap_hi, st);
}
extern "C" int cuna2_inspect_bootstrap_draws(int n, int nbs, unsigned int seed, int *draw, cudaStream_t st) {
  clear_error();
  if (n < 1 || nbs < 1 || !draw || (int64_t)n * nbs > INT_MAX)
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid argument (n=%d nbs=%d)", n, nbs);
  const int64_t total = (int64_t)n * nbs;
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, 8192);
  k_inspect_draws<<<blocks, 256, 0, st>>>((unsigned)n, total, seed, draw);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}
extern "C" int cuna2_inspect_compat_bins_f32(const float *x, const float *y, int n, int ng,
                                             const cuna2_filter_properties_f32 *d, int boot, int *offsets,
                                             void *records, int max_records, int *nrecords, cudaStream_t st) {
  return inspect_compat_bins<float>(x, y, n, ng, d, boot, offsets, records, max_records, nrecords, st);
}
extern "C" int cuna2_inspect_compat_bins_f64(const double *x, const double *y, int n, int ng,
                                             const cuna2_filter_properties_f64 *d, int boot, int *offsets,
                                             void *records, int max_records, int *nrecords, cudaStream_t st) {
  return inspect_compat_bins<double>(x, y, n, ng, d, boot, offsets, records, max_records, nrecords, st);
}

// ---------------------------------------------------------------------------
// cuna2_compat_adjoint_noalloc_f32: cuna2_compat_adjoint_f32 for callers that
// cannot allocate device memory.
//
// Everything the transform needs beyond the caller's x, y, f_hat and filter
// lives in one statically sized device array that the library carries (every
// GPU that loads the library holds it until the process exits): the tile
// counters, the sorted sample records, the FFT scratch slab and the twiddle
// tables.  The entry point therefore never calls cudaMalloc / cudaFree or
// cuFFT.  Limits: n <= kNoAllocMaxN samples and a power-of-two grid of at
// most 2^kNoAllocMaxLogNg cells.
//
// The first call on a device sets that device up: it looks up the array's
// device address with cudaGetSymbolAddress (host code may not use the symbol
// itself as a pointer), fills the twiddle tables with a kernel and
// synchronises the caller's stream.  Make that first call before any stream
// capture.  All calls share the one array, which keeps the previous call's
// contents; the tile counters are cleared at the start of every call.  Calls
// that overlap on the GPU (different streams, or different host threads)
// race on the array: serialise them.
// ---------------------------------------------------------------------------
namespace cuna {
namespace {
constexpr int kNoAllocMaxN = 131072;
constexpr int kNoAllocMaxLogNg = 17;
constexpr size_t kNoAllocOffCounts = 0, kNoAllocOffOffsets = 256, kNoAllocOffCursor = 512;
constexpr size_t kNoAllocOffRecs = 1024;
constexpr size_t kNoAllocOffFft = kNoAllocOffRecs + sizeof(RecF) * 2 * (size_t)kNoAllocMaxN;
constexpr size_t kNoAllocOffTw = kNoAllocOffFft + sizeof(float2) * ((size_t)1 << kNoAllocMaxLogNg);
constexpr size_t kNoAllocTwEntries = 48 * 1024;  // all tables for logL = 0..17 (about 41K entries)
constexpr size_t kNoAllocBytes = kNoAllocOffTw + sizeof(float2) * kNoAllocTwEntries;
constexpr int kNoAllocMaxDevices = 64;
}  // namespace
}  // namespace cuna

static __device__ __align__(256) unsigned char cuna_noalloc_scratch[cuna::kNoAllocBytes];

namespace cuna {
namespace {

// exp(+2 pi i (q * step mod denom) / denom) for q < count, evaluated in double
__global__ void k_noalloc_twiddles(float2 *dst, int count, int step, int denom) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < count) {
    const long long num = ((long long)q * step) % denom;
    double s, c;
    sincospi(2.0 * (double)num / (double)denom, &s, &c);
    dst[q] = make_float2((float)c, (float)s);
  }
}

struct NoAllocDev {
  bool ready = false;
  unsigned char *base = nullptr;
  int sms = 1;
  FftDev<float> tab[kNoAllocMaxLogNg + 1];
};
std::mutex g_noalloc_mu;
NoAllocDev g_noalloc[kNoAllocMaxDevices];

int noalloc_table(float2 *tw, size_t &used, int count, int step, int denom, const float2 **out,
                  cudaStream_t st) {
  if (used + (size_t)count > kNoAllocTwEntries) return fail(CUNA2_ERROR_UNSUPPORTED, "twiddle region too small");
  float2 *dst = tw + used;
  k_noalloc_twiddles<<<(count + 255) / 256, 256, 0, st>>>(dst, count, step, denom);
  CUNA_CK(cudaGetLastError());
  used += (size_t)count;
  *out = dst;
  return CUNA2_SUCCESS;
}

// Once per device: device address of the array, twiddle tables, SM count.
int noalloc_setup(int dev, cudaStream_t st, NoAllocDev **out) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoAllocDev &d = g_noalloc[dev];
  if (!d.ready) {
    // set-up launches kernels and synchronises the stream, which a stream
    // capture cannot contain: refuse before touching anything
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    CUNA_CK(cudaStreamIsCapturing(st, &cs));
    if (cs != cudaStreamCaptureStatusNone)
      return fail(CUNA2_ERROR_UNSUPPORTED,
                  "no-allocation entry point: the first call on a device sets it up and must come before any "
                  "stream capture");
    void *p = nullptr;
    CUNA_CK(cudaGetSymbolAddress(&p, cuna_noalloc_scratch));
    d.base = (unsigned char *)p;
    CUNA_CK(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
    float2 *tw = (float2 *)(d.base + kNoAllocOffTw);
    size_t used = 0;
    for (int logL = 0; logL <= kNoAllocMaxLogNg; ++logL) {
      FftDev<float> &f = d.tab[logL];
      const int L = 1 << logL;
      f.logL = logL;
      if (logL <= kSingleLogF32) {
        f.logL1 = logL;
        f.logL2 = 0;
      } else {
        f.logL1 = (logL + 1) / 2;
        f.logL2 = logL / 2;
      }
      const int L1 = 1 << f.logL1, L2 = 1 << f.logL2, nlo = L < 2048 ? L : 2048;
      CUNA_TRY(noalloc_table(tw, used, L1, 1, L1, &f.tw1, st));
      CUNA_TRY(noalloc_table(tw, used, L2, 1, L2, &f.tw2, st));
      if (logL > kSingleLogF32) {
        CUNA_TRY(noalloc_table(tw, used, nlo, 1, L, &f.twlo, st));
        CUNA_TRY(noalloc_table(tw, used, L / nlo, nlo, L, &f.twhi, st));
      } else {  // single-CTA lengths read tw1 only
        f.twlo = nullptr;
        f.twhi = nullptr;
      }
    }
    CUNA_CK(cudaFuncSetAttribute(k_fft_single_compat<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 200 * 1024));
    CUNA_CK(cudaFuncSetAttribute(k_fft_colpass<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    CUNA_CK(cudaFuncSetAttribute(k_fft_rowpass_compat<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 200 * 1024));
    CUNA_CK(cudaStreamSynchronize(st));
    d.ready = true;
  }
  *out = &d;
  return CUNA2_SUCCESS;
}

int compat_adjoint_noalloc(const float *x, const float *y, float2 *f_hat, int n, int ng,
                           const cuna2_filter_properties_f32 *dfp, cudaStream_t st) {
  clear_error();
  CUNA_TRY(check_args(n, ng, 1, x, f_hat, dfp));
  if (n > kNoAllocMaxN)
    return fail(CUNA2_ERROR_UNSUPPORTED, "no-allocation entry point: n = %d exceeds its maximum of %d samples",
                n, kNoAllocMaxN);
  if ((ng & (ng - 1)) != 0 || ilog2i(ng) > kNoAllocMaxLogNg)
    return fail(CUNA2_ERROR_UNSUPPORTED,
                "no-allocation entry point: ng = %d must be a power of two of at most %d", ng,
                1 << kNoAllocMaxLogNg);
  int dev = 0;
  CUNA_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(CUNA2_ERROR_UNSUPPORTED, "device index %d", dev);
  NoAllocDev *d = nullptr;
  CUNA_TRY(noalloc_setup(dev, st, &d));
  int *counts = (int *)(d->base + kNoAllocOffCounts);
  int *offsets = (int *)(d->base + kNoAllocOffOffsets);
  int *cursor = (int *)(d->base + kNoAllocOffCursor);
  RecF *recs = (RecF *)(d->base + kNoAllocOffRecs);
  float2 *scratch = (float2 *)(d->base + kNoAllocOffFft);
  const int ntiles = (ng + (1 << kCompatLogTL) - 1) >> kCompatLogTL;
  // the counters must start at zero; the rest is fully rewritten below
  CUNA_CK(cudaMemsetAsync(counts, 0, sizeof(int) * ntiles, st));
  if (n > 0) {
    SampCompat<float, false> sp{x, y, dfp, n, ng};
    const size_t smc = sizeof(int) * ntiles;
    const int gcount = (int)std::min<int64_t>((n + 4095) / 4096, 4 * d->sms);
    const int gscat = (int)((n + 512 * kScatterItems - 1) / (512 * kScatterItems));
    k_bin_count<<<gcount, 512, smc, st>>>(sp, counts, ntiles);
    CUNA_CK(cudaGetLastError());
    k_scan_tiles<<<1, 1024, 0, st>>>(counts, offsets, cursor, ntiles);
    CUNA_CK(cudaGetLastError());
    k_bin_scatter<<<gscat, 512, 2 * smc, st>>>(sp, offsets, cursor, recs, ntiles);
    CUNA_CK(cudaGetLastError());
    const size_t smg = compat_grid_smem<float>();
    k_grid_compat<float, false, kCompatThreadsFew><<<dim3(ntiles, 1), kCompatThreadsFew, smg, st>>>(recs, offsets, f_hat, ng, dfp, y, n, 0u);
    CUNA_CK(cudaGetLastError());
  }
  const int logL = ilog2i(ng);
  const FftDev<float> &f = d->tab[logL];
  if (logL <= kSingleLogF32) {
    const int threads = std::max(32, ng / kFftE);
    const size_t smem = sizeof(float2) * (size_t)fft_pitch(ng, 1);
    k_fft_single_compat<float><<<1, threads, smem, st>>>(f_hat, f, dfp, 1);
    CUNA_CK(cudaGetLastError());
    return CUNA2_SUCCESS;
  }
  const int threads = kPassElemsF32 / kFftE;
  const int L1 = 1 << f.logL1, L2 = 1 << f.logL2;
  const int BA = kPassElemsF32 / L1, BB = kPassElemsF32 / L2;
  const size_t smemA = sizeof(float2) * (size_t)BA * fft_pitch(L1, BA);
  const size_t smemB = sizeof(float2) * (size_t)BB * fft_pitch(L2, BB);
  k_fft_colpass<float><<<dim3(L2 / BA, 1), threads, smemA, st>>>(f_hat, scratch, f, (int64_t)ng);
  CUNA_CK(cudaGetLastError());
  k_fft_rowpass_compat<float><<<dim3(L1 / BB, 1), threads, smemB, st>>>(scratch, f_hat, f, dfp, (int64_t)ng, 1);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

}  // namespace
}  // namespace cuna

extern "C" int cuna2_compat_adjoint_noalloc_f32(const float *x, const float *y, float2 *f_hat, int n, int ng,
                                                const cuna2_filter_properties_f32 *d, cudaStream_t st) {
  return compat_adjoint_noalloc(x, y, f_hat, n, ng, d, st);
}
