// accurate_kernels.cuh -- device code of accurate mode, shared by the
// single-series plans (accurate.cu) and the batched plans (batch.cu).
//
//   F_k = sum_j y_j exp(+2 pi i k x_j),  x_j = (t_j - t0)/T - 1/2,
//   k = -nf/2 .. nf/2-1 stored at F[k + nf/2].
//
// Math: Gaussian gridding on a periodic grid of ng = R nf cells with kernel
// psi(d) = exp(-d^2 / (4 tau)), tau = m R / (4 pi (R - 1/2)) (Greengard & Lee
// 2004), taps d = -m+1..m around floor(s_j), s_j = (x_j + 1/2) ng.  The grid is
// real, so it is transformed as ng/2 packed complex points and unpacked in the
// last FFT pass, where the deconvolution 1/psi_hat(k), the (-1)^k phase of the
// x + 1/2 origin shift, output selection |k| <= nf/2 and Hermitian completion
// are fused in.  The grid position is reduced in 64-bit fixed point
// (phase.cuh).
//
// Each kernel's work is a __device__ body taking the per-series parameters,
// so that the single-series kernels and the batched work-list kernels share
// it.
#pragma once
#include <math.h>
#include <algorithm>
#include <type_traits>
#include "binning.cuh"
#include "fft.cuh"
#include "phase.cuh"
#include "rng.cuh"
#include "runtime.h"

namespace cuna {
namespace {

constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ void sincospi_t(float a, float *s, float *c) { sincospif(a, s, c); }
__device__ __forceinline__ void sincospi_t(double a, double *s, double *c) { sincospi(a, s, c); }
__device__ __forceinline__ float exp_t(float a) { return expf(a); }
__device__ __forceinline__ double exp_t(double a) { return exp(a); }
__device__ __forceinline__ float exp2_t(float a) { return exp2f(a); }
__device__ __forceinline__ double exp2_t(double a) { return exp2(a); }

// Everything a kernel needs about the Gaussian and the output.
template <typename T> struct AccParams {
  int64_t ng, nf, K;  // K = nf / 2
  int m, logTL, ntiles;
  T k1, k2;           // E1 = 2^(-k1 f^2), E2 = 2^(k2 f)   (f = fractional cell)
  T e3c;              // E3[d] = exp(e3c d^2)
  T c0, c1;           // 0.5 / psi_hat(k) = c0 exp(c1 k^2)
  T twk;              // 2 / ng  (unpack twiddle angle / pi)
  bool masks;         // the gather masks a record's taps (tail_free_gather)
};

// fractional cell from the low word of S*ng
// (the float version converts a 32-bit integer: 64-bit integer to float
// conversions run on the narrow FP64 pipe of GB300)
__device__ __forceinline__ float frac_of(uint64_t lo, float) {
  return (float)(uint32_t)(lo >> 40) * 5.9604644775390625e-08f;
}
__device__ __forceinline__ double frac_of(uint64_t lo, double) {
  return (double)(lo >> 11) * 1.1102230246251565e-16;
}

// cell and fractional cell of the phase S = frac(x + 1/2) * 2^64
template <typename T>
__device__ __forceinline__ void cell_of_phase(uint64_t S, int64_t ng, int &cell, T &f) {
  if ((ng & (ng - 1)) == 0) {  // ng = 2^g: the top g bits are the cell
    const int g = 63 - __clzll((long long)ng);
    cell = g ? (int)(S >> (64 - g)) : 0;
    f = frac_of(S << g, (T)0);
  } else {
    cell = (int)umulhi64(S, (uint64_t)ng);
    f = frac_of(S * (uint64_t)ng, (T)0);
  }
}

template <typename T>
__device__ __forceinline__ void reduce_sample(double t, const PhaseMul &pm, int64_t ng, int &cell, T &f) {
  cell_of_phase<T>(phase_of(t, pm), ng, cell, f);
}

// ---------------------------------------------------------------------------
// epilogue: real unpack + deconvolution + centring, one output k in [0, K]
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void acc_output(const AccParams<T> &e, int64_t k, typename CxOf<T>::type Zk,
                                           typename CxOf<T>::type Zmc, typename CxOf<T>::type *F) {
  typedef typename CxOf<T>::type C;
  const C A = cadd(Zk, Zmc);
  const C Bv = cmuli(csub(Zmc, Zk));
  T sn, cs;
  const T kf = (T)(int)k;  // k <= nf/2 < 2^31; a 32-bit conversion
  sincospi_t(kf * e.twk, &sn, &cs);
  const C G2 = cadd(A, cmul(cmk(cs, sn), Bv));
  T sc = e.c0 * exp_t(e.c1 * kf * kf);
  if (k & 1) sc = -sc;
  const C Fk = cscale(G2, sc);
  if (k < e.K) F[e.K + k] = Fk;
  if (k >= 1) F[e.K - k] = cconj(Fk);
}

__device__ __forceinline__ int real_slot(int c) { return 2 * pad16(c >> 1) + (c & 1); }

// exclusive scan in place of v[0..n), v[n] = total, by the whole CTA; ends
// with a barrier
__device__ __forceinline__ void cta_scan_in_place(int *v, int n) {
  __shared__ int wsum[32];
  const int nt = blockDim.x, tid = threadIdx.x;
  const int per = (n + nt - 1) / nt;
  const int beg = min(tid * per, n), end = min(beg + per, n);
  int sum = 0;
  for (int i = beg; i < end; ++i) sum += v[i];
  const int lane = tid & 31, w = tid >> 5;
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    int q = lane < (nt >> 5) ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, q, o);
      if (lane >= o) q += u;
    }
    wsum[lane] = q;
  }
  __syncthreads();
  int run = x - sum + (w > 0 ? wsum[w - 1] : 0);
  for (int i = beg; i < end; ++i) {
    const int u = v[i];
    v[i] = run;
    run += u;
  }
  if (tid == nt - 1) v[n] = wsum[(nt >> 5) - 1];
  __syncthreads();
}

// ---------------------------------------------------------------------------
// binning sampler, tiled gridding, last FFT pass
// ---------------------------------------------------------------------------
// Sorted sample record of accurate mode: {cell, fractional cell, value}.
__device__ __forceinline__ void rec_set(RecF &r, int cell, float fr, float y, int idx) {
  r.cell = cell; r.a = fr; r.b = y; r.p = idx;
}
__device__ __forceinline__ void rec_set(RecD &r, int cell, double fr, double y, int idx) {
  r.cell = cell; r.p = idx; r.a = fr; r.b = y; r.v = 0.0;
}

// tiles that the taps of a sample in `cell` reach: their number, 1 or 2
template <typename T> __device__ __forceinline__ int sample_tiles(int cell, const AccParams<T> &e, int *t) {
  const int ng = (int)e.ng;
  int lo = cell - e.m + 1, hi = cell + e.m;
  if (lo < 0) lo += ng;
  if (hi >= ng) hi -= ng;
  t[0] = lo >> e.logTL;
  t[1] = hi >> e.logTL;
  return t[0] == t[1] ? 1 : 2;
}

template <typename T> struct SampAcc {
  typedef typename RecOf<T>::type Rec;
  struct Raw {
    double t;
    T y;
  };
  const double *t;
  const T *y;
  int64_t n;
  PhaseMul pm;
  AccParams<T> e;
  uint64_t *sc = nullptr;  // optional: phases written here for SampAccS
  __device__ __forceinline__ Raw load(int64_t i, bool with_value) const {
    Raw r;
    r.t = t[i];
    if (with_value) r.y = y[i];
    return r;
  }
  __device__ __forceinline__ void prep(int64_t i, const Raw &r, Prep<Rec> &p) const {
    int cell;
    T fr;
    const uint64_t S = phase_of(r.t, pm);
    if (sc) sc[i] = S;
    cell_of_phase<T>(S, e.ng, cell, fr);
    p.nt = sample_tiles(cell, e, p.t);
    rec_set(p.rec, cell, fr, r.y, (int)i);
  }
};

// Sampler over phases cached by a SampAcc pass (sc[i] = phase of t[i]): the
// scatter pass of the binning then skips the phase reduction.
template <typename T> struct SampAccS {
  typedef typename RecOf<T>::type Rec;
  struct Raw {
    uint64_t S;
    T y;
  };
  const uint64_t *sc;
  const T *y;
  int64_t n;
  AccParams<T> e;
  __device__ __forceinline__ Raw load(int64_t i, bool with_value) const {
    Raw r;
    r.S = __ldcg(reinterpret_cast<const unsigned long long *>(sc) + i);  // written by the count pass
    if (with_value) r.y = y[i];
    return r;
  }
  __device__ __forceinline__ void prep(int64_t i, const Raw &r, Prep<Rec> &p) const {
    int cell;
    T fr;
    cell_of_phase<T>(r.S, e.ng, cell, fr);
    p.nt = sample_tiles(cell, e, p.t);
    rec_set(p.rec, cell, fr, r.y, (int)i);
  }
};

// The whole bucket sort of a short series in one launch, by a cluster of eight
// CTAs: each keeps the phases of its eighth of the samples and their tile
// histogram in shared memory; after a cluster barrier every CTA adds up the
// eight histograms through distributed shared memory (the totals, scanned, are
// the offsets; the sum over the CTAs before it is where its own records go) and
// writes its records.  It replaces a memset, a count and a scatter launch, which
// a short transform's host time is made of.  One CTA would be bound by the
// instructions of the phases (n = 10000: 17.9 us; the cluster 8.9; memset
// and two launches of 20 CTAs 8.3 us and three launch gaps).
constexpr int kBinOneCtas = 8, kBinOneThreads = 512;
constexpr int kBinOneN = 16384;  // 2048 samples per CTA
inline size_t bin_one_smem(int64_t n, int ntiles) {
  const int64_t per = (n + kBinOneCtas - 1) / kBinOneCtas;
  return sizeof(uint64_t) * (size_t)per + sizeof(int) * (2 * (size_t)ntiles + 1);
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the 32-bit word at shared address `p` of CTA `rank` of the cluster
__device__ __forceinline__ int cluster_load(const int *p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(r) : "memory");
  return v;
}

template <typename T>
__global__ void __cluster_dims__(kBinOneCtas, 1, 1) __launch_bounds__(kBinOneThreads)
    k_bin_one(SampAcc<T> smp, int *offsets, typename RecOf<T>::type *recs, int ntiles) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int n = (int)smp.n, per = (n + kBinOneCtas - 1) / kBinOneCtas, rank = blockIdx.x;
  const int i0 = rank * per, i1 = min(n, i0 + per);
  uint64_t *ph = reinterpret_cast<uint64_t *>(smem_raw);
  int *hist = reinterpret_cast<int *>(ph + per);  // this CTA's records per tile
  int *cur = hist + ntiles;                       // ntiles + 1: totals, then the next free place of each tile
  pdl_trigger();
  for (int t = threadIdx.x; t < ntiles; t += kBinOneThreads) hist[t] = 0;
  __syncthreads();
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < i1; i += kBinOneThreads) {
    const uint64_t S = phase_of(smp.t[i], smp.pm);
    ph[i - i0] = S;
    int cell, t[2];
    T fr;
    cell_of_phase<T>(S, smp.e.ng, cell, fr);
    const int nt = sample_tiles(cell, smp.e, t);
    for (int q = 0; q < nt; ++q) atomicAdd(&hist[t[q]], 1);
  }
  cluster_barrier();
  constexpr int TPT = kScanFuseTiles / kBinOneThreads;
  int before[TPT];
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int t = threadIdx.x + k * kBinOneThreads;
    before[k] = 0;
    if (t >= ntiles) continue;
    int tot = 0;
#pragma unroll
    for (int c = 0; c < kBinOneCtas; ++c) {
      const int h = cluster_load(hist + t, c);
      before[k] += c < rank ? h : 0;
      tot += h;
    }
    cur[t] = tot;
  }
  __syncthreads();
  cta_scan_in_place(cur, ntiles);
  if (rank == 0)
    for (int t = threadIdx.x; t <= ntiles; t += kBinOneThreads) offsets[t] = cur[t];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < TPT; ++k) {
    const int t = threadIdx.x + k * kBinOneThreads;
    if (t < ntiles) cur[t] += before[k];
  }
  __syncthreads();
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < i1; i += kBinOneThreads) {
    int cell, t[2];
    T fr;
    cell_of_phase<T>(ph[i - i0], smp.e.ng, cell, fr);
    const int nt = sample_tiles(cell, smp.e, t);
    typename RecOf<T>::type r;
    rec_set(r, cell, fr, smp.y[i], i);
    for (int q = 0; q < nt; ++q) rec_store(recs + atomicAdd(&cur[t[q]], 1), r);
  }
  cluster_barrier();  // no CTA leaves while another may read its histogram
}

// ---------------------------------------------------------------------------
// Gridding, gather form.  One CTA owns tile [base, base + TL) of the grid and
// the records binned to it (its own samples plus the halo samples within m
// cells of its edges).  Per chunk of at most CAP records it counting-sorts
// them in shared memory by group of CW consecutive local slots (slot lc =
// cell - base + m; integer atomics only), then every thread sums, for each
// of its CW cells c, the records of the groups covering slots [c - base,
// c - base + 2m): w = y exp(-(d - f)^2 / (4 tau)), d = c - cell (records of
// those groups outside the window are masked, or, in the unmasked form, add
// their negligible tail).  Partial sums stay in registers across chunks and
// are written once, coalesced.  No floating-point atomics.
// ---------------------------------------------------------------------------
template <typename T> struct GridCfg;
template <> struct GridCfg<float> { static constexpr int CAP = 1024; };
template <> struct GridCfg<double> { static constexpr int CAP = 512; };
constexpr int kGridThreads = 256;
constexpr int kGridMaxCpt = 16;  // cells per thread: TL <= 4096

// 2^x with the hardware approximation (relative error < 2^-22 over the range
// used here; arguments are <= 0 and results below 2^-126 flush to zero, far
// beneath the 1e-6 accuracy of the float path).
__device__ __forceinline__ float ex2_fast(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float gauss_w(float y, float dd, float k1) { return y * ex2_fast(-k1 * dd * dd); }
__device__ __forceinline__ double gauss_w(double y, double dd, double k1) { return y * exp2(-k1 * dd * dd); }

// a placed record in shared memory: fractional cell, value, slot
template <typename T> struct __align__(2 * sizeof(T) >= 16 ? 16 : 16) SRec {
  T f, y;
  int lc, pad;
};

// exp2 for the gridding weights: ex2.approx for float (relative error of a
// few ulp), the library exp2 for double
__device__ __forceinline__ float exp2_g(float x) { return ex2_fast(x); }
__device__ __forceinline__ double exp2_g(double x) { return exp2(x); }

// Weights y exp2(-k1 (x + i)^2) of one record for CW consecutive cells,
// i = 0..CW-1, by the fast Gaussian gridding factorisation (Greengard & Lee
// 2004) about the middle cell h = CW/2, xc = x + h:
//   y exp2(-k1 (xc + j)^2) = E Q^j c_j,  E = y exp2(-k1 xc^2),
//   Q = exp2(-2 k1 xc), c_j = exp2(-k1 j^2),
// three exp2 per record and cell group instead of CW.  Centring keeps E and
// the running products inside the float range for every m <= 16.
template <typename T, int CW> struct GaussCW {
  T c[CW / 2 + 1];
  __device__ explicit GaussCW(T k1) {
#pragma unroll
    for (int j = 0; j <= CW / 2; ++j) c[j] = exp2_g(-k1 * (T)(j * j));
  }
};
template <typename T, int CW>
__device__ __forceinline__ void gauss_cw(T y, T x, T k1, const GaussCW<T, CW> &g, T *w) {
  constexpr int H = CW / 2;
  const T xc = x + (T)H;
  const T E = y * exp2_g(-k1 * xc * xc);
  const T Q = exp2_g((T)(-2) * k1 * xc), Qi = exp2_g((T)2 * k1 * xc);
  w[H] = E;
  T u = E;
#pragma unroll
  for (int j = 1; j < CW - H; ++j) {
    u *= Q;
    w[H + j] = u * g.c[j];
  }
  u = E;
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    u *= Qi;
    w[H - j] = u * g.c[j];
  }
}

// a[i] += y exp2(-k1 (x + i)^2) for the cells i a record in slot rel = lc - cl0
// reaches (0 <= rel - i < w2, w2 = 2m), by the centred factorisation of
// gauss_cw; the mask is applied before the last product so that each tap is
// one select and one fused multiply-add.
// MASKED == false adds the record to all CW cells: cells outside its taps
// lie more than m cells from it, where the Gaussian is below 2^(-k1 m^2) of
// its peak; the plan takes this form only where that bound is negligible
// (tail_free_gather), and then each tap is one product and one fused
// multiply-add.
template <typename T, int CW, bool MASKED = true>
__device__ __forceinline__ void gauss_acc(T y, T x, T k1, const GaussCW<T, CW> &g, int rel, int w2, T *a) {
  constexpr int H = CW / 2;
  const T xc = x + (T)H;
  const T E = y * exp2_g(-k1 * xc * xc);
  const T Q = exp2_g((T)(-2) * k1 * xc), Qi = exp2_g((T)2 * k1 * xc);
  if (MASKED) a[H] += (unsigned)(rel - H) < (unsigned)w2 ? E : (T)0;
  else a[H] += E;
  T u = E;
#pragma unroll
  for (int j = 1; j < CW - H; ++j) {
    u *= Q;
    if (MASKED) a[H + j] = fma((unsigned)(rel - H - j) < (unsigned)w2 ? u : (T)0, g.c[j], a[H + j]);
    else a[H + j] = fma(u, g.c[j], a[H + j]);
  }
  u = E;
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    u *= Qi;
    if (MASKED) a[H - j] = fma((unsigned)(rel - H + j) < (unsigned)w2 ? u : (T)0, g.c[j], a[H - j]);
    else a[H - j] = fma(u, g.c[j], a[H - j]);
  }
}

// 2^x of two values, -126 <= x <= 1, on the FP32 pipe: 2^n p(r), n the integer
// nearest x, p the polynomial of degree 6 with the least maximal relative error
// on [-1/2, 1/2] (weighted least squares, Lawson's iteration; 2e-9).  In floats
// 8e-8 at most and 2.7e-8 rms, where ex2.approx has 2^-22.
__device__ __forceinline__ void exp2_pair(f2 x, float &a, float &b) {
  const f2 M = pk2(12582912.f, 12582912.f), t = add2(x, M), r = sub2(x, sub2(t, M));  // n in the low bits of t
  f2 p = pk2(0x1.41d332p-13f, 0x1.41d332p-13f);
  p = fma2(p, r, pk2(0x1.5f456ap-10f, 0x1.5f456ap-10f));
  p = fma2(p, r, pk2(0x1.3b2dbcp-7f, 0x1.3b2dbcp-7f));
  p = fma2(p, r, pk2(0x1.c6aed4p-5f, 0x1.c6aed4p-5f));
  p = fma2(p, r, pk2(0x1.ebfbdap-3f, 0x1.ebfbdap-3f));
  p = fma2(p, r, pk2(0x1.62e43p-1f, 0x1.62e43p-1f));
  p = fma2(p, r, pk2(1.f, 1.f));
  float t0, t1;
  unpk2(t, t0, t1);
  unpk2(p, a, b);
  a = __int_as_float(__float_as_int(a) + (__float_as_int(t0) << 23));
  b = __int_as_float(__float_as_int(b) + (__float_as_int(t1) << 23));
}

// a[i] += y exp2(-k1 (j + i - f)^2), i = 0..3, the weights one by one: j the
// distance in cells of the first one from the record's own, f its fraction.
// The transforms whose FFT one CTA holds gather with it: gauss_acc's powers of Q
// carry the rounding of the middle cell's exponents, which beside their short
// FFTs would show.  From R = 4 on, where three quarters of the FFT's error fall
// outside the band, so would ex2.approx's, hence the polynomial there.
// Relative error of the spectrum, mean of 32 series, by the scatter / gauss_acc
// / ex2.approx per tap / polynomial: n = 1000, Nf = 2048, R = 2: 2.13 / 2.27 /
// 1.97 / 1.93e-7; n = 300, Nf = 2048, R = 4, m = 12: 1.38 / 1.56 / 1.40 /
// 1.24e-7; n = 700, Nf = 1024, R = 4, m = 6: 1.43 / 1.53 / 1.47 / 1.28e-7.
enum GatherForm { kGatherMasked, kGatherFree, kGatherPoly };  // Poly: masked too (x < -126 outside the window)
template <int FORM> __device__ __forceinline__ void gauss_acc4(float y, int j, float f, float k1, int m, float *a) {
  const float fj = (float)j;
  const f2 nf = pk2(-f, -f), nk = pk2(-k1, -k1);
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const f2 d = add2(pk2(fj + (float)i, fj + (float)(i + 1)), nf), x = mul2(mul2(nk, d), d);
    float w0, w1;
    if constexpr (FORM == kGatherPoly) {
      exp2_pair(x, w0, w1);
    } else {
      float x0, x1;
      unpk2(x, x0, x1);
      w0 = exp2_g(x0);
      w1 = exp2_g(x1);
    }
    a[i] = fmaf(FORM == kGatherFree || (unsigned)(m - j - i) < (unsigned)(2 * m) ? w0 : 0.f, y, a[i]);
    a[i + 1] = fmaf(FORM == kGatherFree || (unsigned)(m - j - i - 1) < (unsigned)(2 * m) ? w1 : 0.f, y, a[i + 1]);
  }
}

// ---------------------------------------------------------------------------
// single-CTA transform for small grids
// ---------------------------------------------------------------------------
// Whole transform of one series in one CTA: gridding straight into shared
// memory (the grid is the packed complex FFT buffer), FFT, epilogue.
//
// Two griddings.  Scatter: a thread per sample adds its 2m taps with shared
// atomics (float: compare-and-swap loops, 3 adds per clock and SM).  Gather
// (float): the samples go in chunks of up to small_cap records; a chunk is
// counting-sorted in shared memory by group of four cells (one atomic per
// record ranks it, the gather reads it through an index), then every thread
// sums its groups of four cells over the records in reach, as the tiled gather
// does, with no floating-point atomics.  The gather visits every group once
// per chunk, so it pays on small grids: in a batch (four samples per grid of
// 16 to 32 cells) 21 -> 11 us for 2^10-cell grids and 20 -> 18 us at 2^12
// cells, but 29 -> 34 us at 2^13 and 114 -> 171 us at 2^15; a transform with an
// SM to itself takes it to 2^14 cells.  One transform of n = 1000, Nf = 2048,
// R = 2, m = 8: 28.7 us per call with L / 16 threads and the scatter, 10.3 us
// here (by one cluster, cluster.cuh).
inline bool small_gather(int L, bool alone, bool is_float) { return is_float && L <= (alone ? 8192 : 2048); }
// records of a chunk (0: scatter).  With an SM to itself a transform takes the
// most, fewer chunks of five barriers each; in a batch the shared memory of
// CTAs that share an SM counts.  On the device, with a group's records shared
// out to its idle threads: 2000 samples on 64 cells 160 us in chunks of 32,
// 10.9 in one; 500 samples on 2^11 cells 6.1 either way.
constexpr int kSmallCapMax = 2048;
// Whether a series of n samples is gathered, where the launch has room for it:
// from R = 4 on, whose weights are polynomials, in a batch only with as many
// samples as packed points (1024 resamples of 200 samples, Nf = 1024, R = 4, m =
// 12: 30 us by the scatter, 37 gathered; 4000 series of 300, Nf = 512: 67 and 73;
// 1024 of 2000, Nf = 512: 127 and 104).
__host__ __device__ inline bool small_gathers(int cap, int64_t n, int L, int64_t R) {
  return cap > 0 && (cap == kSmallCapMax || R < 4 || n >= L);
}
inline int small_cap(int L, bool alone, bool is_float) {
  if (!small_gather(L, alone, is_float)) return 0;
  return alone ? kSmallCapMax : std::max(32, std::min(kSmallCapMax, L / 2));
}
// shared bytes: FFT buffer | gather: records, index, group starts; scatter: E3
template <typename T> size_t small_smem(int L, int m, int cap) {
  const size_t fft = sizeof(typename CxOf<T>::type) * (size_t)fft_pitch(L, 1);
  if (cap == 0) return fft + sizeof(T) * (2 * m + 2);
  return ((fft + 15) & ~(size_t)15) + (size_t)cap * (sizeof(SRec<float>) + sizeof(int)) +
         sizeof(int) * ((size_t)(2 * L) / 4 + 1);
}
// threads of a small transform: the FFT keeps L / 16 busy, the samples, groups
// and outputs more; `alone`: the launch has an SM per transform
template <typename T> int small_threads(int L, bool alone, int cap) {
  const int most = sizeof(T) == 4 ? 1024 : 512;
  const int want = cap ? (alone ? std::max(L / 2, 256) : L / 8) : (alone ? most : L / kFftE);
  return std::max(std::max(32, std::min(most, L / kFftE)), std::min(most, want));
}

// the four cells of group g from the sorted records of one chunk, added to
// a[]: records of the groups that hold cells 4g - m .. 4g + m + 2, whose
// indices wrap around the periodic grid (images o = -1, 0, 1)
template <int FORM>
__device__ __forceinline__ void small_gather4(const SRec<float> *srec, const int *order, const int *start, int g, int NG,
                                              int ng, int m, float k1, int part, int step, float *a) {
  const int c0 = 4 * g;
  const int glo = (c0 - m) >> 2, ghi = (c0 + m + 2) >> 2;
#pragma unroll 1
  for (int o = -1; o <= 1; ++o) {
    const int lo = max(glo, o * NG) - o * NG, hi = min(ghi, o * NG + NG - 1) - o * NG;
    if (lo > hi) continue;
    const int c = c0 - o * ng;  // the group's first cell as this image sees it
    const int re = start[hi + 1];
    for (int r = start[lo] + part; r < re; r += step) {
      const SRec<float> q = srec[order[r]];
      gauss_acc4<FORM>(q.y, c - q.lc, q.f, k1, m, a);
    }
  }
}

__device__ __forceinline__ void small_grid_gather(const double *__restrict__ t, const float *__restrict__ y, int64_t n,
                                                  const PhaseMul &pm, const AccParams<float> &e, float *sr,
                                                  SRec<float> *srec, int *order, int *start, int cap) {
  const int ng = (int)e.ng, NG = ng / 4, m = e.m;
  const bool masked = e.masks, poly = e.ng >= 4 * e.nf;
  // Where there are fewer groups than threads, 2^LP threads share a group's
  // records (NG is a power of two: with LP > 0 either all threads have a group
  // or, at LP = 5, whole warps have none).
  int LP = 0;
  while (LP < 5 && (NG << LP) < (int)blockDim.x) ++LP;
  const int part = threadIdx.x & ((1 << LP) - 1), step = 1 << LP;
  int64_t c0 = 0;
  do {
    const int cnt = (int)min((int64_t)cap, n - c0);
    if (c0 > 0) __syncthreads();  // the previous chunk's gather is done with the starts and records
    for (int i = threadIdx.x; i < NG; i += blockDim.x) start[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
      SRec<float> r;
      reduce_sample<float>(t[c0 + i], pm, e.ng, r.lc, r.f);
      r.y = y[c0 + i];
      r.pad = atomicAdd(&start[r.lc >> 2], 1);  // rank within its group
      srec[i] = r;
    }
    __syncthreads();
    cta_scan_in_place(start, NG);
    for (int i = threadIdx.x; i < cnt; i += blockDim.x) order[start[srec[i].lc >> 2] + srec[i].pad] = i;
    __syncthreads();
    for (int g = threadIdx.x >> LP; g < NG; g += blockDim.x >> LP) {
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      if (poly) small_gather4<kGatherPoly>(srec, order, start, g, NG, ng, m, e.k1, part, step, a);
      else if (masked) small_gather4<kGatherMasked>(srec, order, start, g, NG, ng, m, e.k1, part, step, a);
      else small_gather4<kGatherFree>(srec, order, start, g, NG, ng, m, e.k1, part, step, a);
      for (int o = 1; o < step; o <<= 1) {  // whole warps: see LP
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
      }
      if (part == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float &d = sr[real_slot(4 * g + i)];
          d = c0 == 0 ? a[i] : d + a[i];
        }
      }
    }
    c0 += cap;
  } while (c0 < n);
}

template <typename T>
__device__ __forceinline__ void nfft_small_body(const double *__restrict__ t, const T *__restrict__ y,
                                                int64_t n, const PhaseMul &pm, const AccParams<T> &e,
                                                const FftDev<T> &f, typename CxOf<T>::type *F, int cap) {
  typedef typename CxOf<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 1 << f.logL;
  const int pitch = fft_pitch(L, 1);
  C *s = reinterpret_cast<C *>(smem_raw);
  T *sr = reinterpret_cast<T *>(smem_raw);
  if (small_gathers(cap, n, L, e.ng / e.nf)) {
    if constexpr (sizeof(T) == 4) {
      SRec<float> *srec = reinterpret_cast<SRec<float> *>(smem_raw + ((sizeof(C) * pitch + 15) & ~(size_t)15));
      int *order = reinterpret_cast<int *>(srec + cap);
      small_grid_gather(t, y, n, pm, e, sr, srec, order, order + cap, cap);
    }
  } else {
    T *e3 = reinterpret_cast<T *>(s + pitch);
    const int m = e.m, ng = (int)e.ng;
    for (int i = threadIdx.x; i < 2 * pitch; i += blockDim.x) sr[i] = (T)0;
    for (int d = threadIdx.x; d <= 2 * m; d += blockDim.x) e3[d] = exp_t(e.e3c * (T)((d - m) * (d - m)));
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      int cell;
      T fr;
      reduce_sample<T>(t[i], pm, e.ng, cell, fr);
      const T E1 = exp2_t(-e.k1 * fr * fr), E2 = exp2_t(e.k2 * fr);
      const T w0 = y[i] * E1;
      T w = w0;
      for (int d = 0; d <= m; ++d) {
        int c = cell + d;
        if (c >= ng) c -= ng;
        atomicAdd(&sr[real_slot(c)], w * e3[d + m]);
        w *= E2;
      }
      const T E2i = (T)1 / E2;
      w = w0 * E2i;
      for (int d = -1; d > -m; --d) {
        int c = cell + d;
        if (c < 0) c += ng;
        atomicAdd(&sr[real_slot(c)], w * e3[d + m]);
        w *= E2i;
      }
    }
  }
  __syncthreads();
  smem_fft<T>(s, pitch, f.logL, 1, f.tw1);
  for (int64_t k = threadIdx.x; k <= e.K; k += blockDim.x) {
    const C Zk = s[pad16((int)(k & (L - 1)))];
    const C Zm = cconj(s[pad16((int)((L - k) & (L - 1)))]);
    acc_output<T>(e, k, Zk, Zm, F);
  }
}

template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512) k_nfft_small(const double *__restrict__ t, const T *__restrict__ y,
                                                     int64_t n, PhaseMul pm, AccParams<T> e, FftDev<T> f,
                                                     typename CxOf<T>::type *F, const T *__restrict__ wts,
                                                     int cap) {
  // one CTA per output slab: slab b grids wts[b*n + j] when wts is given
  // (bootstrap resample b), else y[j]
  if (wts) {
    y = wts + (int64_t)blockIdx.x * n;
    F += (int64_t)blockIdx.x * e.nf;
  }
  nfft_small_body<T>(t, y, n, pm, e, f, F, cap);
}

__device__ __forceinline__ void store4(float *p, float a, float b, float c, float d) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void store4(double *p, double a, double b, double c, double d) {
  reinterpret_cast<double2 *>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2 *>(p)[1] = make_double2(c, d);
}

// Slots (local cell + m) of a record whose cell is p0 cells right of the tile
// base, for every image p = p0 + j*ng (j in {-1, 0, 1}) in [-m, TL + m); the
// second slot exists only when one tile spans the whole periodic grid.
__device__ __forceinline__ void grid_slots(int p0, int ng, int TL, int m, int &s0, int &s1) {
  if (p0 < 0) p0 += ng;
  const int a = p0 - ng >= -m ? p0 - ng + m : -1;
  const int b = p0 < TL + m ? p0 + m : -1;
  const int c = p0 + ng < TL + m ? p0 + ng + m : -1;
  s0 = a >= 0 ? a : (b >= 0 ? b : c);
  s1 = a >= 0 ? (b >= 0 ? b : c) : (b >= 0 ? c : -1);
}

// eight cells, 32-byte aligned, as one sector (two 16-byte stores of a thread
// reach the L2 as half sectors)
__device__ __forceinline__ void store8(float *p, const float *v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}
// asynchronous copy of a 4-byte value to shared memory (zero unless `in`)
__device__ __forceinline__ void cp_async4(float *dst, const float *src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One grid tile [base, base + 2^logTL) from records [r0, r1), for slabs
// [sbeg, send): slab s grids value wts[s*nvals + p] of sample p when wts is
// given (bootstrap), else the record's own value.
// CW consecutive cells per thread in the gather (4 or 8)
// SG > 1 (slab weights given, CW = 8 on 2048-cell tiles): SG slabs share each
// record's Gaussian, computed once per record visit and scaled by each slab's
// value from shared memory.  Bound by the grid's writes and the latency of the
// values' loads (1024 slabs of 2^16 cells, 5000 records, 268 MB: 117 us with
// eight slabs per CTA and the values loaded between two barriers, 93 with 16
// and copies one group ahead, 80 with 32-byte stores).
template <typename T, int CW, class Src, int SG = 1, bool MASKED = true>
__device__ __forceinline__ void grid_tile_body(const Src &recs, int r0, int r1,
                                               int base, T *__restrict__ grid, const AccParams<T> &e,
                                               const T *__restrict__ wts, int64_t nvals, int sbeg, int send,
                                               int64_t slab_stride) {
  typedef typename RecOf<T>::type Rec;
  constexpr int CAP = GridCfg<T>::CAP;
  // cells per thread: up to 16 in groups of 4 (TL <= 4096), or one group of
  // 8 (TL = 2048)
  constexpr int MAXC = CW == 8 ? 8 : kGridMaxCpt;
  constexpr int RPT = CAP / kGridThreads;  // records per thread per chunk
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int TL = 1 << e.logTL, m = e.m, W = TL + 2 * m;
  // records are counting-sorted into groups of CW consecutive slots (slot =
  // local cell + m), the unit of a thread's cell group: NG + 1 counters
  const int NG = (W + CW - 1) / CW;
  const int ng = (int)e.ng;
  int *start = reinterpret_cast<int *>(smem_raw);                                       // NG + 1 groups
  SRec<T> *srec = reinterpret_cast<SRec<T> *>(smem_raw + sizeof(int) * ((W + 2 + 3) & ~3));  // placed records
  int *sp = reinterpret_cast<int *>(srec + CAP);                                         // sample index
  // SG > 1: yv[s * CAP + r], value of slab s for placed record r, two buffers
  T *yv = reinterpret_cast<T *>(sp + CAP);
  static_assert(SG == 1 || CW == 8, "slab groups run with 8-cell groups on 2048-cell tiles");
  __shared__ int wsum[kGridThreads / 32];
  // a single tile spanning the whole grid maps a record to up to two slots;
  // halve the chunk then so that placements never exceed CAP
  const int chunk = (TL + 2 * m > ng) ? CAP / 2 : CAP;
  const int npass = (TL + kGridThreads * CW - 1) / (kGridThreads * CW);  // <= MAXC / CW
  const int nchunks = (r1 - r0 + chunk - 1) / chunk;
  const GaussCW<T, CW> gw(e.k1);
  // the records are sorted once for all slabs when they fit in one chunk
  for (int slab = sbeg; slab < send; slab += SG) {
    T acc[SG][MAXC];
#pragma unroll
    for (int g = 0; g < SG; ++g)
#pragma unroll
      for (int q = 0; q < MAXC; ++q) acc[g][q] = (T)0;
    for (int ck = 0; ck < nchunks; ++ck) {
      const int c0 = r0 + ck * chunk;
      const int cnt = min(chunk, r1 - c0);
      if (nchunks > 1 || slab == sbeg) {
        for (int i = threadIdx.x; i <= NG; i += kGridThreads) start[i] = 0;
        __syncthreads();
        // load this thread's records; each maps to up to two slots (two only
        // when the tile wraps onto itself, i.e. one tile spans the whole grid)
        Rec rc[RPT];
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
          const int i = threadIdx.x + u * kGridThreads;
          if (i < cnt) rc[u] = recs[c0 + i];
        }
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
          const int i = threadIdx.x + u * kGridThreads;
          if (i < cnt) {
            int s0, s1;
            grid_slots(rc[u].cell - base, ng, TL, m, s0, s1);
            if (s0 >= 0) atomicAdd(&start[s0 / CW], 1);
            if (s1 >= 0) atomicAdd(&start[s1 / CW], 1);
          }
        }
        __syncthreads();
        // exclusive scan of start[0..NG]: group g occupies [start[g], start[g+1])
        {
          const int per = (NG + 1 + kGridThreads - 1) / kGridThreads;
          const int b0 = min((int)threadIdx.x * per, NG + 1), b1 = min(b0 + per, NG + 1);
          int sum = 0;
          for (int i = b0; i < b1; ++i) sum += start[i];
          const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
          int v = sum;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
          }
          if (lane == 31) wsum[w] = v;
          __syncthreads();
          if (w == 0) {
            int t = lane < kGridThreads / 32 ? wsum[lane] : 0;
#pragma unroll
            for (int o = 1; o < kGridThreads / 32; o <<= 1) {
              const int u2 = __shfl_up_sync(0xffffffffu, t, o);
              if (lane >= o) t += u2;
            }
            if (lane < kGridThreads / 32) wsum[lane] = t;
          }
          __syncthreads();
          int run = v - sum + (w > 0 ? wsum[w - 1] : 0);
          for (int i = b0; i < b1; ++i) {
            const int c = start[i];
            start[i] = run;
            run += c;
          }
        }
        __syncthreads();
        // place: afterwards start[g] is the END of group g
#pragma unroll
        for (int u = 0; u < RPT; ++u) {
          const int i = threadIdx.x + u * kGridThreads;
          if (i >= cnt) continue;
          int sl[2];
          grid_slots(rc[u].cell - base, ng, TL, m, sl[0], sl[1]);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int lc = sl[q];
            if (lc < 0) continue;
            const int pos = atomicAdd(&start[lc / CW], 1);
            SRec<T> r;
            r.f = rc[u].a;
            r.y = rc[u].b;
            r.lc = lc;
            r.pad = __float_as_int((float)lc);  // the slot as a float (exact), for the unmasked gather
            srec[pos] = r;
            sp[pos] = rc[u].p;
          }
        }
        __syncthreads();
      }
      if (SG == 1 && wts) {  // this slab's values for the placed records
        const int placed = start[(W - 1) / CW];
        const T *ws = wts + (int64_t)slab * nvals;
        for (int i = threadIdx.x; i < placed; i += kGridThreads) srec[i].y = ws[sp[i]];
        __syncthreads();
      }
      const T *yb = yv;
      if constexpr (SG > 1) {
        // the group's values (0 past the last slab): asynchronous copies, the
        // next group's while this one's are gathered where the records stay
        const int placed = start[(W - 1) / CW];
        auto fetch = [&](int first, T *dst) {
#pragma unroll
          for (int g = 0; g < SG; ++g) {
            const bool in = first + g < send;
            const T *ws = wts + (int64_t)(in ? first + g : sbeg) * nvals;
            for (int i = threadIdx.x; i < placed; i += kGridThreads) cp_async4(dst + g * CAP + i, ws + sp[i], in);
          }
        };
        if (nchunks > 1) {
          fetch(slab, yv);
          cp_async_wait();
          __syncthreads();
        } else {
          const int odd = ((slab - sbeg) / SG) & 1;
          if (slab == sbeg) fetch(slab, yv);
          cp_async_wait();
          __syncthreads();  // and the last group's gather is done with the other buffer
          yb = yv + odd * SG * CAP;
          if (slab + SG < send) fetch(slab + SG, yv + (1 - odd) * SG * CAP);
        }
      }
      // gather: the thread's cells cl0 .. cl0+CW-1 (local) take the records in
      // slots cl0 .. cl0 + CW - 1 + 2m - 1; record slot lc reaches cell c iff
      // 0 <= lc - c < 2m
#pragma unroll
      for (int q = 0; q < MAXC / CW; ++q) {
        const int cl0 = (threadIdx.x + q * kGridThreads) * CW;
        if (q >= npass || cl0 >= TL) continue;
        // the groups holding slots cl0 .. cl0 + CW + 2m - 2 (cl0 is a
        // multiple of CW; the last group may hold up to CW - 1 slots beyond
        // the window, whose records the masks drop or, unmasked, add below
        // 2^(-k1 m^2))
        const int g0 = cl0 / CW, g1 = (cl0 + CW + 2 * m - 2) / CW;
        const int rb = g0 == 0 ? 0 : start[g0 - 1];
        const int re = start[g1];
        // SG > 1 has one pass (CW = MAXC = 8) and accumulates into acc directly
        T a[1][CW];
#pragma unroll
        for (int i = 0; i < CW; ++i) a[0][i] = (T)0;
        const int ctr = cl0 + m, w2 = 2 * m;
        const float ctrf = (float)ctr;
        for (int r = rb; r < re; ++r) {
          const SRec<T> rr = srec[r];
          const int rel = rr.lc - cl0;  // lc - c for c = cl0
          // d - f for c = cl0; unmasked float tiles take the slot as a float
          // (a difference of small integers, exact) and skip the conversion
          T dd0;
          if constexpr (!MASKED && sizeof(T) == 4) dd0 = (ctrf - __int_as_float(rr.pad)) - rr.f;
          else dd0 = (T)(ctr - rr.lc) - rr.f;
          if constexpr (SG == 1) {
            gauss_acc<T, CW, MASKED>(rr.y, dd0, e.k1, gw, rel, w2, a[0]);
          } else {
            T w[CW];
            gauss_cw<T, CW>((T)1, dd0, e.k1, gw, w);
            if constexpr (MASKED) {
#pragma unroll
              for (int i = 0; i < CW; ++i) w[i] = (unsigned)(rel - i) < (unsigned)w2 ? w[i] : (T)0;
            }
#pragma unroll
            for (int g = 0; g < SG; ++g) {
              const T yg = yb[g * CAP + r];
#pragma unroll
              for (int i = 0; i < CW; ++i) acc[g][i] = fma(yg, w[i], acc[g][i]);
            }
          }
        }
        if constexpr (SG == 1) {
#pragma unroll
          for (int i = 0; i < CW; ++i) acc[0][CW * q + i] += a[0][i];
        }
      }
      if (SG == 1 || nchunks > 1) __syncthreads();
    }
#pragma unroll
    for (int g = 0; g < SG; ++g) {
      if (slab + g >= send) break;
      T *out = grid + (int64_t)(slab + g) * slab_stride + base;
#pragma unroll
      for (int q = 0; q < MAXC / CW; ++q) {
        const int cl0 = (threadIdx.x + q * kGridThreads) * CW;
        // TL is a power of two >= CW (gather tiles have >= 512 cells or span
        // the grid, ng >= 4m >= 4 and CW = 4 there), so groups are whole
        if (q < npass && cl0 < TL) {
          if constexpr (CW == 8 && sizeof(T) == 4) store8(out + cl0, acc[g]);
          else
#pragma unroll
            for (int i = 0; i < CW; i += 4)
              store4(out + cl0 + i, acc[g][CW * q + i], acc[g][CW * q + i + 1], acc[g][CW * q + i + 2],
                     acc[g][CW * q + i + 3]);
        }
      }
    }
  }
}

// slab groups sharing each record's Gaussian (bootstrap resamples, channels)
template <typename T, bool MASKED = true>
__global__ void __launch_bounds__(kGridThreads, sizeof(T) == 4 ? 3 : 2) k_grid_acc_sg4(
    const typename RecOf<T>::type *recs, const int *off, T *grid, AccParams<T> e, const T *wts, int64_t nvals,
    int nslab, int group, int64_t slab_stride) {
  pdl_trigger();
  pdl_wait();  // records and offsets come from the binning
  const int tile = blockIdx.x;
  const int sbeg = blockIdx.y * group, send = min(nslab, sbeg + group);
  const CgSrc<typename RecOf<T>::type> rp{recs};
  const int r0 = __ldcg(off + tile), r1 = __ldcg(off + tile + 1);
  if constexpr (sizeof(T) == 4)
    grid_tile_body<T, 8, CgSrc<typename RecOf<T>::type>, 4, MASKED>(rp, r0, r1, tile << e.logTL, grid, e, wts, nvals,
                                                                     sbeg, send, slab_stride);
  else  // double plans keep one slab per pass (four accumulator sets do not fit)
    grid_tile_body<T, 8>(rp, r0, r1, tile << e.logTL, grid, e, wts, nvals, sbeg, send, slab_stride);
}

template <typename T, int CW, bool MASKED = true>
__global__ void __launch_bounds__(kGridThreads, sizeof(T) == 4 ? 4 : 2) k_grid_acc(
    const typename RecOf<T>::type *recs, const int *off, T *grid, AccParams<T> e, const T *wts, int64_t nvals,
    int nslab, int group, int64_t slab_stride) {
  pdl_trigger();
  pdl_wait();  // records and offsets come from the binning
  // a CTA per (tile, group of slabs)
  const int tile = blockIdx.x;
  const int sbeg = blockIdx.y * group, send = min(nslab, sbeg + group);
  const CgSrc<typename RecOf<T>::type> rp{recs};
  grid_tile_body<T, CW, CgSrc<typename RecOf<T>::type>, 1, MASKED>(rp, __ldcg(off + tile), __ldcg(off + tile + 1),
                                                                    tile << e.logTL, grid, e, wts, nvals, sbeg, send,
                                                                    slab_stride);
}

// Whether a float plan's gather may add each record to whole cell groups
// without the tap masks: every cell beyond a record's taps lies more than m
// cells from it, where the Gaussian exp(-d^2 / (4 tau)) is below
// exp(-m^2 / (4 tau)); below 1e-8 of the peak (under float rounding) the
// extra terms only bring the kernel closer to the untruncated Gaussian that
// the deconvolution divides by.  Double plans keep the masks.
inline bool tail_free_gather(bool is_float, int m, double tau) {
  return is_float && (double)m * m / (4.0 * tau) >= 18.43;  // exp(-18.43) = 1e-8
}

// Scatter form of the same tile gridding: the tile's cells accumulate in
// shared memory, one thread per (record, tap) pair adds its Gaussian weight
// with a shared-memory atomic, and the tile is flushed to HBM once, in cell
// order, with vector stores (no global atomics).  A block step covers
// floor(256 / 2m) records, thread t taking tap t mod 2m of record t / 2m, so
// every lane of a warp does useful work whatever the record density.  A tap
// lands in cell (cell + d) mod ng, kept when it falls in this tile; ng is a
// power of two.  Summation order within a cell follows the atomics.
template <typename T, class Src>
__device__ __forceinline__ void grid_tile_scatter(const Src &recs, int r0, int r1,
                                                  int base, T *__restrict__ grid, const AccParams<T> &e,
                                                  const T *__restrict__ wts, int64_t nvals, int sbeg, int send,
                                                  int64_t slab_stride) {
  typedef typename RecOf<T>::type Rec;
  constexpr int CAP = GridCfg<T>::CAP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int TL = 1 << e.logTL, m = e.m, W2 = 2 * m;
  const int gmask = (int)e.ng - 1;
  T *acc = reinterpret_cast<T *>(smem_raw);                          // TL cells
  SRec<T> *srec = reinterpret_cast<SRec<T> *>(smem_raw + sizeof(T) * TL);  // CAP staged records
  int *sp = reinterpret_cast<int *>(srec + CAP);                       // sample index (weights)
  const int per = kGridThreads / W2;  // records per block step (W2 <= 32)
  const int rr = threadIdx.x / W2;
  const int d = (int)threadIdx.x - rr * W2 - m + 1;  // tap offset in [-m+1, m]
  const T dT = (T)d;
  const bool active = rr < per;
  const int nchunks = (r1 - r0 + CAP - 1) / CAP;
  for (int slab = sbeg; slab < send; ++slab) {
    for (int i = 4 * threadIdx.x; i < TL; i += 4 * kGridThreads) store4(acc + i, (T)0, (T)0, (T)0, (T)0);
    for (int ck = 0; ck < nchunks; ++ck) {
      const int c0 = r0 + ck * CAP;
      const int cnt = min(CAP, r1 - c0);
      if (nchunks > 1 || slab == sbeg) {
        for (int i = threadIdx.x; i < cnt; i += kGridThreads) {
          const Rec rc = recs[c0 + i];
          SRec<T> r;
          r.f = rc.a;
          r.y = rc.b;
          r.lc = rc.cell - base;
          r.pad = 0;
          srec[i] = r;
          sp[i] = rc.p;
        }
      }
      if (wts) {
        __syncthreads();
        const T *ws = wts + (int64_t)slab * nvals;
        for (int i = threadIdx.x; i < cnt; i += kGridThreads) srec[i].y = ws[sp[i]];
      }
      __syncthreads();
      if (active) {
        for (int r = rr; r < cnt; r += per) {
          const SRec<T> q = srec[r];
          const int lc = (q.lc + d) & gmask;
          const T w = gauss_w(q.y, dT - q.f, e.k1);
          if (lc < TL) atomicAdd(&acc[lc], w);
        }
      }
      __syncthreads();
    }
    // fixed-order flush; TL is a power of two >= 4, so groups of four are whole
    T *out = grid + (int64_t)slab * slab_stride + base;
    for (int i = 4 * threadIdx.x; i < TL; i += 4 * kGridThreads) store4(out + i, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(kGridThreads, sizeof(T) == 4 ? 6 : 3) k_grid_scatter(
    const typename RecOf<T>::type *recs, const int *off, T *grid, AccParams<T> e, const T *wts, int64_t nvals,
    int nslab, int group, int64_t slab_stride) {
  pdl_trigger();
  pdl_wait();  // records and offsets come from the binning
  const int tile = blockIdx.x;
  const int sbeg = blockIdx.y * group, send = min(nslab, sbeg + group);
  const CgSrc<typename RecOf<T>::type> rp{recs};
  grid_tile_scatter<T>(rp, __ldcg(off + tile), __ldcg(off + tile + 1), tile << e.logTL, grid, e, wts, nvals, sbeg,
                       send, slab_stride);
}

// Fixed-point form: one thread per record, all 2m taps from the fast Gaussian
// factorisation  y exp2(-k1 (d - f)^2) = [y exp2(-k1 f^2)] Q^d exp2(-k1 d^2),
// Q = exp2(2 k1 f)  (three exp2 per record, two multiplies per tap), each
// tap added into the shared tile as an integer with a native shared-memory
// integer atomic.  The tile's fixed-point scale comes from a bound on every
// cell's sum: |y| <= Ymax over the tile's records and at most 2 hmax records
// reach one cell, hmax the largest count of records in a bucket of
// max(2m, 16) consecutive cells (a cell's 2m-cell window meets two buckets);
// weights are <= 1.  With the sum bounded by 2^30 (float, int32 cells) or
// 2^50 (double, int64 cells, as two 32-bit words where hmax <= 2048) units,
// the quantum is 2^-30 (2^-50) of the
// bound.  Integer sums do not depend on the order of the atomics, so the grid
// is bit-reproducible run to run.  A non-finite value makes its tiles NaN.
// records [c0, c0 + cnt) -> srec (values from ws when given); returns the
// thread's max |value| (NaN once one is not finite)
// max(ym, |v|), NaN once a value was not finite (double: |v| to 2^-23 below,
// without the conversions of the FP64 pipe; the tile's range has room for it)
__device__ __forceinline__ float value_bound(float ym, float v) {
  return isfinite(v) && !isnan(ym) ? fmaxf(ym, fabsf(v)) : __int_as_float(0x7fffffff);
}
__device__ __forceinline__ float value_bound(float ym, double v) {
  const bool finite = (__double2hiint(v) & 0x7ff00000) != 0x7ff00000;
  return finite && !isnan(ym) ? fmaxf(ym, fabsf(df_from_double(v).hi)) : __int_as_float(0x7fffffff);
}
template <typename T, int NT> __host__ __device__ constexpr int fixed_cap() { return GridCfg<T>::CAP > NT ? GridCfg<T>::CAP : NT; }
template <typename T, int NT, class Src>
__device__ __forceinline__ float fixed_stage(const Src &recs, int c0, int cnt,
                                            int base, const T *__restrict__ ws, SRec<T> *srec) {
  float ym = 0.f;
#pragma unroll 1
  for (int i = threadIdx.x; i < cnt; i += NT) {
    const typename RecOf<T>::type rc = recs[c0 + i];
    SRec<T> r;
    r.f = rc.a;
    r.y = ws ? ws[rc.p] : rc.b;
    r.lc = rc.cell - base;
    r.pad = rc.p;
    srec[i] = r;
    ym = value_bound(ym, r.y);
  }
  return ym;
}

// clear a fixed-point tile of TL cells (TL a multiple of 4, acc 16-byte
// aligned) with 16-byte stores
template <int NT, typename A> __device__ __forceinline__ void fixed_clear(A *acc, int TL) {
  int4 *v = reinterpret_cast<int4 *>(acc);
  const int nv = TL * (int)sizeof(A) / 16;
  for (int i = threadIdx.x; i < nv; i += NT) v[i] = make_int4(0, 0, 0, 0);
}
// cells [i, i + 4) of a fixed-point tile as values: 16-byte shared loads
__device__ __forceinline__ void fixed_load4(const int *acc, int i, float inv, float &a, float &b, float &c,
                                            float &d) {
  const int4 v = *reinterpret_cast<const int4 *>(acc + i);
  a = (float)v.x * inv;
  b = (float)v.y * inv;
  c = (float)v.z * inv;
  d = (float)v.w * inv;
}
__device__ __forceinline__ void fixed_load4(const long long *acc, int i, double inv, double &a, double &b,
                                            double &c, double &d) {
  const longlong2 u = *reinterpret_cast<const longlong2 *>(acc + i);
  const longlong2 v = *reinterpret_cast<const longlong2 *>(acc + i + 2);
  a = (double)u.x * inv;
  b = (double)u.y * inv;
  c = (double)v.x * inv;
  d = (double)v.y * inv;
}

// Double tiles in split form: each int64 tap v enters two 32-bit integer
// atomics instead of one 64-bit one (slower in shared memory: 212 against
// 179 us for a 2^22-cell float64 grid of 1e6 samples): hi[c] +=
// floor(v / 2^20) (signed) and lo[c] += v mod 2^20
// (unsigned), arrays of TL words each in the space of the int64 tile.  The
// cell's sum is hi * 2^20 + lo exactly when neither array overflows: a cell
// takes at most 2 hmax taps, so lo stays below 2 hmax 2^20 <= 2^32 for hmax
// <= 2048, and |hi| below 2^30 + 4 hmax (each |v| <= 2^50 / (2 hmax) + 1).
// The integer sums, hence the grid's bits, equal the int64 form's.
constexpr int kSplitBits = 20;
constexpr int kSplitMaxH = 2048;
struct SplitAdd {
  int *hi;
  unsigned *lo;
  // the integer h 2^20 + l
  __device__ __forceinline__ void operator()(int c, int h, int l) const {
    atomicAdd(lo + c, (unsigned)l & ((1u << kSplitBits) - 1u));
    atomicAdd(hi + c, h + (l >> kSplitBits));
  }
};
struct WideAdd {  // one 64-bit atomic
  long long *acc;
  __device__ __forceinline__ void operator()(int c, int h, int l) const {
    FixAcc<double>::add(acc + c, ((long long)h << kSplitBits) + l);
  }
};
// cells [i, i + 4) of a split tile as values: 16-byte shared loads
__device__ __forceinline__ void fixed_load4_split(const int *hi, const unsigned *lo, int i, double inv, double &a,
                                                  double &b, double &c, double &d) {
  const int4 h = *reinterpret_cast<const int4 *>(hi + i);
  const uint4 l = *reinterpret_cast<const uint4 *>(lo + i);
  constexpr long long U = 1ll << kSplitBits;
  a = (double)((long long)h.x * U + l.x) * inv;
  b = (double)((long long)h.y * U + l.y) * inv;
  c = (double)((long long)h.z * U + l.z) * inv;
  d = (double)((long long)h.w * U + l.w) * inv;
}

// A double plan's coefficients exp2(-k1 d^2), d = 0..m, in shared memory: the
// float-float value with each half twice (hi, hi, lo, lo), the packed operand.
constexpr int kTapCoefBytes = 17 * 16 > 32 * 4 ? 17 * 16 : 32 * 4;

// All 2m taps of a record into the tile as integers scaled by sc.  Float: the
// taps d = k and d = -k share the coefficient exp2(-k1 k^2) (c[k - 1], k =
// 1..m, read four at a time); a product, a conversion and an atomic per tap.
__device__ __forceinline__ void fixed_taps(float y, float f, int p0, float sc, const AccParams<float> &e,
                                           const float *c, int *acc, int TL, int gmask) {
  const int m = e.m;
  const float E = y * sc * exp2_g(-e.k1 * f * f);
  const float Q = exp2_g(e.k2 * f), Qi = exp2_g(-e.k2 * f);
  float u = E, v = E;
  if (p0 - m + 1 >= 0 && p0 + m < TL) {  // every tap inside the tile
    int *p = acc + p0;
    FixAcc<float>::add(p, FixAcc<float>::to_fix(E));
    auto pair = [&](int k, float ck) {
      u *= Q;
      v *= Qi;
      FixAcc<float>::add(p + k, FixAcc<float>::to_fix(u * ck));
      FixAcc<float>::add(p - k, FixAcc<float>::to_fix(v * ck));
    };
    int k = 1;
#pragma unroll 1
    for (; k + 4 <= m; k += 4) {
      const float4 ck = *reinterpret_cast<const float4 *>(c + k - 1);
      pair(k, ck.x);
      pair(k + 1, ck.y);
      pair(k + 2, ck.z);
      pair(k + 3, ck.w);
    }
#pragma unroll 1
    for (; k < m; ++k) pair(k, c[k - 1]);
    FixAcc<float>::add(p + m, FixAcc<float>::to_fix(u * Q * c[m - 1]));
  } else {  // near the tile edge: wrap, keep the taps inside the tile
    auto tap = [&](int lc, float w) {
      lc &= gmask;
      if (lc < TL) FixAcc<float>::add(acc + lc, FixAcc<float>::to_fix(w));
    };
    tap(p0, E);
#pragma unroll 1
    for (int k = 1; k <= m; ++k) {
      const float ck = c[k - 1];
      u *= Q;
      v *= Qi;
      tap(p0 + k, u * ck);
      if (k < m) tap(p0 - k, v * ck);
    }
  }
}

// a tap p + e (|p| <= 2^50, e its rounding remainder) as the integer nearest it,
// h 2^20 + l: h from p alone (exact: p has 24 bits, so either p / 2^20 is an
// integer or its nearest integer is below 2^24), l from what is left
__device__ __forceinline__ void tap_fix(float p, float e, int &h, int &l) {
  h = __float2int_rn(p * 0x1p-20f);
  l = __float2int_rn(fmaf((float)h, -0x1p20f, p) + e);
}

struct TapConst {  // the exponent constants in float-float
  dfl k1, k2;
  __device__ explicit TapConst(const AccParams<double> &e) : k1(df_from_double(e.k1)), k2(df_from_double(e.k2)) {}
};
// Double: the taps d = k and d = -k of a record as one packed pair in
// float-float (about 48 bits, below the 2^-50 quantum's reach only where a tap
// is far below its tile's bound), E Q^k and E Q^-k by running products with the
// shared coefficient c_k; only the two conversions from double use the FP64
// pipe.  13 packed operations per pair of taps and 9 scalar ones per tap to
// split it into the two words, where scalar products and a 64-bit integer took
// 60 per tap (1e6 samples on 2^22 cells: 120 -> 80 us, flushing float-float
// cells included; 71 with unstaged records and the scale's divisions by one
// warp).
template <class Add>
__device__ __forceinline__ void fixed_taps_df(double y, double f, int p0, double sc, const TapConst &tc, int m,
                                              const ulonglong2 *cw, const Add &add, int TL, int gmask) {
  const f2 m1 = pk2(-1.0f, -1.0f);
  const dfl fw = df_from_double(f);
  // E = y sc 2^(-k1 f^2), Q = 2^(k2 f), 1/Q
  const dfl E = df_from_double(y * sc) * df_exp2(-(tc.k1 * fw * fw));
  const dfl Q = df_exp2(tc.k2 * fw), Qi = df_rcp(Q);
  const f2 Qh = pk2(Q.hi, Qi.hi), Ql = pk2(Q.lo, Qi.lo), nQh = mul2(Qh, m1);
  f2 Uh = pk2(E.hi, E.hi), Ul = pk2(E.lo, E.lo);
  auto taps = [&](auto tap) {
    tap(p0, E.hi, E.lo);
#pragma unroll 2
    for (int k = 1; k <= m; ++k) {
      {  // U <- U Q: float-float product, renormalised
        const f2 p = mul2(Uh, Qh), w = fma2(Uh, nQh, p);
        const f2 r = sub2(fma2(Ul, Qh, mul2(Uh, Ql)), w);
        Uh = add2(p, r);
        Ul = sub2(r, sub2(Uh, p));
      }
      const ulonglong2 c = cw[k];
      const f2 p = mul2(Uh, c.x);
      const f2 r = fma2(Ul, c.x, fma2(Uh, c.y, fma2(Uh, c.x, mul2(p, m1))));
      float ph, pl, rh, rl;
      unpk2(p, ph, pl);
      unpk2(r, rh, rl);
      tap(p0 + k, ph, rh);
      if (k < m) tap(p0 - k, pl, rl);
    }
  };
  if (p0 - m + 1 >= 0 && p0 + m < TL) {  // every tap inside the tile
    taps([&](int c, float p, float r) {
      int h, l;
      tap_fix(p, r, h, l);
      add(c, h, l);
    });
  } else {  // near the tile edge: wrap, keep the taps inside the tile
    taps([&](int c, float p, float r) {
      c &= gmask;
      if (c < TL) {
        int h, l;
        tap_fix(p, r, h, l);
        add(c, h, l);
      }
    });
  }
}

// the tile's fixed-point scale from the per-warp maxima of |value| (NaN once
// one was not finite) and the largest bucket count hmax
template <typename T, int NT>
__device__ __forceinline__ T fixed_scale(const float *red, int hmax) {
  float y = 0.f;
  bool bad = false;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    bad |= isnan(red[w]);
    y = fmaxf(y, red[w]);
  }
  // bound on any cell's |sum| in value units; the scale maps it to `range`
  const T B = (T)y * (T)(2 * hmax);
  T sc = B > (T)0 ? FixAcc<T>::range / B : (T)0;
  if (isinf(sc)) sc = (T)0;
  return bad ? (T)NAN : sc;
}

// the taps of srec[0, cnt) into the tile, in split form when asked (double)
template <typename T, int NT>
__device__ __forceinline__ void tile_taps(bool split, const SRec<T> *srec, int cnt, T sc, const AccParams<T> &e,
                                          const void *cd, typename FixAcc<T>::type *acc, int TL, int gmask) {
  if constexpr (sizeof(T) == 8) {
    const ulonglong2 *cw = static_cast<const ulonglong2 *>(cd);
    const TapConst tc(e);
    const SplitAdd sa{reinterpret_cast<int *>(acc), reinterpret_cast<unsigned *>(acc) + TL};
#pragma unroll 1
    for (int i = threadIdx.x; i < cnt; i += NT) {
      const SRec<double> q = srec[i];
      if (split) fixed_taps_df(q.y, q.f, q.lc, sc, tc, e.m, cw, sa, TL, gmask);
      else fixed_taps_df(q.y, q.f, q.lc, sc, tc, e.m, cw, WideAdd{acc}, TL, gmask);
    }
  } else {
#pragma unroll 1
    for (int i = threadIdx.x; i < cnt; i += NT)
      fixed_taps(srec[i].y, srec[i].f, srec[i].lc, sc, e, static_cast<const float *>(cd), acc, TL, gmask);
  }
}

// The flush's factor inv = 1 / scale as f 2^-50 p: 2^50 inv, the tile's bound, is
// near the values themselves, where inv alone is 2^-50 of them and would leave
// the float range long before they do.  p is a power of two, f a float-float in
// [1, 2) (outside only where the bound is beyond the float range; 0 for an empty
// tile, NaN for a non-finite value), so products with f lose nothing to
// underflow and those with p round only where a cell leaves the float range.
// (inv itself as a float-float: 9e-6 relative at values of 1e-26, all zero at
// 1e-31.  One warp forms it for the CTA: 1e6 samples on 2^22 cells, the whole
// transform 189.0 us as one float-float per thread, 188.2 here.)
struct FlushScale {
  dfl f;
  float p;
  FlushScale() = default;
  __device__ explicit FlushScale(double inv) {
    const int e = ((__double2hiint(inv) >> 20) & 0x7ff) - 1023 + 50, pe = min(max(e, -126), 127);
    f = dfl(inv * __hiloint2double((1023 + 50 - pe) << 20, 0));
    p = __int_as_float((127 + pe) << 23);
  }
};
// Two cells h 2^20 + l (l < 2^32) times inv as one float-float complex value:
// each integer, in units of 2^50, as three exact floats (h rounded to 24 bits;
// the remainder with l's high half; l's low half) added up, the product
// renormalised.
__device__ __forceinline__ dcx fixed_pair_df(int h0, unsigned l0, int h1, unsigned l1, const FlushScale &inv) {
  const float f0 = (float)h0, f1 = (float)h1;
  const int r0 = h0 - (int)f0, r1 = h1 - (int)f1;  // |r| <= 64
  const f2 a = mul2(pk2(f0, f1), pk2(0x1p-30f, 0x1p-30f));
  const f2 b = mul2(pk2((float)(r0 * 16 + (int)(l0 >> 16)), (float)(r1 * 16 + (int)(l1 >> 16))), pk2(0x1p-34f, 0x1p-34f));
  const f2 c = mul2(pk2((float)(l0 & 0xffffu), (float)(l1 & 0xffffu)), pk2(0x1p-50f, 0x1p-50f));
  const f2 s = add2(a, b), v = sub2(s, a);
  const f2 e = add2(add2(sub2(a, sub2(s, v)), sub2(b, v)), c);
  const f2 xh = add2(s, e), xl = sub2(e, sub2(xh, s));
  const f2 ih = pk2(inv.f.hi, inv.f.hi), p = mul2(xh, ih);
  const f2 r = sub2(fma2(xl, ih, mul2(xh, pk2(inv.f.lo, inv.f.lo))), fma2(xh, pk2(-inv.f.hi, -inv.f.hi), p));
  const f2 oh = add2(p, r), ol = sub2(r, sub2(oh, p)), pw = pk2(inv.p, inv.p);
  dcx o;
  o.h = mul2(oh, pw);
  o.l = mul2(ol, pw);
  return o;
}

// the tile into the grid as float-float (pairs of cells are the complex points
// of the FFT), for the float-float passes: integer and FP32 operations only,
// where the double cells cost two FP64-pipe operations each here and as many
// conversions in the column pass
template <int NT>
__device__ __forceinline__ void tile_flush_df(bool split, const long long *acc, int TL, const FlushScale &iv, double *out) {
  ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out);
  const int *hi = reinterpret_cast<const int *>(acc);
  const unsigned *lo = reinterpret_cast<const unsigned *>(acc) + TL;
  for (int i = 2 * threadIdx.x; i < TL; i += 2 * NT) {
    int2 h;
    uint2 l;
    if (split) {
      h = *reinterpret_cast<const int2 *>(hi + i);
      l = *reinterpret_cast<const uint2 *>(lo + i);
    } else {
      const longlong2 v = *reinterpret_cast<const longlong2 *>(acc + i);
      h = make_int2((int)(v.x >> kSplitBits), (int)(v.y >> kSplitBits));
      l = make_uint2((unsigned)v.x & ((1u << kSplitBits) - 1u), (unsigned)v.y & ((1u << kSplitBits) - 1u));
    }
    const dcx w = fixed_pair_df(h.x, l.x, h.y, l.y, iv);
    o[i >> 1] = make_ulonglong2(w.h, w.l);
  }
}

// fixed-order flush of the tile: out[i] = cell i * inv (inv = 1 / scale)
template <typename T, int NT>
__device__ __forceinline__ void tile_flush(bool split, const typename FixAcc<T>::type *acc, int TL, T inv, T *out) {
  if constexpr (sizeof(T) == 8) {
    if (split) {
      const int *hi = reinterpret_cast<const int *>(acc);
      const unsigned *lo = reinterpret_cast<const unsigned *>(acc) + TL;
      for (int i = 4 * threadIdx.x; i < TL; i += 4 * NT) {
        T a, b, c, d;
        fixed_load4_split(hi, lo, i, inv, a, b, c, d);
        store4(out + i, a, b, c, d);
      }
      return;
    }
  }
  for (int i = 4 * threadIdx.x; i < TL; i += 4 * NT) {
    T a, b, c, d;
    fixed_load4(acc, i, inv, a, b, c, d);
    store4(out + i, a, b, c, d);
  }
}

template <typename T> struct SegSrc;  // a tile's records as runs, below

// NT threads; dfout (double): cells written in float-float
template <typename T, class Src, int NT = kGridThreads>
__device__ __forceinline__ void grid_tile_fixed(const Src &recs, int r0, int r1,
                                                int base, T *__restrict__ grid, const AccParams<T> &e,
                                                const T *__restrict__ wts, int64_t nvals, int sbeg, int send,
                                                int64_t slab_stride, bool dfout = false) {
  typedef FixAcc<T> FA;
  typedef typename FA::type A;
  constexpr int CAP = fixed_cap<T, NT>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[NT / 32];
  __shared__ int redi[NT / 32];
  __shared__ T scale_s;
  __shared__ FlushScale flush_s;
  const int TL = 1 << e.logTL, m = e.m;
  const int gmask = (int)e.ng - 1;
  int logBS = 4;
  while ((1 << logBS) < 2 * m) ++logBS;
  const int NB = ((TL + 2 * m) >> logBS) + 1;
  A *acc = reinterpret_cast<A *>(smem_raw);                                  // TL cells
  SRec<T> *srec = reinterpret_cast<SRec<T> *>(smem_raw + sizeof(A) * TL);    // CAP staged records
  // coefficients exp2(-k1 d^2): float d = 1..m; double d = 0..m, packed float-float
  // (tiles of one slab of the records' own values stage none)
  constexpr bool kOwn = !std::is_same<Src, SegSrc<T>>::value;
  const bool own = kOwn && !wts && sbeg + 1 == send;
  void *cd = own ? srec : srec + CAP;
  int *hist = reinterpret_cast<int *>(static_cast<char *>(cd) + kTapCoefBytes);  // NB buckets
  const int nchunks = (r1 - r0 + CAP - 1) / CAP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if constexpr (sizeof(T) == 8) {
    for (int d = threadIdx.x; d <= m; d += NT) {
      const dfl c = df_from_double(exp2_g(-e.k1 * (T)(d * d)));
      static_cast<ulonglong2 *>(cd)[d] = make_ulonglong2(pk2(c.hi, c.hi), pk2(c.lo, c.lo));
    }
  } else {
    for (int d = threadIdx.x; d < m; d += NT) static_cast<T *>(cd)[d] = exp2_g(-e.k1 * (T)((d + 1) * (d + 1)));
  }
  // bucket histogram of the tile's records (slab independent); a record of
  // this tile lies in [base - m, base + TL + m) modulo ng
  for (int b = threadIdx.x; b < NB; b += NT) hist[b] = 0;
  if constexpr (kOwn) {
    if (own) {
      // One slab of the records' own values: a first read of the records builds
      // the histogram and bounds |value|, a second one makes the taps, from
      // registers for a thread's first KEEP records, else from the L2.  No
      // staging (bound by the shared-memory pipe, of which the staging and a
      // coefficient read per tap were a quarter: 64 series of 2e5 samples, m =
      // 10: 224 -> 166 us; 5.4e8 cells, 5.8e7 samples, m = 8: 1107 -> 1044 us).
      typedef typename RecOf<T>::type Rec;
      constexpr int KEEP = 2;
      const int cnt = r1 - r0;
      fixed_clear<NT>(acc, TL);
      __syncthreads();
      float ym = 0.f;
      int hm = 0;
      // few records: the largest bucket count is the largest count an atomic
      // returned; many: the buckets are read back (an atomic that returns
      // nothing is cheaper where a warp's samples share a bucket)
      const bool few = cnt <= 4 * NT;
      auto see = [&](const Rec &r) {
        int *h = &hist[((r.cell - base + m) & gmask) >> logBS];
        if (few) hm = max(hm, atomicAdd(h, 1) + 1);
        else atomicAdd(h, 1);
        ym = value_bound(ym, r.b);
      };
      Rec rc[KEEP], nx[KEEP];
#pragma unroll
      for (int k = 0; k < KEEP; ++k)
        if (threadIdx.x + k * NT < cnt) rc[k] = recs[r0 + threadIdx.x + k * NT];
#pragma unroll
      for (int k = 0; k < KEEP; ++k)
        if (threadIdx.x + k * NT < cnt) see(rc[k]);
#pragma unroll 1
      for (int i = threadIdx.x + KEEP * NT; i < cnt; i += KEEP * NT) {
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
          if (i + k * NT < cnt) nx[k] = recs[r0 + i + k * NT];
#pragma unroll
        for (int k = 0; k < KEEP; ++k)
          if (i + k * NT < cnt) see(nx[k]);
      }
      if (!few) {
        __syncthreads();
        for (int b = threadIdx.x; b < NB; b += NT) hm = max(hm, hist[b]);
      }
      for (int o = 16; o > 0; o >>= 1) {
        const float u = __shfl_xor_sync(0xffffffffu, ym, o);
        ym = (isnan(u) || isnan(ym)) ? __int_as_float(0x7fffffff) : fmaxf(ym, u);
        hm = max(hm, __shfl_xor_sync(0xffffffffu, hm, o));
      }
      if (lane == 0) {
        red[warp] = ym;
        redi[warp] = hm;
      }
      __syncthreads();
      int hmax = 0;
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) hmax = max(hmax, redi[w]);
      T sc, inv;
      auto scale = [&] {
        sc = fixed_scale<T, NT>(red, hmax);
        inv = sc > (T)0 ? (T)1 / sc : (sc == sc ? (T)0 : sc);
      };
      if constexpr (sizeof(T) == 4) {
        scale();
      } else {  // two FP64 divisions, by one warp: all of them would fill the FP64 pipe
        __shared__ T scale_i;
        if (warp == 0) {
          scale();
          if (lane == 0) {
            scale_s = sc;
            scale_i = inv;
            if (dfout) flush_s = FlushScale(inv);
          }
        }
        __syncthreads();
        sc = scale_s;
        inv = scale_i;
      }
      const bool split = sizeof(T) == 8 && hmax <= kSplitMaxH;
      auto each = [&](auto taps) {
        Rec r = rc[0];
#pragma unroll 1
        for (int i = threadIdx.x; i < cnt; i += NT) {
          Rec n = rc[1];  // the next one, on its way
          if (i >= NT && i + NT < cnt) n = recs[r0 + i + NT];
          taps(r);
          r = n;
        }
      };
      if (sc > (T)0) {
        if constexpr (sizeof(T) == 4) {
          const float *c = static_cast<const float *>(cd);
          each([&](const Rec &r) { fixed_taps(r.b, r.a, r.cell - base, sc, e, c, acc, TL, gmask); });
        } else {
          const ulonglong2 *cw = static_cast<const ulonglong2 *>(cd);
          const TapConst tc(e);
          const SplitAdd sa{reinterpret_cast<int *>(acc), reinterpret_cast<unsigned *>(acc) + TL};
          if (split) each([&](const Rec &r) { fixed_taps_df(r.b, r.a, r.cell - base, sc, tc, m, cw, sa, TL, gmask); });
          else each([&](const Rec &r) { fixed_taps_df(r.b, r.a, r.cell - base, sc, tc, m, cw, WideAdd{acc}, TL, gmask); });
        }
      }
      __syncthreads();
      T *out = grid + (int64_t)sbeg * slab_stride + base;
      if constexpr (sizeof(T) == 8)
        if (dfout) {
          tile_flush_df<NT>(split, acc, TL, flush_s, out);
          return;
        }
      tile_flush<T, NT>(split, acc, TL, inv, out);
      return;
    }
  }
  if (!kOwn && !wts && sbeg + 1 == send && nchunks <= 1) {
    // One slab of the records' own values, one staging chunk: a single read
    // of the records stages them, builds the histogram and bounds |value|;
    // the largest bucket count is the largest count an atomic returned.
    // Three barriers per tile instead of six; same scale, same bits.
    constexpr int PER = CAP / NT;
    const int cnt = r1 - r0;
    fixed_clear<NT>(acc, TL);
    __syncthreads();
    typename RecOf<T>::type rc[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (threadIdx.x + k * NT < cnt) rc[k] = recs[r0 + threadIdx.x + k * NT];
    float ym = 0.f;
    int hm = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i >= cnt) continue;
      SRec<T> r;
      r.f = rc[k].a;
      r.y = rc[k].b;
      r.lc = rc[k].cell - base;
      r.pad = rc[k].p;
      srec[i] = r;
      hm = max(hm, atomicAdd(&hist[((rc[k].cell - base + m) & gmask) >> logBS], 1) + 1);
      ym = value_bound(ym, r.y);
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float u = __shfl_xor_sync(0xffffffffu, ym, o);
      ym = (isnan(u) || isnan(ym)) ? __int_as_float(0x7fffffff) : fmaxf(ym, u);
      hm = max(hm, __shfl_xor_sync(0xffffffffu, hm, o));
    }
    if (lane == 0) {
      red[warp] = ym;
      redi[warp] = hm;
    }
    __syncthreads();
    int hmax = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) hmax = max(hmax, redi[w]);
    const T sc = fixed_scale<T, NT>(red, hmax);
    const bool split = sizeof(T) == 8 && hmax <= kSplitMaxH;
    if (sc > (T)0) tile_taps<T, NT>(split, srec, cnt, sc, e, cd, acc, TL, gmask);
    __syncthreads();
    const T inv = sc > (T)0 ? (T)1 / sc : (sc == sc ? (T)0 : sc);
    tile_flush<T, NT>(split, acc, TL, inv, grid + (int64_t)sbeg * slab_stride + base);
    return;
  }
  __syncthreads();
#pragma unroll 1
  for (int i = r0 + threadIdx.x; i < r1; i += NT)
    atomicAdd(&hist[((recs[i].cell - base + m) & gmask) >> logBS], 1);
  __syncthreads();
  int hmax = 0;
  for (int b = threadIdx.x; b < NB; b += NT) hmax = max(hmax, hist[b]);
  for (int o = 16; o > 0; o >>= 1) hmax = max(hmax, __shfl_xor_sync(0xffffffffu, hmax, o));
  if (lane == 0) redi[warp] = hmax;
  __syncthreads();
  hmax = 0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) hmax = max(hmax, redi[w]);
  const bool split = sizeof(T) == 8 && hmax <= kSplitMaxH;
  for (int slab = sbeg; slab < send; ++slab) {
    const T *ws = wts ? wts + (int64_t)slab * nvals : nullptr;
    float ym = 0.f;
    if (slab > sbeg) __syncthreads();  // the previous slab's flush is done with acc and srec
    if (nchunks == 1) {
      ym = fixed_stage<T, NT>(recs, r0, r1 - r0, base, ws, srec);
    } else {  // bound pass over all of the tile's records
#pragma unroll 1
      for (int i = r0 + threadIdx.x; i < r1; i += NT) {
        const T v = ws ? ws[recs[i].p] : recs[i].b;
        ym = value_bound(ym, v);
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float u = __shfl_xor_sync(0xffffffffu, ym, o);
      ym = (isnan(u) || isnan(ym)) ? __int_as_float(0x7fffffff) : fmaxf(ym, u);
    }
    if (lane == 0) red[warp] = ym;
    fixed_clear<NT>(acc, TL);
    __syncthreads();
    if (threadIdx.x == 0) scale_s = fixed_scale<T, NT>(red, hmax);
    __syncthreads();
    const T sc = scale_s;
    for (int ck = 0; ck < nchunks; ++ck) {
      const int c0 = r0 + ck * CAP;
      const int cnt = min(CAP, r1 - c0);
      if (nchunks > 1) {
        if (ck > 0) __syncthreads();
        fixed_stage<T, NT>(recs, c0, cnt, base, ws, srec);
        __syncthreads();
      }
      if (sc > (T)0) tile_taps<T, NT>(split, srec, cnt, sc, e, cd, acc, TL, gmask);
    }
    __syncthreads();
    // fixed-order flush: cell = integer / scale
    const T inv = sc > (T)0 ? (T)1 / sc : (sc == sc ? (T)0 : sc);
    T *out = grid + (int64_t)slab * slab_stride + base;
    if constexpr (sizeof(T) == 8)
      if (dfout) {
        tile_flush_df<NT>(split, acc, TL, FlushScale(inv), out);
        continue;
      }
    tile_flush<T, NT>(split, acc, TL, inv, out);
  }
}

// NT = 256, or 1024 for double launches that do not give every SM two tiles
// (one transform of 2^19 cells is 128 tiles of 4096: 54 us with eight warps per
// SM and scalar taps, 23 us here).
// These do not let the column pass launch before they end: its CTAs would all
// start on the few SMs that have no tile, and how many do depends on the
// cycle (2e5 samples, Nf = 2^18, forward: 67 us with an early launch, 71 with
// the bound's exponent apart as above, 50 without).
template <typename T, int NT>
__global__ void __launch_bounds__(NT, NT > 256 ? 1 : (sizeof(T) == 4 ? 6 : 4)) k_grid_fixed(
    const typename RecOf<T>::type *recs, const int *off, T *grid, AccParams<T> e, const T *wts, int64_t nvals,
    int nslab, int group, int64_t slab_stride, bool dfout) {
  if (NT == kGridThreads) pdl_trigger();
  pdl_wait();  // records and offsets come from the binning
  const int tile = blockIdx.x;
  const int sbeg = blockIdx.y * group, send = min(nslab, sbeg + group);
  const CgSrc<typename RecOf<T>::type> rp{recs};
  grid_tile_fixed<T, CgSrc<typename RecOf<T>::type>, NT>(rp, __ldcg(off + tile), __ldcg(off + tile + 1), tile << e.logTL,
                                                         grid, e, wts, nvals, sbeg, send, slab_stride, dfout);
}

// own: tiles of one slab of the records' own values, which stage no records
template <typename T, int NT = kGridThreads> size_t grid_fixed_smem_bytes(int logTL, int m, bool own = false) {
  int logBS = 4;
  while ((1 << logBS) < 2 * m) ++logBS;
  const size_t NB = ((((size_t)1 << logTL) + 2 * m) >> logBS) + 1;
  const size_t staged = own ? 0 : (size_t)fixed_cap<T, NT>();
  return sizeof(typename FixAcc<T>::type) * ((size_t)1 << logTL) + sizeof(SRec<T>) * staged +
         kTapCoefBytes + sizeof(int) * NB;
}

// ---------------------------------------------------------------------------
// Tiles fed by the single-pass chunk-local binning (k_bin_local): a tile's
// records are nch runs, one per input chunk, located by loc[tile nch + c] =
// start | count << 16 within chunk c's region recs[c ch2 ..].
// ---------------------------------------------------------------------------
constexpr int kSegMaxChunks = 1024;

// element v of a tile's record list: binary search over the runs
template <typename T> struct SegSrc {
  typedef typename RecOf<T>::type Rec;
  const Rec *recs;
  const int *pre;   // shared, nch + 1: run c holds list elements [pre[c], pre[c+1])
  const int *base;  // shared, nch: record index of run c's first element
  int nch;
  __device__ __forceinline__ Rec operator[](int v) const {
    int lo = 0, hi = nch - 1;
    while (lo < hi) {  // last run with pre <= v (a non-empty one)
      const int mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= v) lo = mid;
      else hi = mid - 1;
    }
    return recs[base[lo] + (v - pre[lo])];
  }
};

// CTA-wide: the runs of `tile` into shared memory sh (2 nch + 1 ints);
// returns the length of the tile's record list.  Ends with a barrier.
__device__ __forceinline__ int seg_setup(const int *__restrict__ loc, int tile, int nch, int ch2, int *sh) {
  int *pre = sh, *cnt = sh + nch + 1;
  const int *row = loc + (int64_t)tile * nch;
  for (int c = threadIdx.x; c < nch; c += blockDim.x) cnt[c] = (unsigned)row[c] >> 16;
  __syncthreads();
  cta_exclusive_scan(cnt, pre, nch);
  for (int c = threadIdx.x; c < nch; c += blockDim.x) cnt[c] = c * ch2 + (row[c] & 0xffff);  // now the run bases
  __syncthreads();
  return pre[nch];
}

#define CUNA_SEG_KERNEL(NAME, BODY, OCC32, OCC64)                                                              \
  template <typename T, int CW>                                                                               \
  __global__ void __launch_bounds__(kGridThreads, sizeof(T) == 4 ? OCC32 : OCC64) NAME(                        \
      const typename RecOf<T>::type *__restrict__ recs, const int *__restrict__ loc, int nch, int ch2,          \
      int seg_off, T *__restrict__ grid, AccParams<T> e, const T *__restrict__ wts, int64_t nvals, int nslab,    \
      int group, int64_t slab_stride) {                                                                         \
    extern __shared__ __align__(16) unsigned char smem_raw[];                                                   \
    int *sh = reinterpret_cast<int *>(smem_raw + seg_off);                                                      \
    const int tile = blockIdx.x;                                                                                \
    const int sbeg = blockIdx.y * group, send = min(nslab, sbeg + group);                                       \
    const int total = seg_setup(loc, tile, nch, ch2, sh);                                                       \
    const SegSrc<T> src{recs, sh, sh + nch + 1, nch};                                                           \
    BODY(src, 0, total, tile << e.logTL, grid, e, wts, nvals, sbeg, send, slab_stride);                          \
  }
CUNA_SEG_KERNEL(k_grid_acc_seg, (grid_tile_body<T, CW>), 4, 2)
CUNA_SEG_KERNEL(k_grid_scatter_seg, grid_tile_scatter<T>, 6, 3)
CUNA_SEG_KERNEL(k_grid_fixed_seg, grid_tile_fixed<T>, 6, 2)
#undef CUNA_SEG_KERNEL

template <typename T> size_t grid_scatter_smem_bytes(int logTL) {
  return sizeof(T) * ((size_t)1 << logTL) + (sizeof(SRec<T>) + sizeof(int)) * (size_t)GridCfg<T>::CAP;
}

template <typename T> size_t grid_smem_bytes(int logTL, int m, int sg = 1) {
  const int W = (1 << logTL) + 2 * m;
  const size_t CAP = GridCfg<T>::CAP;
  return sizeof(int) * ((W + 2 + 3) & ~3) + sizeof(SRec<T>) * CAP + sizeof(int) * CAP +
         (sg > 1 ? 2 * sizeof(T) * sg * CAP : 0);
}

// Last four-step pass of the packed real transform: CTA owns row pairs
// (p, L1 - p), p in [p0, p0 + P), so both Z[k] and Z[L - k] are on chip.
template <typename T> struct PairRowSrc {
  const typename CxOf<T>::type *p;
  int logL2, L1, p0, npairs;
  __device__ __forceinline__ typename CxOf<T>::type load(int seq, int i) const {
    const int pp = p0 + (seq >> 1);
    const int row = (seq & 1) ? ((L1 - pp) & (L1 - 1)) : pp;
    return pp < npairs ? p[((int64_t)row << logL2) + i] : cmk((T)0, (T)0);
  }
};

// Last four-step pass of the packed real transform for row pairs (p, L1 - p),
// p in [p0, p0 + P): both Z[k] and Z[L - k] are on chip for the unpack.
template <typename T>
__device__ __forceinline__ void rowpass_acc_body(const typename CxOf<T>::type *__restrict__ in,
                                                 const FftDev<T> &f, const AccParams<T> &e,
                                                 typename CxOf<T>::type *F, int pblock) {
  typedef typename CxOf<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int L1 = 1 << f.logL1, L2 = 1 << f.logL2;
  const int logB = ilog2i((int64_t)blockDim.x * kFftE) - f.logL2;
  const int B = 1 << logB, logP = logB - 1, P = B >> 1;
  const int pitch = fft_pitch(L2, B);
  const int p0 = pblock * P, npairs = L1 / 2 + 1;
  const int tot = B << f.logL2;
  PairRowSrc<T> src{in, f.logL2, L1, p0, npairs};
  fft_fused<T, false, false, false>(s, pitch, f.logL2, logB, f.tw2, src, NoDst());
  for (int idx = threadIdx.x; idx < tot; idx += blockDim.x) {
    const int i = idx & (P - 1), half = (idx >> logP) & 1, k2 = idx >> (logP + 1);
    const int p = p0 + i;
    if (p >= npairs) continue;
    const int rowA = p, rowB = (L1 - p) & (L1 - 1);
    if (half && rowA == rowB) continue;
    const int k1 = half ? rowB : rowA;
    const int64_t k = (int64_t)k1 + ((int64_t)k2 << f.logL1);
    if (k > e.K) continue;
    const int k2m = k1 == 0 ? ((L2 - k2) & (L2 - 1)) : (L2 - 1 - k2);
    const C Zk = s[(2 * i + half) * pitch + pad16(k2)];
    const C Zm = cconj(s[(2 * i + 1 - half) * pitch + pad16(k2m)]);
    acc_output<T>(e, k, Zk, Zm, F);
  }
}

template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256) k_fft_rowpass_acc(const typename CxOf<T>::type *__restrict__ in,
                                                         FftDev<T> f, AccParams<T> e,
                                                         typename CxOf<T>::type *F) {
  // slab blockIdx.y
  rowpass_acc_body<T>(in + ((int64_t)blockIdx.y << f.logL), f, e, F + (int64_t)blockIdx.y * e.nf, blockIdx.x);
}

// ---------------------------------------------------------------------------
// bootstrap: resample b draws n indices d = xorshift32(wang_hash(seed + b*n +
// i)) % n with replacement; gridding resample b is gridding every original
// sample p with weight (number of times p was drawn) * y[p].
// ---------------------------------------------------------------------------
constexpr int kBootSmemN = 40960;  // int counters in shared memory (160 KB)

template <typename T>
__global__ void __launch_bounds__(1024) k_boot_weights(const T *__restrict__ y, int n, unsigned seed,
                                                       T *__restrict__ wts) {
  extern __shared__ int cnt[];
  pdl_trigger();
  const int b = blockIdx.x;
  T *w = wts + (int64_t)b * n;
  const unsigned s0 = seed + (unsigned)b * (unsigned)n;
  if (n <= kBootSmemN) {
    for (int p = threadIdx.x; p < n; p += blockDim.x) cnt[p] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      atomicAdd(&cnt[boot_draw(s0, (unsigned)i, (unsigned)n)], 1);
    __syncthreads();
    for (int p = threadIdx.x; p < n; p += blockDim.x) w[p] = (T)cnt[p] * y[p];
  } else {
    // w was zeroed; adding identical values y[d] is exact in any order
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const unsigned d = boot_draw(s0, (unsigned)i, (unsigned)n);
      atomicAdd(&w[d], y[d]);
    }
  }
  pdl_wait();  // a sort launched before runs beside this; who waits for this waits for both
}

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
size_t align_up(size_t v) { return (v + 255) & ~(size_t)255; }

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

}  // namespace
}  // namespace cuna

