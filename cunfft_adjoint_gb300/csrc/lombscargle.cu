// lombscargle.cu -- generalised Lomb-Scargle periodogram on top of the adjoint
// NFFT (the use the reference library was written for, its README).
//
// Floating-mean periodogram (Zechmeister & Kuerster 2009) with weights
// w_j = 1/dy_j^2 normalised to sum 1 (uniform without dy), at frequencies
// f_k = (k + 1) df, k = 0 .. nfreq-1:
//   A_k = sum_j w_j (y_j - ybar) e^{i w t_j},  B_k = sum_j w_j e^{i w t_j},
//   YC = Re A, YS = Im A, C = Re B_k, S = Im B_k, C2 = Re B_2k, S2 = Im B_2k,
//   CC = (1 + C2)/2 - C^2, SS = (1 - C2)/2 - S^2, CS = S2/2 - C S,
//   P = (SS YC^2 + CC YS^2 - 2 CS YC YS) / (YY (CC SS - CS^2)),
//   YY = sum_j w_j (y_j - ybar)^2.
// A and B come from one two-channel adjoint NFFT (cuna2_adjoint_multi: shared
// binning and gridding) of an accurate plan with period T = 1/df, so output
// bin k is frequency k df; the common phase factor of the
// x = (t - t0)/T - 1/2 origin multiplies A_k, B_k by (-1)^k and B_2k by 1,
// which leaves P unchanged.
#include <math.h>
#include <map>
#include <mutex>
#include <tuple>
#include "common.cuh"
#include "runtime.h"

namespace cuna {
namespace {

// CTAs of two warps: the FP64 pipe takes a warp's instruction 16 cycles, and
// these short kernels are chains of them (divisions, shuffled sums), so few
// warps per SM finish sooner (a periodogram of 5003 samples at 50000
// frequencies: 50.5 us with eight warps per CTA, 44.4 with two)
constexpr int kLsThreads = 64;
constexpr int kLsMaxBlocks = 1024;  // CTAs of the sums pass
constexpr int kLsPowerThreads = 128;

// Partial sums of w, w y and w y^2 (double), three per CTA, added up in CTA
// order by every later reader (ls_totals): no memset and no atomics, and the
// same totals on every run.
template <typename T>
__global__ void __launch_bounds__(kLsThreads) k_ls_sums(const T *__restrict__ y, const T *__restrict__ dy, int64_t n,
                                                        double *part) {
  __shared__ double sh[3][kLsThreads / 32];
  double a = 0, b = 0, c = 0;
  pdl_trigger();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double w = dy ? 1.0 / ((double)dy[i] * (double)dy[i]) : 1.0;
    const double v = (double)y[i];
    a += w;
    b += w * v;
    c += w * v * v;
  }
  pdl_wait();  // runs beside the binning, which must be complete when the weights are
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    c += __shfl_down_sync(0xffffffffu, c, o);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
    sh[0][w] = a;
    sh[1][w] = b;
    sh[2][w] = c;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0;
    for (int q = 0; q < kLsThreads / 32; ++q) s += sh[threadIdx.x][q];
    part[3 * blockIdx.x + threadIdx.x] = s;
  }
}

// the totals of np partial sums, for every thread of the CTA (a warp adds one
// sum at a time); part is read through L2: its writer may still have been
// running when this kernel started
__device__ __forceinline__ void ls_totals(const double *part, int np, double *tot) {
  __shared__ double sh[3];
  const int lane = threadIdx.x & 31;
  for (int w = threadIdx.x >> 5; w < 3; w += blockDim.x >> 5) {
    double s = 0;
    for (int q = lane; q < np; q += 32) s += __ldcg(part + 3 * q + w);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) sh[w] = s;
  }
  __syncthreads();
  tot[0] = sh[0];
  tot[1] = sh[1];
  tot[2] = sh[2];
}

// w_j / sum w and w_j (y_j - ybar) / sum w
template <typename T>
__global__ void __launch_bounds__(kLsThreads) k_ls_weights(const T *__restrict__ y, const T *__restrict__ dy, int64_t n,
                                                           const double *part, int np, T *w, T *wy) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const double wj = i < n && dy ? 1.0 / ((double)dy[i] * (double)dy[i]) : 1.0;
  pdl_trigger();
  pdl_wait();  // the partial sums
  double s[3];
  ls_totals(part, np, s);
  if (i >= n) return;
  const double W = s[0], ybar = s[1] / s[0];
  const double wi = wj / W;
  w[i] = (T)wi;
  wy[i] = (T)(wi * ((double)y[i] - ybar));
}

// P of one frequency from A_k, B_k, B_2k and YY.  Float spectra: in float-float
// (48 bits, where the result keeps 24), because some fifty FP64 operations per
// frequency bound this kernel (50000 frequencies 9.5 us, 6.3 us here); the
// values are first scaled by a power of two that brings YY near 1, so that
// neither large nor small data leave the float range.
__device__ __forceinline__ double ls_value(double2 a, double2 b, double2 b2, double YY) {
  const double YC = a.x, YS = a.y, C = b.x, S = b.y, C2 = b2.x, S2 = b2.y;
  const double CC = 0.5 * (1.0 + C2) - C * C;
  const double SS = 0.5 * (1.0 - C2) - S * S;
  const double CS = 0.5 * S2 - C * S;
  const double D = CC * SS - CS * CS;
  const double num = SS * YC * YC + CC * YS * YS - 2.0 * CS * YC * YS;
  return YY > 0 && D > 0 ? num / (YY * D) : 0.0;
}
__device__ __forceinline__ float ls_value(float2 a, float2 b, float2 b2, double YY) {
  if (!(YY > 0)) return 0.f;
  const int k = ((int)((__double_as_longlong(YY) >> 52) & 0x7ff) - 1023) / 2;
  const dfl yy = df_from_double(ldexp(YY, -2 * k));
  const dfl YC(ldexpf(a.x, -k), 0.f), YS(ldexpf(a.y, -k), 0.f), C(b.x, 0.f), S(b.y, 0.f), h(0.5f, 0.f);
  const dfl CC = h * (dfl(1.f, 0.f) + dfl(b2.x, 0.f)) - C * C;
  const dfl SS = h * (dfl(1.f, 0.f) - dfl(b2.x, 0.f)) - S * S;
  const dfl CS = h * dfl(b2.y, 0.f) - C * S;
  const dfl D = CC * SS - CS * CS;
  const dfl c = CS * YC * YS;
  const dfl num = SS * YC * YC + CC * YS * YS - (c + c);
  const dfl v = num * df_rcp(yy * D);
  return D.hi > 0.f ? v.hi + v.lo : 0.f;
}

template <typename T>
__global__ void __launch_bounds__(kLsPowerThreads) k_ls_power(const typename CxOf<T>::type *A,
                                                              const typename CxOf<T>::type *B, int64_t K,
                                                              int64_t nfreq, const double *part, int np, T *P) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // frequency (k + 1) df
  __shared__ double yy;
  pdl_wait();  // the spectra (and, long before, the partial sums)
  double sums[3];
  ls_totals(part, np, sums);
  if (threadIdx.x == 0) {  // once per CTA: the divisions are on the FP64 pipe
    const double W = sums[0], ybar = sums[1] / W;
    yy = sums[2] / W - ybar * ybar;
  }
  __syncthreads();
  if (k >= nfreq) return;
  const int64_t q = k + 1;
  P[k] = ls_value(A[K + q], B[K + q], B[K + 2 * q], yy);
}

// The plans of one stream, as its workspace: the caller never sees them, so
// calls on two streams must not share the records and grids of one.  The mutex
// is held while a call is enqueued: another thread's call on the same stream
// uses the same buffers and comes after all of it.
struct LsStream {
  std::mutex mu;
  std::map<std::tuple<int, int64_t, int, int>, cuna2_plan> plans;  // (dtype, nf, R, m)
};
std::mutex g_ls_mu;
std::map<std::pair<int, cudaStream_t>, LsStream> *g_ls = new std::map<std::pair<int, cudaStream_t>, LsStream>();
LsStream &ls_stream(int dev, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_ls_mu);
  return (*g_ls)[std::make_pair(dev, st)];  // never erased: the reference stays valid
}

template <typename T>
int ls_run(int dtype, const double *t, const T *y, const T *dy, int64_t n, int64_t nfreq, double df, double t0,
           int R, int m, T *P, cudaStream_t st) {
  typedef typename CxOf<T>::type C;
  if (n < 2 || !t || !y || !P || nfreq < 1 || !(df > 0) || !std::isfinite(df) || !std::isfinite(t0))
    return fail(CUNA2_ERROR_INVALID_VALUE, "invalid argument (n=%lld nfreq=%lld df=%g)", (long long)n,
                (long long)nfreq, df);
  // outputs up to 2 (nfreq) df are needed: nf / 2 > 2 nfreq, nf a power of two
  int64_t nf = 2;
  while (nf / 2 <= 2 * nfreq) nf *= 2;
  int dev = 0;
  CUNA_CK(cudaGetDevice(&dev));
  LsStream &ls = ls_stream(dev, st);
  std::lock_guard<std::mutex> lk(ls.mu);
  cuna2_plan plan = nullptr;
  const auto key = std::make_tuple(dtype, nf, R, m);
  const auto it = ls.plans.find(key);
  if (it == ls.plans.end()) {
    CUNA_TRY(cuna2_plan_create(&plan, dtype, nf, R, m));
    ls.plans[key] = plan;
  } else {
    plan = it->second;
  }
  // workspace: partial sums | channels [wy; w] | outputs [A; B]
  const int np = (int)std::min<int64_t>(std::min(kLsMaxBlocks, 4 * device_sm_count()), (n + kLsThreads - 1) / kLsThreads);
  const size_t o_ch = 3 * sizeof(double) * kLsMaxBlocks, o_A = o_ch + ((2 * sizeof(T) * n + 255) & ~(size_t)255);
  void *ws = nullptr;
  CUNA_TRY(stream_workspace(st, o_A + 2 * sizeof(C) * nf, &ws));
  char *w8 = (char *)ws;
  double *part = (double *)w8;
  T *wy = (T *)(w8 + o_ch), *w = wy + n;
  C *A = (C *)(w8 + o_A), *B = A + nf;
  // both channels in one fused transform (shared binning and gridding); the
  // sums and weights run beside its binning
  struct Work {
    const T *y, *dy;
    int64_t n;
    double *part;
    int np;
    T *w, *wy;
    cudaStream_t st;
  } work{y, dy, n, part, np, w, wy, st};
  const MultiValues values{[](void *c, bool after) -> int {
                             const Work &k = *static_cast<const Work *>(c);
                             const dim3 th(kLsThreads);
                             if (after) CUNA_CK(launch_pdl(k_ls_sums<T>, dim3(k.np), th, 0, k.st, k.y, k.dy, k.n, k.part));
                             else k_ls_sums<T><<<k.np, th, 0, k.st>>>(k.y, k.dy, k.n, k.part);
                             CUNA_CK(cudaGetLastError());
                             CUNA_CK(launch_pdl(k_ls_weights<T>, dim3((unsigned)((k.n + kLsThreads - 1) / kLsThreads)), th,
                                                0, k.st, k.y, k.dy, k.n, (const double *)k.part, k.np, k.w, k.wy));
                             return CUNA2_SUCCESS;
                           },
                           &work};
  const double T_ = 1.0 / df;
  CUNA_TRY(adjoint_multi_values(plan, t, wy, A, n, 2, t0, T_, values, st));
  CUNA_CK(launch_pdl(k_ls_power<T>, dim3((unsigned)((nfreq + kLsPowerThreads - 1) / kLsPowerThreads)),
                     dim3(kLsPowerThreads), 0, st, (const C *)A, (const C *)B, nf / 2, nfreq, (const double *)part, np, P));
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

}  // namespace
}  // namespace cuna

using namespace cuna;

extern "C" int cuna2_lomb_scargle(int dtype, const double *t, const void *y, const void *dy, int64_t n,
                                  int64_t nfreq, double df, double t0, int R, int m, void *power,
                                  cudaStream_t stream) {
  clear_error();
  if (dtype == CUNA2_F32)
    return ls_run<float>(dtype, t, (const float *)y, (const float *)dy, n, nfreq, df, t0, R, m, (float *)power,
                         stream);
  if (dtype == CUNA2_F64)
    return ls_run<double>(dtype, t, (const double *)y, (const double *)dy, n, nfreq, df, t0, R, m, (double *)power,
                          stream);
  return fail(CUNA2_ERROR_INVALID_VALUE, "dtype %d", dtype);
}
