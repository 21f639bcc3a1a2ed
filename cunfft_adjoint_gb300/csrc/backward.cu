// backward.cu -- backward (vector-Jacobian product) of the accurate transform.
//
// With g_k = dL/dRe F_k + i dL/dIm F_k for the stored outputs,
//   h_k = g_k (-1)^k / psi_hat(k),      R_c = Re sum_k h_k exp(-2 pi i k c / ng),
//   dL/dy_j = sum_d R_{b+d} psi(d - f),
//   dL/dt_j = (ng / T) y_j sum_d R_{b+d} (d - f) / (2 tau) psi(d - f),
// d = -m+1..m, b + f = s_j the grid position.  R is real: with the Hermitian
// part H_k = (h_k + conj(h_{-k})) / 2 of h, R = DFT_-(H) is computed as one
// complex DFT of length L = ng/2 of Zin[k] = E[k] + i O[k], E[k] = H_k +
// H_{k+L}, O[k] = (H_k - H_{k+L}) exp(-2 pi i k / ng), whose output is
// R[2n] + i R[2n+1].  DFT_- = conj(DFT_+(conj(.))); the conjugations are fused
// into the load and store functors of the (inverse-sign) FFT passes.
//
// Kernels: k_bwd_small (one CTA per series holds the whole grid), else
// k_ct_bwd_col + k_ct_bwd_row (four-step passes of compile-time geometry, the
// spectrum formed by the column pass's loads) + k_bwd_interp.
#include <math.h>
#include <algorithm>
#include <type_traits>
#include "accurate_kernels.cuh"
#include "backward.h"
#include "fftpass_core.cuh"

namespace cuna {
namespace {

// conj(Zin[q]) of one series.  The output band is |k| <= K, K = nf/2 <= L/2,
// so of H_q and H_{q+L} = H_{q-L} at most one is non-zero for a given q in
// [0, L), H_q for q <= K, H_{q-L} for q >= L - K; both exist only where q = K
// = L/2.  Two loads of G and one deconvolution factor (even in k) per point.
// (A general h(k) for each of the four terms, with its 64-bit remainders and
// exps, took 285 us of the 64 x 2^18-point float batch, 117 us here.)
// The float sums round as that form did, term by term: dL/dt leaves in
// double, where a change of rounding would show.
template <typename T> struct BwdSpec {
  typedef typename CxOf<T>::type C;
  const C *G;  // the series' G[k + K] at k = 0
  int K, L;
  T c0b, c1;   // 1 / psi_hat(k) = c0b exp(c1 k^2)
  // H_k, |k| <= K
  __device__ __forceinline__ C herm(int k) const {
    const T kf = (T)k;
    T sc = c0b * exp_t(c1 * kf * kf);
    if (k & 1) sc = -sc;
    C a = cmk((T)0, (T)0), b = a;
    if (k < K) a = G[k];
    if (k > -K) b = G[-k];
    if constexpr (sizeof(T) == 4)
      return cmk(__fmul_rn(__fadd_rn(__fmul_rn(a.x, sc), __fmul_rn(b.x, sc)), 0.5f),
                 __fmul_rn(__fadd_rn(__fmul_rn(a.y, sc), -__fmul_rn(b.y, sc)), 0.5f));
    else
      return cscale(cmk(a.x + b.x, a.y - b.y), sc * (T)0.5);
  }
  __device__ __forceinline__ C zin_conj(int q, T cs, T sn) const {  // cs + i sn = exp(+2 pi i q / ng)
    const bool first = q <= K;
    const int k = first ? q : q - L;
    if (k < -K) return cmk((T)0, (T)0);
    C E = herm(k), D = first ? E : cmk(-E.x, -E.y);
    if (first && q == L - K) {  // q = K = L/2
      const C Hp = herm(-K);
      D = csub(E, Hp);
      E = cadd(E, Hp);
    }
    const C O = cmul(D, cmk(cs, -sn));  // (H_q - H_{q+L}) e^{-2 pi i q / ng}
    return cconj(cadd(E, cmuli(O)));
  }
};

// c_j = exp2(-k1 j^2), j = 0..: the Gaussian's coefficients about its centre
// cell, and j c_j
constexpr int kBwdCoefs = 24;
template <typename T> struct BwdCoef {
  T c[kBwdCoefs], jc[kBwdCoefs];
  T k1, inv2tau;
};

// Both interpolation sums at one sample from the W = NG V cells at base b0 (a
// multiple of V, V = 16 bytes of cells; the 2M-cell window starts at cell a =
// 0..V-1 of them): W/V vector loads instead of 2M scalar ones.  Only the first
// and the last groups hold cells outside the window; they are set to zero.
//  - float: exp2 per tap (the hardware's, whose bits exp2f returns for the
//    exponents above -126 that taps have) and the sums in tap order; what is
//    not a sum runs on two taps at a time in the packed instructions, which
//    round each half as the scalar ones do.
//  - double: with h the centre cell, x0 = b0 + h - s and the factorisation
//    exp2(-k1 (j + x0)^2) = E Q^j c_j (E = exp2(-k1 x0^2), Q = exp2(-2 k1 x0),
//    c_j = exp2(-k1 j^2)), the sums run as two Horner chains outwards-in:
//    right in Q, left in 1/Q.  Three FP64 exp2 per sample instead of 2M.
template <typename T, int M> struct BwdWin {
  static constexpr int V = sizeof(T) == 4 ? 4 : 2;
  static constexpr int NG = (2 * M + V - 1 + V - 1) / V;  // groups that cover any alignment
  static constexpr int W = NG * V;
  static constexpr int H = M + (V == 4 ? 1 : 0);  // centre cell: |x0| <= 2 (float), 1 (double)
};
// ordinary (coherent) loads: neighbouring samples' windows overlap, so the L1
// serves most of them
template <typename T, int V> struct BwdVec;
template <> struct BwdVec<float, 4> {
  __device__ static __forceinline__ void load(const float *p, float *v) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
};
template <> struct BwdVec<double, 2> {
  __device__ static __forceinline__ void load(const double *p, double *v) {
    const double2 q = *reinterpret_cast<const double2 *>(p);
    v[0] = q.x, v[1] = q.y;
  }
};
template <typename T, int M>
__device__ __forceinline__ void bwd_window(const T *R, int ng, int cell, T fr, const BwdCoef<T> &cf, T &sy, T &st) {
  typedef BwdWin<T, M> X;
  constexpr int V = X::V, W = X::W, H = X::H;
  const int lo = cell - M + 1;
  const int b0 = lo & ~(V - 1), a = lo - b0;
  T v[W];
  if ((unsigned)b0 <= (unsigned)(ng - W)) {
#pragma unroll
    for (int g = 0; g < X::NG; ++g) BwdVec<T, V>::load(R + b0 + g * V, v + g * V);
  } else {  // wraps around the period
#pragma unroll
    for (int g = 0; g < X::NG; ++g) {
      int b = b0 + g * V;
      if (b < 0) b += ng;
      else if (b >= ng) b -= ng;
      BwdVec<T, V>::load(R + b, v + g * V);
    }
  }
  // cells before the window (i < a <= V - 1) and after it (i >= a + 2M)
#pragma unroll
  for (int i = 0; i < W; ++i) {
    if (i < V - 1) v[i] = i < a ? (T)0 : v[i];
    if (i >= 2 * M) v[i] = i < a + 2 * M ? v[i] : (T)0;
  }
  if constexpr (sizeof(T) == 4) {
    const float d0 = (float)(b0 - cell);
    const f2 nk = pk2(-cf.k1, -cf.k1), nf = pk2(-fr, -fr), two = pk2(2.f, 2.f);
    f2 D = pk2(d0, d0 + 1.f);  // the cells' whole distances, exact
    sy = 0.f;
    st = 0.f;
#pragma unroll
    for (int i = 0; i < W; i += 2) {
      const f2 dd = add2(D, nf);
      float x0, x1, w0, w1, u0, u1;
      unpk2(mul2(mul2(nk, dd), dd), x0, x1);
      const f2 w = mul2(pk2(v[i], v[i + 1]), pk2(exp2_g(x0), exp2_g(x1)));
      unpk2(w, w0, w1);
      unpk2(mul2(w, dd), u0, u1);
      sy += w0;
      st = fmaf(u0, cf.inv2tau, st);
      sy += w1;
      st = fmaf(u1, cf.inv2tau, st);
      D = add2(D, two);
    }
  } else {
    const T x0 = (T)(b0 + H - cell) - fr;
    const T E = exp2_t(-cf.k1 * x0 * x0), Q = exp2_t((T)(-2) * cf.k1 * x0), Qi = (T)1 / Q;
    T r = (T)0, rt = (T)0, l = (T)0, lt = (T)0;  // sums of p and of j p, |x0| <= 1
#pragma unroll
    for (int i = W - 1; i >= H; --i) {
      r = fma(r, Q, v[i] * cf.c[i - H]);
      rt = fma(rt, Q, v[i] * cf.jc[i - H]);
    }
#pragma unroll
    for (int i = 0; i < H; ++i) {
      l = fma(l, Qi, v[i] * cf.c[H - i]);
      lt = fma(lt, Qi, v[i] * -cf.jc[H - i]);
    }
    const T S = fma(l, Qi, r);
    sy = E * S;
    st = E * fma(x0, S, fma(lt, Qi, rt)) * cf.inv2tau;
  }
}

// float -> double by the bit fields for normal values and zero (the
// conversion instruction runs on the narrow FP64 pipe)
__device__ __forceinline__ double to_double(double v) { return v; }
__device__ __forceinline__ double to_double(float v) {
  const unsigned u = __float_as_uint(v), e = (u >> 23) & 0xff;
  if (e == 0 || e == 255) return (double)v;
  return __hiloint2double((int)((u & 0x80000000u) | (((u >> 3) & 0x0fffffffu) + 0x38000000u)), (int)(u << 29));
}

// Interpolation at every sample of the series blockIdx.y from its real field.
// Bound by the instruction issue (float, 64 series of 2e5 sorted samples, m =
// 10: 276 us with 2m scalar loads, wraps and a 64-bit division per sample, 191
// us with scalar arithmetic and a wrap test per group, 170 us here) and, for
// double, by the FP64 pipe (2e5 samples: 217 us with an exp2
// per tap, 65 us here).
template <typename T, int M>
__global__ void __launch_bounds__(256) k_bwd_interp(const double *__restrict__ t, const T *__restrict__ y, int64_t n,
                                                    const __grid_constant__ BwdSeries ser, int64_t ng,
                                                    const __grid_constant__ BwdCoef<T> cf, const T *R, T *gy,
                                                    double *gt) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int s = blockIdx.y;
  const int64_t o = (int64_t)s * n + j;
  int cell = 0;
  T fr = (T)0;
  if (j < n) reduce_sample<T>(t[o], ser.pm[s], ng, cell, fr);
  pdl_wait();  // the field comes from the row pass
  if (j >= n) return;
  T a, b;
  bwd_window<T, M>(R + (int64_t)s * ng, (int)ng, cell, fr, cf, a, b);
  if (gy) gy[o] = a;
  if (gt) gt[o] = ser.tscale[s] * to_double(y[o]) * to_double(b);
}

// Single CTA per series: spectrum -> shared memory -> FFT -> interpolation at
// every sample.  CTA b handles series b of the batch.  The same sums as
// bwd_window, over the 2m taps of the window.  Latency-bound: 48 series of
// 3001 samples, L = 4096, 44 us with 256 threads and a general h(k), 22 us
// here.
template <typename T>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512) k_bwd_small(
    const double *__restrict__ t, const T *__restrict__ y, int64_t n, const __grid_constant__ BwdSeries ser,
    const __grid_constant__ BwdCoef<T> cf, BwdSpec<T> sp, int m, FftDev<T> f, T *__restrict__ gy,
    double *__restrict__ gt) {
  typedef typename CxOf<T>::type C;
  const int b = blockIdx.x;
  const PhaseMul pm = ser.pm[b];
  const double tscale = ser.tscale[b];
  t += (int64_t)b * n;
  if (y) y += (int64_t)b * n;
  if (gy) gy += (int64_t)b * n;
  if (gt) gt += (int64_t)b * n;
  sp.G += (int64_t)b * 2 * sp.K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 1 << f.logL, ng = 2 * L;
  const int pitch = fft_pitch(L, 1);
  C *s = reinterpret_cast<C *>(smem_raw);
  const T *sr = reinterpret_cast<const T *>(smem_raw);
  const T twk = (T)1 / (T)L;
  for (int q = threadIdx.x; q < L; q += blockDim.x) {
    T sn, cs;
    sincospi_t((T)q * twk, &sn, &cs);
    s[pad16(q)] = sp.zin_conj(q, cs, sn);
  }
  __syncthreads();
  smem_fft<T>(s, pitch, f.logL, 1, f.tw1);
  // output z[nn] = conj(FFT result): R[2nn] = Re, R[2nn+1] = -Im
  auto R = [&](int c) -> T {
    const T v = sr[real_slot(c)];
    return (c & 1) ? -v : v;
  };
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x) {
    int cell;
    T fr;
    reduce_sample<T>(t[j], pm, ng, cell, fr);
    T a, bt;
    if constexpr (sizeof(T) == 4) {
      a = (T)0;
      bt = (T)0;
      for (int d = -m + 1; d <= m; ++d) {
        int c = cell + d;
        if (c < 0) c += ng;
        else if (c >= ng) c -= ng;
        const T dd = (T)d - fr;
        const T w = R(c) * exp2_g(-cf.k1 * dd * dd);
        a += w;
        bt += w * dd * cf.inv2tau;
      }
    } else {
      const T E = exp2_t(-cf.k1 * fr * fr), Q = exp2_t((T)2 * cf.k1 * fr), Qi = exp2_t((T)(-2) * cf.k1 * fr);
      T r = (T)0, rt = (T)0, l = (T)0, lt = (T)0;
      for (int d = m; d >= 0; --d) {
        int c = cell + d;
        if (c >= ng) c -= ng;
        const T p = R(c) * cf.c[d];
        r = fma(r, Q, p);
        rt = fma(rt, Q, p * ((T)d - fr));
      }
      for (int d = -m + 1; d < 0; ++d) {
        int c = cell + d;
        if (c < 0) c += ng;
        const T p = R(c) * cf.c[-d];
        l = fma(l, Qi, p);
        lt = fma(lt, Qi, p * ((T)d - fr));
      }
      a = E * fma(l, Qi, r);
      bt = E * fma(lt, Qi, rt) * cf.inv2tau;
    }
    if (gy) gy[j] = a;
    if (gt) gt[j] = tscale * to_double(y[j]) * to_double(bt);
  }
}

// four-step pass A: columns of conj(Zin) formed from G by the first stage's
// loads.  exp(2 pi i q / ng), q = i L2 + c: float calls sincospif; double, for
// which that costs the FP64 pipe more than the FFT, takes exp(2 pi i (i / 2) /
// L1) (the FFT's own table) times a per-column factor for i's parity from
// shared memory.
template <typename T, int LOG1, int LOG2> struct CtSpecSrc {
  typedef typename CxOf<T>::type C;
  BwdSpec<T> sp;
  const C *tw1;
  const C *twc;  // double, shared: twc[2 seq + parity] = exp(2 pi i (c0 + seq + parity L2) / ng)
  int c0;
  __device__ __forceinline__ C load(int seq, int j, int dr) const {
    const int i = j + dr, q = (i << LOG2) + c0 + seq;
    if constexpr (sizeof(T) == 4) {
      T sn, cs;
      sincospi_t((T)q * ((T)1 / (T)(1 << (LOG1 + LOG2))), &sn, &cs);
      return sp.zin_conj(q, cs, sn);
    } else {
      const C w = cmul(ldtw(tw1 + (i >> 1)), twc[2 * seq + (i & 1)]);
      return sp.zin_conj(q, w.x, w.y);
    }
  }
};

// float: each output times its W_L^{c k} from the two-level table (one
// rounding less than CtColDst's)
template <int LOG1, int LOG2> struct CtColDstTw {
  float2 *p;  // slab + c0
  FftDev<float> f;
  int c0;
  template <int R, int LOGNS> __device__ __forceinline__ void store(int seq, int idxD, float2 *v) const {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = idxD + (r << LOGNS);
      p[(k << LOG2) + seq] = cmul(v[r], twiddle_L(f, (c0 + seq) * k));
    }
  }
};

template <typename T, int LOGL, int LOGE>
__global__ void __launch_bounds__(1 << (LOGE - 4)) k_ct_bwd_col(BwdSpec<T> sp, typename CxOf<T>::type *z, FftDev<T> f) {
  typedef typename CxOf<T>::type C;
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2;
  constexpr int LOGB = LOGE - LOG1, B = 1 << LOGB;
  constexpr int PITCH = fft_pitch(1 << LOG1, B);
  constexpr int LNS = last_logns<LOG1>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  C *steps = s + PITCH * B, *twc = steps + 17 * B;
  const int c0 = blockIdx.x * B;
  pdl_trigger();
  sp.G += (int64_t)blockIdx.y * 2 * sp.K;  // series blockIdx.y of a batch
  z += (int64_t)blockIdx.y << LOGL;
  if constexpr (sizeof(T) == 8) {
    for (int i = threadIdx.x; i < 16 * B; i += 1 << (LOGE - 4))
      steps[(i >> 4) * 17 + (i & 15)] = twiddle_L(f, (c0 + (i >> 4)) * ((i & 15) << LNS));
    for (int i = threadIdx.x; i < 2 * B; i += 1 << (LOGE - 4)) {
      T sn, cs;
      sincospi_t((T)(c0 + (i >> 1) + ((i & 1) << LOG2)) / (T)(1 << LOGL), &sn, &cs);
      twc[i] = cmk(cs, sn);
    }
    __syncthreads();  // the first stage's loads read twc
  }
  CtSpecSrc<T, LOG1, LOG2> src{sp, f.tw1, twc, c0};
  if constexpr (sizeof(T) == 4) {
    CtColDstTw<LOG1, LOG2> dst{z + c0, f, c0};
    ct_fft<T, LOG1, LOGB, true, true, true, true>(s, f.tw1, src, dst);
  } else {
    CtColDst<T, LOG1, LOG2, LOGB> dst{z + c0, steps, f, c0};
    ct_fft<T, LOG1, LOGB, true, true, true>(s, f.tw1, src, dst);
  }
}

// pass B: rows -> real field R (conjugated outputs, interleaved re/im)
template <typename T, int LOG2> struct CtBwdRowSrc {
  const typename CxOf<T>::type *p;  // first row of the block
  __device__ __forceinline__ typename CxOf<T>::type load(int seq, int j, int dr) const {
    return __ldcg(p + (seq << LOG2) + j + dr);  // through L2: the column pass may still be writing
  }
};
template <typename T, int LOG1> struct CtConjDst {
  typename CxOf<T>::type *r;  // R viewed as L complex values, at the block's first row
  template <int R, int LOGNS>
  __device__ __forceinline__ void store(int seq, int idxD, typename CxOf<T>::type *v) const {
#pragma unroll
    for (int q = 0; q < R; ++q) r[seq + ((idxD + (q << LOGNS)) << LOG1)] = cconj(v[q]);
  }
};

template <typename T, int LOGL, int LOGE>
__global__ void __launch_bounds__(1 << (LOGE - 4)) k_ct_bwd_row(const typename CxOf<T>::type *z,
                                                                typename CxOf<T>::type *r, FftDev<T> f) {
  typedef typename CxOf<T>::type C;
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2;
  constexpr int LOGB = LOGE - LOG2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  const int r0 = blockIdx.x << LOGB;
  pdl_trigger();
  pdl_wait();  // the rows come from the column pass
  CtBwdRowSrc<T, LOG2> src{z + ((int64_t)blockIdx.y << LOGL) + ((int64_t)r0 << LOG2)};
  CtConjDst<T, LOG1> dst{r + ((int64_t)blockIdx.y << LOGL) + r0};
  ct_fft<T, LOG2, LOGB, true, false, true, true>(s, f.tw2, src, dst);
}

// Dependent launch for the float kernels only.  The double ones are bound by
// the FP64 pipe: CTAs that become resident early crowd the SMs that happen to
// have room and then share their pipes (2e5 samples, Nf = 2^18, forward and
// backward: 287 us with dependent launches, 225 without).
template <typename T, typename... KArgs, typename... Args>
cudaError_t launch_bwd(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  if (sizeof(T) == 4) return launch_pdl(k, grid, block, smem, st, args...);
  k<<<grid, block, smem, st>>>(static_cast<KArgs>(args)...);
  return cudaGetLastError();
}

// double, one series of 2^18 points: the two passes 178 + 43 us with the
// general spectrum and 64 CTAs of 4096 points, 61 + 21 us here (near the FP64
// pipe's rate for the butterflies, twiddles and one exp per point)
template <typename T, int LOGL, int LOGE>
int bwd_passes_sized(const BwdSpec<T> &sp, typename CxOf<T>::type *z, typename CxOf<T>::type *r, const FftDev<T> &f,
                     int ns, cudaStream_t st) {
  typedef typename CxOf<T>::type C;
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2, BA = 1 << (LOGE - LOG1), BB = 1 << (LOGE - LOG2);
  constexpr size_t smA = ct_colpass_smem<T, LOGL, LOGE>() + sizeof(C) * 2 * BA;
  constexpr size_t smB = sizeof(C) * (size_t)fft_pitch(1 << LOG2, BB) * BB;
  static SetupFlag attr;
  if (!setup_done(&attr)) {
    CUNA_CK(cudaFuncSetAttribute(k_ct_bwd_col<T, LOGL, LOGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smA));
    CUNA_CK(cudaFuncSetAttribute(k_ct_bwd_row<T, LOGL, LOGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smB));
    mark_setup_done(&attr);
  }
  k_ct_bwd_col<T, LOGL, LOGE><<<dim3((1 << LOG2) / BA, ns), 1 << (LOGE - 4), smA, st>>>(sp, z, f);
  CUNA_CK(cudaGetLastError());
  CUNA_CK(launch_bwd<T>(k_ct_bwd_row<T, LOGL, LOGE>, dim3((1 << LOG1) / BB, ns), dim3(1 << (LOGE - 4)), smB, st, z, r, f));
  return CUNA2_SUCCESS;
}

template <typename T, int LOGL>
int bwd_passes_at(const BwdSpec<T> &sp, typename CxOf<T>::type *z, typename CxOf<T>::type *r, const FftDev<T> &f,
                  int ns, cudaStream_t st) {
  if (pass_few<T>(LOGL, ns, sizeof(T) == 4 ? 4 : 1)) return bwd_passes_sized<T, LOGL, PassFew<T, LOGL>::LOGE>(sp, z, r, f, ns, st);
  return bwd_passes_sized<T, LOGL, PassCfg<T>::LOGE>(sp, z, r, f, ns, st);
}

// lengths above the one-CTA limit up to the plans' largest
template <typename T>
int bwd_passes(int logL, const BwdSpec<T> &sp, typename CxOf<T>::type *z, typename CxOf<T>::type *r,
               const FftDev<T> &f, int ns, cudaStream_t st) {
#define CUNA_BWD(LG) \
  case LG: return bwd_passes_at<T, LG>(sp, z, r, f, ns, st);
  if constexpr (sizeof(T) == 4) {
    switch (logL) { CUNA_BWD(15) CUNA_BWD(16) CUNA_BWD(17) CUNA_BWD(18) CUNA_BWD(19) CUNA_BWD(20) CUNA_BWD(21) CUNA_BWD(22) CUNA_BWD(23) CUNA_BWD(24) CUNA_BWD(25) }
  } else {
    switch (logL) { CUNA_BWD(14) CUNA_BWD(15) CUNA_BWD(16) CUNA_BWD(17) CUNA_BWD(18) CUNA_BWD(19) CUNA_BWD(20) CUNA_BWD(21) CUNA_BWD(22) CUNA_BWD(23) }
  }
#undef CUNA_BWD
  return fail(CUNA2_ERROR_UNSUPPORTED, "no backward pass for grids of 2^%d points", logL + 1);
}

template <typename T, int M>
int interp_at(const BwdArgs<T> &a, const BwdCoef<T> &cf, cudaStream_t st) {
  const dim3 grid((unsigned)((a.n + 255) / 256), a.ns);
  CUNA_CK(launch_bwd<T>(k_bwd_interp<T, M>, grid, dim3(256), 0, st, a.t, a.y, a.n, *a.ser, a.ng, cf, (const T *)a.r, a.gy,
                     a.gt));
  return CUNA2_SUCCESS;
}

template <typename T> int interp(const BwdArgs<T> &a, const BwdCoef<T> &cf, cudaStream_t st) {
#define CUNA_BWI(M) \
  case M: return interp_at<T, M>(a, cf, st);
  switch (a.m) { CUNA_BWI(1) CUNA_BWI(2) CUNA_BWI(3) CUNA_BWI(4) CUNA_BWI(5) CUNA_BWI(6) CUNA_BWI(7) CUNA_BWI(8) CUNA_BWI(9) CUNA_BWI(10) CUNA_BWI(11) CUNA_BWI(12) CUNA_BWI(13) CUNA_BWI(14) CUNA_BWI(15) CUNA_BWI(16) }
#undef CUNA_BWI
  return fail(CUNA2_ERROR_UNSUPPORTED, "filter half-width %d", a.m);
}

}  // namespace

template <typename T> int backward_group(const BwdArgs<T> &a, cudaStream_t st) {
  typedef typename CxOf<T>::type C;
  const FftDev<T> f = to_dev<T>(a.g);
  const int L = 1 << a.g.logL;
  BwdSpec<T> sp;
  sp.K = (int)(a.nf / 2);
  sp.L = L;
  sp.G = a.G + sp.K;
  sp.c0b = (T)(1.0 / sqrt(4.0 * kPi * a.tau));
  sp.c1 = (T)(4.0 * kPi * kPi * a.tau / ((double)a.ng * (double)a.ng));
  BwdCoef<T> cf;
  for (int j = 0; j < kBwdCoefs; ++j) {
    cf.c[j] = (T)exp(-(double)(j * j) / (4.0 * a.tau));
    cf.jc[j] = (T)j * cf.c[j];
  }
  cf.k1 = (T)(1.0 / (4.0 * a.tau * log(2.0)));
  cf.inv2tau = (T)2.0 * (T)(1.0 / (4.0 * a.tau));
  if (a.small) {
    static SetupFlag attr;
    if (!setup_done(&attr)) {
      CUNA_CK(cudaFuncSetAttribute(k_bwd_small<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
      mark_setup_done(&attr);
    }
    const size_t smem = sizeof(C) * (size_t)fft_pitch(L, 1);
    // the FFT uses L / 16 threads; the spectrum and the samples more of them
    // where a series has an SM to itself
    const int most = sizeof(T) == 4 ? 1024 : 512;
    const int threads = std::max(std::min(most, L / kFftE), a.ns <= device_sm_count() ? most : 128);
    k_bwd_small<T><<<a.ns, threads, smem, st>>>(a.t, a.y, a.n, *a.ser, cf, sp, a.m, f, a.gy, a.gt);
    CUNA_CK(cudaGetLastError());
    return CUNA2_SUCCESS;
  }
  CUNA_TRY(bwd_passes<T>(a.g.logL, sp, a.z, a.r, f, a.ns, st));
  return interp<T>(a, cf, st);
}

template int backward_group<float>(const BwdArgs<float> &, cudaStream_t);
template int backward_group<double>(const BwdArgs<double> &, cudaStream_t);

}  // namespace cuna
