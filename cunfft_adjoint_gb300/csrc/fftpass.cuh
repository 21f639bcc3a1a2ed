// fftpass.cuh -- the accurate transform's four-step row pass (real unpack,
// deconvolution and centring fused in) with compile-time geometry; the
// stages and the column pass are in fftpass_core.cuh.
#pragma once
#include "accurate_kernels.cuh"
#include "fftpass_core.cuh"

namespace cuna {
namespace {

// ---------------------------------------------------------------------------
// row pass with the accurate epilogue: a CTA owns the row-pair slots
// p in [p0, p0 + B/2), transforms their rows (length L2) into shared memory,
// then unpacks, deconvolves and centres every output k = k1 + L1 k2 <= K.
// Slot p >= 1 holds rows (p, L1 - p), whose outputs need each other's
// values; rows 0 and L1/2 each pair with themselves and share slot 0, so
// there are exactly L1/2 slots and every CTA's slots are all used.
// ---------------------------------------------------------------------------
template <int LOG1> __host__ __device__ constexpr int ct_pair_row(int p, int half) {
  return half ? (p == 0 ? (1 << LOG1) / 2 : (1 << LOG1) - p) : p;
}

// Sequence seq of the CTA's buffer holds row ct_pair_row(p0 + i, half) with
// seq = half P + i (first rows k1 of the CTA's slots, then their partners), so
// that the epilogue's lanes, which take consecutive slots i, read rows one
// odd pitch apart: conflict-free 8-byte shared loads.
template <typename T, int LOG1, int LOG2, int LOGP> struct CtPairSrc {
  const typename CxOf<T>::type *p;  // slab
  int p0;
  __device__ __forceinline__ typename CxOf<T>::type load(int seq, int j, int dr) const {
    // through L2: the column pass may still have been writing when this kernel started
    return __ldcg(p + (ct_pair_row<LOG1>(p0 + (seq & ((1 << LOGP) - 1)), seq >> LOGP) << LOG2) + j + dr);
  }
};

struct CtNoDst {
  template <int R, int LOGNS, typename C> __device__ void store(int, int, C *) const {}
};

// Outputs of the CTA's transformed rows in s: the real unpack, deconvolution and
// centring of every k = k1 + L1 k2 <= K, to Fs[0 .. nf).
// A thread keeps one row (the CTA's threads are a multiple of its 2P = B
// rows) and steps through its outputs k = k1 + L1 k2 <= K: the row's indices,
// twiddle and partner are formed once, and the columns beyond K cost nothing
// (the pass is near its instruction issue, 94 per point; with half the outputs
// skipped in a 16-step loop the bootstrap of 1024 x 2^15 points took 332 us,
// 325 here).
template <typename T, int LOG1, int LOG2, int LOGB, int THREADS>
__device__ __forceinline__ void rowpass_outputs(const typename CxOf<T>::type *s, const typename CxOf<T>::type *twr,
                                                const typename CxOf<T>::type *twc, int p0, const AccParams<T> &e,
                                                typename CxOf<T>::type *Fs) {
  typedef typename CxOf<T>::type C;
  constexpr int L2 = 1 << LOG2, LOGP = LOGB - 1, P = 1 << LOGP, PITCH = fft_pitch(L2, 1 << LOGB);
  const int i = threadIdx.x & (P - 1), half = (threadIdx.x >> LOGP) & 1;
  const int p = p0 + i, k1 = ct_pair_row<LOG1>(p, half);
  // Z[L - k] is in row (L1 - k1) mod L1: the slot's other row, or the same row
  // for the self-paired rows 0 and L1/2 of slot 0
  const C *zk = s + (half * P + i) * PITCH, *zm = s + (p == 0 ? half * P + i : (1 - half) * P + i) * PITCH;
  const C tw1 = twr[2 * i + half];
  const int mlast = k1 == 0 ? L2 : L2 - 1, K = (int)e.K;
  const T c0 = e.c0, c1 = e.c1 * (T)1.4426950408889634;
  C *Fp = Fs + K, *Fn = Fs + K;
#pragma unroll 4
  for (int k2 = threadIdx.x >> LOGB; k2 <= (K - k1) >> LOG1; k2 += THREADS >> LOGB) {
    const int k = k1 + (k2 << LOG1), k2m = (mlast - k2) & (L2 - 1);
    const C Zk = zk[cpad16(k2)], Zm = cconj(zm[cpad16(k2m)]);
    // real unpack, deconvolution c0 exp2(c1 k^2) with the (-1)^k of the origin
    const C G2 = cadd(cadd(Zk, Zm), cmul(cmul(tw1, twc[k2]), cmuli(csub(Zm, Zk))));
    const T kf = (T)k;
    const T sc = c0 * exp2_g(c1 * kf * kf);
    const C Fk = cscale(G2, (k & 1) ? -sc : sc);
    if (k < K) Fp[k] = Fk;
    if (k >= 1) Fn[-k] = cconj(Fk);
  }
}

// row-pair block `pblock` of one packed grid z; outputs Fs[0 .. nf)
template <typename T, int LOGL, int LOGE = PassCfg<T>::LOGE>
__device__ __forceinline__ void ct_rowpass_body(const typename CxOf<T>::type *slab, const FftDev<T> &f,
                                                const AccParams<T> &e,
                                                typename CxOf<T>::type *Fs, int pblock) {
  typedef typename CxOf<T>::type C;
  constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2;
  constexpr int L2 = 1 << LOG2;
  constexpr int LOGB = LOGE - LOG2;
  constexpr int B = 1 << LOGB, LOGP = LOGB - 1, P = B >> 1;
  constexpr int PITCH = fft_pitch(L2, B);
  constexpr int THREADS = 1 << (LOGE - 4);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *s = reinterpret_cast<C *>(smem_raw);
  // unpack twiddles W_ng^k = W_ng^{k1} W_ng^{k2 L1} from two small tables
  // behind the FFT buffer: the CTA's 2P rows and all L2 columns
  C *twr = s + PITCH * B, *twc = twr + B;
  const int p0 = pblock * P;
  pdl_trigger();
  for (int u = threadIdx.x; u < B + L2; u += THREADS) {
    const int q = u < B ? ct_pair_row<LOG1>(p0 + (u >> 1), u & 1) : (u - B) << LOG1;
    T sn, cs;
    sincospi_t((T)q * e.twk, &sn, &cs);
    twr[u] = cmk(cs, sn);  // twr[B + k2] is twc[k2]
  }
  pdl_wait();  // the rows come from the column pass
  CtPairSrc<T, LOG1, LOG2, LOGP> src{slab, p0};
  ct_fft<T, LOG2, LOGB, false, false, false>(s, f.tw2, src, CtNoDst());
  rowpass_outputs<T, LOG1, LOG2, LOGB, THREADS>(s, twr, twc, p0, e, Fs);
}

// three CTAs per SM for the short rows of many small grids (bootstrap), where
// the pass streams from HBM and more bytes in flight pay
template <typename T, int LOGL, int LOGE> constexpr int ct_rowpass_min_ctas() {
  return LOGE < PassCfg<T>::LOGE ? 1 : ((sizeof(T) == 4 && LOGL <= 15) ? 3 : 2);
}
template <typename T, int LOGL, int LOGE = PassCfg<T>::LOGE>
__global__ void __launch_bounds__(1 << (LOGE - 4), ct_rowpass_min_ctas<T, LOGL, LOGE>()) k_ct_rowpass_acc(
    const typename CxOf<T>::type *grid, FftDev<T> f, AccParams<T> e,
    typename CxOf<T>::type *F) {
  ct_rowpass_body<T, LOGL, LOGE>(grid + ((int64_t)blockIdx.y << LOGL), f, e, F + (int64_t)blockIdx.y * e.nf,
                                 blockIdx.x);
}

// CTAs per packed grid of the row pass: L1/2 slots, B/2 per CTA
template <typename T, int LOGL, int LOGE = PassCfg<T>::LOGE> constexpr int ct_rowpass_ctas() {
  return ((1 << ((LOGL + 1) / 2)) / 2) / ((1 << (LOGE - LOGL / 2)) / 2);
}

template <typename T, int LOGL, int LOGE = PassCfg<T>::LOGE> constexpr size_t ct_rowpass_smem() {
  constexpr int LOG2 = LOGL / 2;
  constexpr int B = 1 << (LOGE - LOG2);
  return sizeof(typename CxOf<T>::type) * ((size_t)fft_pitch(1 << LOG2, B) * B + B + (1 << LOG2));
}

}  // namespace
}  // namespace cuna
