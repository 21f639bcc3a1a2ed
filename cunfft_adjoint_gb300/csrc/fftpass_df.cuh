// fftpass_df.cuh -- four-step FFT passes of the float64 plan in float-float
// arithmetic (dfl, common.cuh), on the FP32 pipe.
//
// What bounds them is the instruction stream.  A radix-16 butterfly in
// float-float is about 2,700 scalar operations; unrolled with its 16-value
// exchange a pass is 130 KB of straight-line code, which every warp fetches
// once per CTA: 7.4 of 12 stall cycles per instruction were instruction
// fetches (column pass of 2^18 points: 53 us for 3.4 us of issue slots, on 64
// or 256 CTAs alike).  So here:
//  - a thread holds 8 values, one radix-8 butterfly, and the stages of a pass
//    are a loop over one body with run-time shifts (one kernel for every
//    length);
//  - a complex value is two packed pairs, (re.hi, im.hi) and (re.lo, im.lo),
//    and the arithmetic runs on both parts at once (add/mul/fma .f32x2), half
//    the instructions;
//  - between the passes the values stay float-float (the same 16 bytes as a
//    complex double), without the conversions to and from double, which run on
//    the FP64 pipe;
//  - the unpack twiddles come from the FFT's tables, not from FP64 sincospi
//    (L2 + B of them per CTA).
// One transform of 2^21 points: column pass 108 -> 65 us, row pass 125 -> 54 us;
// the whole float64 transform of 1e6 samples 369 -> 275 us.
#pragma once
#include "accurate_kernels.cuh"

namespace cuna {

__device__ __forceinline__ dcx dc_fast(f2 s, f2 e) {  // s + e renormalised, |s| >= |e|
  dcx r;
  r.h = add2(s, e);
  r.l = sub2(e, sub2(r.h, s));
  return r;
}
// sums as dfl's operator+, both parts at once
__device__ __forceinline__ dcx cadd(dcx a, dcx b) {
  const f2 s = add2(a.h, b.h), v = sub2(s, a.h);
  const f2 e = add2(sub2(a.h, sub2(s, v)), sub2(b.h, v));
  return dc_fast(s, add2(e, add2(a.l, b.l)));
}
__device__ __forceinline__ dcx csub(dcx a, dcx b) {
  const f2 s = sub2(a.h, b.h), v = sub2(s, a.h);
  const f2 e = sub2(sub2(a.h, sub2(s, v)), add2(b.h, v));
  return dc_fast(s, add2(e, sub2(a.l, b.l)));
}
// (x, y) -> (-y, x), i times a
__device__ __forceinline__ f2 rot2(f2 a) {
  float x, y;
  unpk2(a, x, y);
  return pk2(-y, x);
}
__device__ __forceinline__ dcx cmuli(dcx a) {
  dcx r;
  r.h = rot2(a.h);
  r.l = rot2(a.l);
  return r;
}
__device__ __forceinline__ dcx cconj(dcx a) {
  dcx r;
  r.h = a.h ^ 0x8000000000000000ull;
  r.l = a.l ^ 0x8000000000000000ull;
  return r;
}
// a times the real (h + l): both parts by the same factor
__device__ __forceinline__ dcx cscale(dcx a, float h, float l) {
  const f2 ph = pk2(h, h), p = mul2(a.h, ph);
  const f2 w = fma2(a.h, neg2(ph), p);  // p - a.h h, exact
  const f2 u = fma2(a.l, ph, mul2(a.h, pk2(l, l)));
  return dc_fast(p, sub2(u, w));
}
// a b: the four partial products' rounding errors (exact by FMA) and low
// parts in one low sum, the two leading products by a two-sum
__device__ __forceinline__ dcx cmul(dcx a, dcx b) {
  float bxh, byh, bxl, byl;
  unpk2(b.h, bxh, byh);
  unpk2(b.l, bxl, byl);
  const f2 xh = pk2(bxh, bxh), yh = pk2(byh, byh), rh = rot2(a.h);  // a b = a b.x + (i a) b.y
  const f2 p = mul2(a.h, xh), q = mul2(rh, yh);
  const f2 w = fma2(a.h, neg2(xh), p), z = fma2(rh, neg2(yh), q);
  f2 u = mul2(a.h, pk2(bxl, bxl));
  u = fma2(a.l, xh, u);
  u = fma2(rh, pk2(byl, byl), u);
  u = fma2(rot2(a.l), yh, u);
  u = sub2(u, add2(w, z));
  const f2 s = add2(p, q), v = sub2(s, p);
  const f2 e = add2(sub2(p, sub2(s, v)), sub2(q, v));
  return dc_fast(s, add2(e, u));
}

__device__ __forceinline__ dcx dc_pack(dfl x, dfl y) {
  dcx r;
  r.h = pk2(x.hi, y.hi);
  r.l = pk2(x.lo, y.lo);
  return r;
}
__device__ __forceinline__ dcx dc_load(double2 v) { return dc_pack(df_from_double(v.x), df_from_double(v.y)); }
__device__ __forceinline__ double2 dc_to_double(dcx a) {
  float xh, yh, xl, yl;
  unpk2(a.h, xh, yh);
  unpk2(a.l, xl, yl);
  return make_double2((double)xh + (double)xl, (double)yh + (double)yl);
}
__device__ __forceinline__ dcx ldtw(const dcx *p) {
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(p));
  dcx r;
  r.h = v.x;
  r.l = v.y;
  return r;
}
__device__ __forceinline__ dcx dc_ldcg(const dcx *p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2 *>(p));
  dcx r;
  r.h = v.x;
  r.l = v.y;
  return r;
}

namespace {

__device__ __forceinline__ void df_bf4(dcx &a0, dcx &a1, dcx &a2, dcx &a3) {
  const dcx t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = cmuli(csub(a1, a3));
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cadd(t1, t3);
  a3 = csub(t1, t3);
}
__device__ __forceinline__ void df_dft8(dcx *v) {
  constexpr float ch = 0.70710678118654752440, cl = 0.70710678118654752440 - (double)ch;
  dcx e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  dcx o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  df_bf4(e0, e1, e2, e3);
  df_bf4(o0, o1, o2, o3);
  const dcx i1 = cmuli(o1), i3 = cmuli(o3);
  const dcx t1 = cscale(cadd(o1, i1), ch, cl);  // W8^1 o1
  const dcx t2 = cmuli(o2);                     // W8^2 o2
  const dcx t3 = cscale(csub(i3, o3), ch, cl);  // W8^3 o3
  v[0] = cadd(e0, o0); v[4] = csub(e0, o0);
  v[1] = cadd(e1, t1); v[5] = csub(e1, t1);
  v[2] = cadd(e2, t2); v[6] = csub(e2, t2);
  v[3] = cadd(e3, t3); v[7] = csub(e3, t3);
}

// Shared index of point i of a sequence: one 16-byte element of padding per
// eight, so that the strided stores of the first stages spread over the banks.
__device__ __forceinline__ int df_pad(int i) { return i + (i >> 3); }
// Pitch (elements) of sequences of length L stored side by side: congruent to
// 8 / nseq mod 8, so that lanes that take consecutive sequences do too.
__host__ __device__ __forceinline__ int df_pitch(int L, int nseq) {
  const int base = L + (L >> 3) + 1, want = nseq >= 8 ? 1 : 8 / nseq;
  return base + ((want - base) & 7);
}

// Inverse FFT of the CTA's 2^logB sequences of length 2^logL, 8 values per
// thread, from src.load(seq, i) to shared memory s[seq pitch + df_pad(k)],
// followed by a barrier.  One leading stage of radix 2, 4 or 8, then radix 8.
// SEQ_FAST: consecutive threads take consecutive sequences, else points.
template <bool SEQ_FAST, class Src>
__device__ __forceinline__ void df_fft(dcx *s, int pitch, int logL, int logB, const dcx *__restrict__ tw,
                                       const Src &src) {
  const int r0 = logL % 3 == 0 ? 3 : logL % 3;
  dcx v[8];
  {
    const int sh = logL - r0, nthr = blockDim.x;
    // 8 >> r0 butterflies of radix 2^r0 per thread; value (u, r) in v[u 2^r0 + r]
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int u = q >> r0, r = q & ((1 << r0) - 1), g = threadIdx.x + u * nthr;
      const int seq = SEQ_FAST ? g & ((1 << logB) - 1) : g >> sh, j = SEQ_FAST ? g >> logB : g & ((1 << sh) - 1);
      v[q] = src.load(seq, j + (r << sh));
    }
    if (r0 == 3) {
      df_dft8(v);
    } else if (r0 == 2) {
      df_bf4(v[0], v[1], v[2], v[3]);
      df_bf4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        const dcx a = v[q];
        v[q] = cadd(a, v[q + 1]);
        v[q + 1] = csub(a, v[q + 1]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int u = q >> r0, r = q & ((1 << r0) - 1), g = threadIdx.x + u * nthr;
      const int seq = SEQ_FAST ? g & ((1 << logB) - 1) : g >> sh, j = SEQ_FAST ? g >> logB : g & ((1 << sh) - 1);
      s[seq * pitch + df_pad((j << r0) + r)] = v[q];
    }
  }
  __syncthreads();
  const int sh = logL - 3, g = threadIdx.x;
  const int seq = SEQ_FAST ? g & ((1 << logB) - 1) : g >> sh, j = SEQ_FAST ? g >> logB : g & ((1 << sh) - 1);
  dcx *b = s + seq * pitch;
#pragma unroll 1
  for (int ns = r0; ns < logL; ns += 3) {
    const int k = j & ((1 << ns) - 1), step = k << (sh - ns);
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = b[df_pad(j + (r << sh))];
#pragma unroll
    for (int r = 1; r < 8; ++r) v[r] = cmul(v[r], ldtw(tw + r * step));
    df_dft8(v);
    __syncthreads();
    const int d = ((j >> ns) << (ns + 3)) + k;
#pragma unroll
    for (int r = 0; r < 8; ++r) b[df_pad(d + (r << ns))] = v[r];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// column pass: FFTs down the columns [c0, c0 + 2^logB) of the L1 x L2 grid
// (complex double), times W_L^{c k}, stored in place in float-float.
// ---------------------------------------------------------------------------
struct DfColSrc {
  const double2 *p;  // slab + c0
  int logL2;
  bool df;  // the gridding wrote float-float (tile_flush_df), else double
  __device__ __forceinline__ dcx load(int seq, int i) const {
    // through L2: the gridding may still have been writing when this kernel started
    const double2 *q = p + ((int64_t)i << logL2) + seq;
    return df ? dc_ldcg(reinterpret_cast<const dcx *>(q)) : dc_load(__ldcg(q));
  }
};

__global__ void __launch_bounds__(1024, 1) k_df_colpass(double2 *grid, FftDev<dfl> f, int logB, bool df_in) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dcx *s = reinterpret_cast<dcx *>(smem_raw);
  const int L1 = 1 << f.logL1, B = 1 << logB, pitch = df_pitch(L1, B);
  dcx *steps = s + pitch * B;  // steps[8 seq + e] = W_L^{c e L1 / 8}
  const int c0 = blockIdx.x << logB;
  double2 *z = grid + ((int64_t)blockIdx.y << f.logL) + c0;
  pdl_trigger();
  for (int i = threadIdx.x; i < 8 * B; i += blockDim.x)
    steps[i] = twiddle_L(f, (c0 + (i >> 3)) * ((i & 7) << (f.logL1 - 3)));
  pdl_wait();  // the grid comes from the gridding
  // every read precedes the first barrier, every write follows it: in place is safe
  df_fft<true>(s, pitch, f.logL1, logB, f.tw1, DfColSrc{z, f.logL2, df_in});
  const int seq = threadIdx.x & (B - 1), k0 = threadIdx.x >> logB;
  const dcx w0 = twiddle_L(f, (c0 + seq) * k0);
  ulonglong2 *out = reinterpret_cast<ulonglong2 *>(z) + seq;
#pragma unroll 2
  for (int e = 0; e < 8; ++e) {
    const int k = k0 + (e << (f.logL1 - 3));
    const dcx w = cmul(s[seq * pitch + df_pad(k)], cmul(w0, steps[8 * seq + e]));
    out[(int64_t)k << f.logL2] = make_ulonglong2(w.h, w.l);
  }
}

// ---------------------------------------------------------------------------
// row pass with the accurate epilogue, as ct_rowpass_body (fftpass.cuh): row
// pairs (p, L1 - p), rows 0 and L1/2 in slot 0; sequence half P + i holds
// slot p0 + i's first (half 0) or second row.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int df_pair_row(int logL1, int p, int half) {
  return half ? (p == 0 ? 1 << (logL1 - 1) : (1 << logL1) - p) : p;
}
struct DfPairSrc {
  const dcx *p;  // slab
  int logL1, logL2, logP, p0;
  __device__ __forceinline__ dcx load(int seq, int i) const {
    const int row = df_pair_row(logL1, p0 + (seq & ((1 << logP) - 1)), seq >> logP);
    return dc_ldcg(p + ((int64_t)row << logL2) + i);  // through L2, as the column pass's reads
  }
};

__global__ void __launch_bounds__(1024, 1) k_df_rowpass_acc(const dcx *grid, FftDev<dfl> f, AccParams<double> e,
                                                            double2 *F, int logB) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dcx *s = reinterpret_cast<dcx *>(smem_raw);
  const int logL1 = f.logL1, logL2 = f.logL2, L2 = 1 << logL2;
  const int B = 1 << logB, logP = logB - 1, P = B >> 1, pitch = df_pitch(L2, B);
  const int p0 = blockIdx.x << logP;
  // unpack twiddle of k = k1 + L1 k2: exp(pi i k / L) = exp(2 pi i (k2 / 2) / L2)
  // (the row FFT's table) times exp(pi i (k1 + L1 (k2 mod 2)) / L)
  dcx *twr = s + pitch * B;
  pdl_trigger();
  for (int u = threadIdx.x; u < 2 * B; u += blockDim.x) {
    const int row = u >> 1;
    const int q = df_pair_row(logL1, p0 + (row & (P - 1)), row >> logP) + ((u & 1) << logL1);
    double sn, cs;
    sincospi((double)q * e.twk, &sn, &cs);
    twr[u] = dc_pack(dfl(cs), dfl(sn));
  }
  pdl_wait();  // the rows come from the column pass
  df_fft<false>(s, pitch, logL2, logB, f.tw2, DfPairSrc{grid + ((int64_t)blockIdx.y << f.logL), logL1, logL2, logP, p0});
  F += (int64_t)blockIdx.y * e.nf;
  const dfl c0 = dfl(e.c0), c1 = dfl(e.c1 * 1.4426950408889634);
  const int K = (int)e.K;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < (B << logL2); idx += blockDim.x) {
    const int i = idx & (P - 1), half = (idx >> logP) & 1, k2 = idx >> logB;
    const int p = p0 + i, seq = half * P + i;
    const int k1 = df_pair_row(logL1, p, half);
    const int k = k1 + (k2 << logL1);
    if (k > K) continue;
    const int k2m = k1 == 0 ? ((L2 - k2) & (L2 - 1)) : (L2 - 1 - k2);
    const int seqm = p == 0 ? seq : (1 - half) * P + i;
    const dcx Zk = s[seq * pitch + df_pad(k2)], Zm = cconj(s[seqm * pitch + df_pad(k2m)]);
    const dcx tw = cmul(ldtw(f.tw2 + (k2 >> 1)), twr[2 * seq + (k2 & 1)]);
    const dcx G2 = cadd(cadd(Zk, Zm), cmul(cmuli(csub(Zm, Zk)), tw));
    const dfl kf((float)k, 0.f);  // k <= nf / 2 <= 2^24: exact
    dfl sc = c0 * df_exp2(c1 * kf * kf);
    if (k & 1) sc = -sc;
    const double2 Fk = dc_to_double(cscale(G2, sc.hi, sc.lo));
    if (k < K) F[K + k] = Fk;
    if (k >= 1) F[K - k] = make_double2(Fk.x, -Fk.y);
  }
}

// elements per CTA (log2): 4096, fewer where that leaves SMs idle, at least
// two sequences (a row pair; columns of whole 32-byte sectors)
inline int df_log_elems(int logL, int logLseq, int nslab) {
  int le = 12;
  while (le > 10 && ((int64_t)nslab << logL >> le) < 2 * device_sm_count()) --le;
  return std::max(le, logLseq + 1);
}

// Both passes of nslab packed grids of 2^f.logL points at z; 0 on success
inline int df_colpass(double2 *z, const FftDev<dfl> &f, int nslab, bool df_in, cudaStream_t st) {
  const int le = df_log_elems(f.logL, f.logL1, nslab), logB = le - f.logL1;
  const size_t sm = sizeof(dcx) * ((size_t)df_pitch(1 << f.logL1, 1 << logB) + 8) << logB;
  static SetupFlag attr;
  if (!setup_done(&attr)) {
    CUNA_CK(cudaFuncSetAttribute(k_df_colpass, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    CUNA_CK(cudaFuncSetAttribute(k_df_rowpass_acc, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    mark_setup_done(&attr);
  }
  CUNA_CK(launch_pdl(k_df_colpass, dim3(1 << (f.logL2 - logB), nslab), dim3(1 << (le - 3)), sm, st, z, f, logB, df_in));
  return CUNA2_SUCCESS;
}
inline int df_rowpass(const double2 *z, const FftDev<dfl> &f, const AccParams<double> &e, double2 *F, int nslab,
                      cudaStream_t st) {
  const int le = df_log_elems(f.logL, f.logL2, nslab), logB = le - f.logL2;
  const size_t sm = sizeof(dcx) * ((size_t)df_pitch(1 << f.logL2, 1 << logB) + 2) << logB;
  CUNA_CK(launch_pdl(k_df_rowpass_acc, dim3(1 << (f.logL1 - logB), nslab), dim3(1 << (le - 3)), sm, st,
                     reinterpret_cast<const dcx *>(z), f, e, F, logB));
  return CUNA2_SUCCESS;
}

}  // namespace
}  // namespace cuna
