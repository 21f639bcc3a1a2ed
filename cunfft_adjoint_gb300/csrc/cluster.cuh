// cluster.cuh -- a whole float transform of up to 2^15 packed points in one
// launch, by a cluster of eight CTAs whose shared memory holds the grid.
//
// A short transform on the tiled path is a chain of four launches of a few CTAs
// each, and their gaps and the host's enqueue are most of its time (n = 10000,
// Nf = 16384: 17.5 us per call).  Here the steps are phases of one kernel between
// cluster barriers:
//   1. each CTA takes an eighth of the samples and sends each one's record to
//      the shared-memory list of the CTA whose run of ng/8 cells it touches
//      (with the halo, one or two), at a slot from an atomic on the owner's
//      counter, one per run and warp;
//   2. each CTA counting-sorts its list by group of four cells and gathers four
//      cells per thread into its shared tile, as small_gather4;
//   3. column FFTs: the CTA's L2/8 columns are read from the eight tiles through
//      distributed shared memory and, twiddled, written to the CTAs that own
//      their row pairs;
//   4. row FFTs, unpack, deconvolution and centring, as ct_rowpass_body.
// Grids of less than 2^13 points run phases 1 and 2 alike and leave the FFT to
// the first CTA.  n = 10000, Nf = 16384: 17.5 -> 13.0 us per call; with the
// records exchanged through device memory instead, after an exchange of counts,
// 16.5.
// What bounds it is the latency of its phases: the samples' loads and the
// remote atomics 6 of about 20 thousand cycles, sort and gather 7, the FFT
// passes with their remote accesses and the barriers the rest.
#pragma once
#include "accurate_kernels.cuh"
#include "fftpass.cuh"

namespace cuna {
namespace {

constexpr int kClusterLo = 13, kClusterHi = 15;  // log2 of the packed length, FFT over the cluster
constexpr int kClusterN = 16384;
constexpr int kClusterCtas = 8, kClusterThreads = 512;
constexpr int kClusterItems = kClusterN / kClusterCtas / kClusterThreads;  // samples per thread
// Records of a list.  Where a run gets more, the samples are sent in rounds of
// one per thread, which fit whatever their times.
constexpr int kClusterCap = kClusterCtas * kClusterThreads;
constexpr int kClusterSlack = 64;  // places after the sorted list that a gather may read

// Grids of less than 2^kClusterLo points: the first CTA transforms the whole
// grid.  (2^12 points over the cluster take 2 us less, but its four-step FFT has
// two more rounded products per point than the one-CTA FFT: 1.76e-7 of the
// spectrum of n = 300, Nf = 2048, R = 4 against 1.38e-7.)
constexpr int kClusterSmallN = 700, kClusterSmallN12 = 500;

// a record touches at most two runs of ng/8 cells
inline bool cluster_fits(int logL, int m) { return logL <= kClusterHi && logL >= 4 && (1 << (logL - 2)) >= 2 * m; }
// Measured against the other paths (us; n samples, 2^L packed points).  Below
// 2^13 points one CTA does it all in less while the samples are few, on the
// device, one CTA and here: R = 2, 2^9 points: n = 600 7.9 and 7.8, 700 8.3 and
// 7.9; 2^11: 700 8.4 and 8.7, 900 8.8 and 8.8; 2^12: 400 11.0 and 11.1, 600 11.3
// and 11.3, 1000 12.0 and 11.4; R = 4 (dearer weights), 2^10: 300 7.3 and 7.9,
// 500 7.9 and 8.1; 2^11: 300 8.8 and 8.6, 500 9.5 and 8.7; 2^12: 200 11.3 and
// 10.9.  Above, the tiled path, per call: n = 10000, 2^14: 17.5 against 13.0
// here; 2^15: n = 8000 17.8 against 16.4, n = 16384 17.5 against 18.5; 2^16: n =
// 2000 17.5 against 18.5 -- eight SMs are too few for the cells and samples
// from there on.
inline bool cluster_takes(int logL, int R, int64_t n, int nslab) {
  if (n > kClusterN || nslab * kClusterCtas > device_sm_count()) return false;
  if (logL >= kClusterLo) return (n << logL) <= (1 << 28);
  return n > (logL == kClusterLo - 1 ? kClusterSmallN12 : kClusterSmallN) >> (R >= 4);
}

template <int LOGL> struct ClusterCfg {
  static constexpr int LOG1 = (LOGL + 1) / 2, LOG2 = LOGL / 2, L1 = 1 << LOG1, L2 = 1 << LOG2;
  static constexpr int LOGE = LOGL - 3;                     // packed points per CTA
  static constexpr int FT = 1 << (LOGE - 4);                // threads of the FFTs
  static constexpr int LOGB1 = LOGE - LOG1, B1 = 1 << LOGB1;  // columns per CTA
  static constexpr int LOGB2 = LOGE - LOG2, B2 = 1 << LOGB2;  // rows per CTA
  static constexpr int TC = 2 << LOGE;                      // cells per CTA
  static constexpr int PITCH1 = fft_pitch(L1, B1), PITCH2 = fft_pitch(L2, B2);
  static constexpr int MAXM = 16;
  static constexpr size_t fft_bytes = 8 * (size_t)(PITCH1 * B1 > PITCH2 * B2 ? PITCH1 * B1 : PITCH2 * B2);
  static constexpr size_t sort_bytes =
      sizeof(SRec<float>) * (2 * kClusterCap + kClusterSlack) + sizeof(int) * ((TC + 2 * MAXM) / 4 + 4);
  static constexpr size_t rows_bytes = 8 * ((size_t)1 << LOGE);
  static constexpr size_t work_bytes =
      ((rows_bytes + fft_bytes > sort_bytes ? rows_bytes + fft_bytes : sort_bytes) + 15) & ~(size_t)15;
  // tile | list, sorted list and group starts, or rows and FFT buffer | steps | row and column unpack twiddles
  static constexpr size_t smem = sizeof(float) * TC + work_bytes + 8 * (17 * B1 + B2 + L2);
};

// address in CTA `rank`'s shared memory of this CTA's shared address p
__device__ __forceinline__ unsigned cluster_addr(const void *p, int rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

// columns of the grid from the eight tiles
template <int LOG1, int LOG2> struct ClusterColSrc {
  const float2 *tile;  // this CTA's tile: L1/8 rows of L2
  int c0;
  __device__ __forceinline__ float2 load(int seq, int j, int dr) const {
    const int i = j + dr;
    const unsigned a = cluster_addr(tile + ((i & ((1 << (LOG1 - 3)) - 1)) << LOG2) + c0 + seq, i >> (LOG1 - 3));
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
    return v;
  }
};
// twiddled columns to the owners of the rows (slot p: rows p and L1 - p; rows 0
// and L1/2 in slot 0; sequence half P + p of the owner's buffer)
template <int LOG1, int LOG2> struct ClusterColDst {
  float2 *rows;
  const float2 *steps;
  FftDev<float> f;
  int c0;
  template <int R, int LOGNS> __device__ __forceinline__ void store(int seq, int idxD, float2 *v) const {
    static_assert(R == 16 || LOGNS == 0, "the storing stage is radix 16 or the only stage");
    constexpr int L1 = 1 << LOG1, LOGP = LOG1 - 4;  // L1/16 slots per CTA
    const float2 w0 = twiddle_L(f, (c0 + seq) * idxD);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = idxD + (r << LOGNS);
      const float2 w = r == 0 ? w0 : cmul(w0, steps[seq * 17 + r]);
      const float2 x = cmul(v[r], w);
      const int half = k >= L1 / 2 ? 1 : 0, p = half ? (L1 - k) & (L1 / 2 - 1) : k;
      const unsigned a =
          cluster_addr(rows + (((half << LOGP) + (p & ((1 << LOGP) - 1))) << LOG2) + c0 + seq, p >> LOGP);
      asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x.x), "f"(x.y) : "memory");
    }
  }
};
template <int LOG2> struct ClusterRowSrc {
  const float2 *rows;
  __device__ __forceinline__ float2 load(int seq, int j, int dr) const { return rows[(seq << LOG2) + j + dr]; }
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// the records of items [IT0, IT1) of a thread to the lists of the runs they
// touch; slots beyond the list's end are counted, not written
template <int IT0, int IT1>
__device__ __forceinline__ void cluster_send(int LOGTC, const int *cell, const float *f, const float *y, const bool *on,
                                             int m, int gmask, int *count, SRec<float> *list) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned same[IT1 - IT0];
  int slot[IT1 - IT0], run[IT1 - IT0];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    bool any = q == 0;
#pragma unroll
    for (int it = IT0; it < IT1; ++it) {
      const int lo = ((cell[it] - m + 1) & gmask) >> LOGTC, hi = ((cell[it] + m) & gmask) >> LOGTC;
      run[it - IT0] = !on[it] ? -1 : (q == 0 ? lo : (hi == lo ? -1 : hi));
      any |= run[it - IT0] >= 0;
    }
    if (q == 1 && !__any_sync(full, any)) break;
#pragma unroll
    for (int k = 0; k < IT1 - IT0; ++k) {
      same[k] = __match_any_sync(full, run[k]);
      slot[k] = 0;
      if (run[k] >= 0 && lane == __ffs(same[k]) - 1)
        asm volatile("atom.shared::cluster.add.u32 %0, [%1], %2;"
                     : "=r"(slot[k]) : "r"(cluster_addr(count, run[k])), "r"(__popc(same[k])) : "memory");
    }
#pragma unroll
    for (int k = 0; k < IT1 - IT0; ++k) {
      const int s = __shfl_sync(full, slot[k], __ffs(same[k]) - 1) + __popc(same[k] & ((1u << lane) - 1));
      const int lc = (cell[IT0 + k] - (run[k] << LOGTC) + m) & gmask;  // local cell + m
      if (run[k] >= 0 && s < kClusterCap)
        asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %3};" ::"r"(cluster_addr(list + s, run[k])),
                     "r"(__float_as_int(f[IT0 + k])), "r"(__float_as_int(y[IT0 + k])), "r"(lc) : "memory");
    }
  }
}

// list[0, c) sorted by group of four cells, and the sums of the run's TC cells
// into the tile (onto it unless first).  start: zeroed, NG + 1 group counts.
// Where there are fewer groups than threads, 2^LP threads share a group's
// records.  ONE >= 0: weights one by one, in that form (gauss_acc4).
template <bool MASKED, int ONE>
__device__ __forceinline__ void cluster_gather(int TC, const SRec<float> *list, SRec<float> *sorted, int *start, int c,
                                               int m, float k1, float *tile, bool first) {
  constexpr int TH = kClusterThreads, PER = kClusterCap / TH;
  const int NG = (TC + 2 * m + 3) / 4;
  int rank[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * TH;
    if (i < c) rank[k] = atomicAdd(&start[list[i].lc >> 2], 1);
  }
  __syncthreads();
  cta_scan_in_place(start, NG);
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * TH;
    if (i < c) {
      const SRec<float> r = list[i];
      sorted[start[r.lc >> 2] + rank[k]] = r;
    }
  }
  __syncthreads();
  const GaussCW<float, 4> gw(k1);
  int LP = 0;
  while (LP < 5 && (TC / 4 << LP) < TH) ++LP;
  const int part = threadIdx.x & ((1 << LP) - 1), step = 1 << LP;
  for (int g = threadIdx.x >> LP; g < TC / 4; g += TH >> LP) {
    const int cl0 = 4 * g, re = start[(cl0 + 2 * m + 2) / 4 + 1];
    float a[4] = {0.f, 0.f, 0.f, 0.f};
    int r = start[g] + part;
    SRec<float> q = sorted[r];  // up to 2 step - 1 beyond the last record, in the array
    // sums of up to 32 records: a thousand samples in a few cells lose to one
    // long sum (10000 in 60 cells: 8e-7 of the spectrum, 3e-7 here; 0.2 us of a
    // transform of 10000 uniform ones)
    while (r < re) {
      const int rs = min(re, r + 32 * step);
      float b[4] = {0.f, 0.f, 0.f, 0.f};
      for (; r < rs; r += step) {
        const SRec<float> nx = sorted[r + step];
        const int rel = q.lc - cl0;
        if constexpr (ONE >= 0) gauss_acc4<ONE>(q.y, m - rel, q.f, k1, m, b);
        else gauss_acc<float, 4, MASKED>(q.y, (float)(m - rel) - q.f, k1, gw, rel, 2 * m, b);
        q = nx;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] += b[i];
    }
    for (int o = 1; o < step; o <<= 1) {  // a group's threads are in one warp
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] += __shfl_xor_sync(0xffffffffu, a[i], o);
    }
    if (part == 0) {
      float4 *o = reinterpret_cast<float4 *>(tile + cl0);
      float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *o;
      *o = make_float4(v.x + a[0], v.y + a[1], v.z + a[2], v.w + a[3]);
    }
  }
}

// Phases 1 and 2: this CTA's run of TC = 2^LOGTC cells of the grid of n samples
// into its tile.  tables() runs while the records travel.  Ends without a
// barrier.
template <bool MASKED, int ONE, class Tables>
__device__ __forceinline__ void cluster_grid(int LOGTC, const double *__restrict__ t, const float *__restrict__ y, int n,
                                             const PhaseMul &pm, const AccParams<float> &e, float *tile,
                                             unsigned char *work, const Tables &tables) {
  constexpr int TH = kClusterThreads, NC = kClusterCtas;
  __shared__ int count;  // records sent to this CTA
  SRec<float> *list = reinterpret_cast<SRec<float> *>(work), *sorted = list + kClusterCap;
  int *start = reinterpret_cast<int *>(sorted + kClusterCap + kClusterSlack);
  const int TC = 1 << LOGTC, m = e.m, NG = (TC + 2 * m + 3) / 4, gmask = NC * TC - 1;
  if (threadIdx.x == 0) count = 0;
  cluster_arrive();  // the counter is ready for the others
  const int per = (n + NC - 1) / NC, i0 = blockIdx.x * per, i1 = min(n, i0 + per);
  int cell[kClusterItems];
  float fr[kClusterItems], yv[kClusterItems];
  bool on[kClusterItems];
  {
    double tv[kClusterItems];
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it) {
      const int i = i0 + it * TH + threadIdx.x;
      on[it] = i < i1;
      tv[it] = on[it] ? t[i] : 0.0;
      yv[it] = on[it] ? y[i] : 0.f;
    }
    for (int i = threadIdx.x; i <= NG; i += TH) start[i] = 0;
#pragma unroll
    for (int it = 0; it < kClusterItems; ++it) reduce_sample<float>(tv[it], pm, e.ng, cell[it], fr[it]);
  }
  cluster_wait();
  cluster_send<0, kClusterItems>(LOGTC, cell, fr, yv, on, m, gmask, &count, list);
  cluster_arrive();
  tables();
  cluster_wait();
  const int over = threadIdx.x < NC ? cluster_load(&count, threadIdx.x) > kClusterCap : 0;
  if (!__syncthreads_or(over)) {
    cluster_gather<MASKED, ONE>(TC, list, sorted, start, count, m, e.k1, tile, true);
  } else {
    auto round = [&](auto it) {
      constexpr int IT = decltype(it)::value;
      cluster_barrier();  // all have read the counters, or gathered the last round
      if (threadIdx.x == 0) count = 0;
      for (int i = threadIdx.x; i <= NG; i += TH) start[i] = 0;
      cluster_barrier();
      cluster_send<IT, IT + 1>(LOGTC, cell, fr, yv, on, m, gmask, &count, list);
      cluster_barrier();
      cluster_gather<MASKED, ONE>(TC, list, sorted, start, count, m, e.k1, tile, IT == 0);
    };
    static_assert(kClusterItems == 4, "rounds");
    round(std::integral_constant<int, 0>());
    round(std::integral_constant<int, 1>());
    round(std::integral_constant<int, 2>());
    round(std::integral_constant<int, 3>());
  }
}

template <int LOGL, bool MASKED>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_nfft_cluster(const double *__restrict__ t, const float *__restrict__ y, int n, PhaseMul pm, AccParams<float> e,
                   FftDev<float> f, float2 *F) {
  typedef ClusterCfg<LOGL> G;
  constexpr int LOG1 = G::LOG1, LOG2 = G::LOG2, TH = kClusterThreads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float *tile = reinterpret_cast<float *>(smem_raw);
  unsigned char *work = reinterpret_cast<unsigned char *>(tile + G::TC);
  float2 *rows = reinterpret_cast<float2 *>(work);
  float2 *s = reinterpret_cast<float2 *>(work + G::rows_bytes);
  float2 *steps = reinterpret_cast<float2 *>(work + G::work_bytes);
  float2 *twr = steps + 17 * G::B1, *twc = twr + G::B2;
  const int rank = blockIdx.x;
  y += (int64_t)blockIdx.y * n;
  F += (int64_t)blockIdx.y * e.nf;
  constexpr int LNS = last_logns<LOG1>(), P = G::B2 / 2;
  const int c0 = rank * G::B1, p0 = rank * P;
  cluster_grid<MASKED, -1>(G::LOGE + 1, t, y, n, pm, e, tile, work, [&] {
    for (int i = threadIdx.x; i < 16 * G::B1; i += TH)
      steps[(i >> 4) * 17 + (i & 15)] = twiddle_L(f, (c0 + (i >> 4)) * ((i & 15) << LNS));
    for (int u = threadIdx.x; u < G::B2 + G::L2; u += TH) {
      const int q = u < G::B2 ? ct_pair_row<LOG1>(p0 + (u >> 1), u & 1) : (u - G::B2) << LOG1;
      float sn, cs;
      sincospif((float)q * e.twk, &sn, &cs);
      twr[u] = cmk(cs, sn);  // twr[B2 + k2] is twc[k2]
    }
  });
  cluster_barrier();
  // 3. columns
  if (threadIdx.x < G::FT) {
    ClusterColSrc<LOG1, LOG2> src{reinterpret_cast<const float2 *>(tile), c0};
    ClusterColDst<LOG1, LOG2> dst{rows, steps, f, c0};
    ct_fft<float, LOG1, G::LOGB1, true, true, true, false, true>(s, f.tw1, src, dst);
  }
  cluster_barrier();
  // 4. rows and epilogue
  if (threadIdx.x < G::FT) {
    ClusterRowSrc<LOG2> src{rows};
    ct_fft<float, LOG2, G::LOGB2, false, false, false, false, true>(s, f.tw2, src, CtNoDst());
  }
  __syncthreads();
  rowpass_outputs<float, LOG1, LOG2, G::LOGB2, TH>(s, twr, twc, p0, e, F);
}

// The same for a grid that one CTA's FFT holds: the eight tiles are sent to the
// first CTA, which transforms them as nfft_small_body.
inline size_t cluster_small_smem(int logL) {
  const size_t TC = (size_t)2 << (logL - 3);
  return sizeof(float) * TC + sizeof(SRec<float>) * (2 * kClusterCap + kClusterSlack) +
         ((sizeof(int) * ((TC + 32) / 4 + 4) + 15) & ~(size_t)15) + sizeof(float2) * fft_pitch(1 << logL, 1);
}
template <int FORM>
__global__ void __cluster_dims__(kClusterCtas, 1, 1) __launch_bounds__(kClusterThreads, 1)
    k_nfft_cluster_small(const double *__restrict__ t, const float *__restrict__ y, int n, PhaseMul pm,
                         AccParams<float> e, FftDev<float> f, float2 *F) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = 1 << f.logL, LOGTC = f.logL - 2, TC = 1 << LOGTC, pitch = fft_pitch(L, 1);
  float *tile = reinterpret_cast<float *>(smem_raw);
  unsigned char *work = reinterpret_cast<unsigned char *>(tile + TC);
  float2 *s = reinterpret_cast<float2 *>(work + sizeof(SRec<float>) * (2 * kClusterCap + kClusterSlack) +
                                         ((sizeof(int) * ((TC + 32) / 4 + 4) + 15) & ~(size_t)15));
  y += (int64_t)blockIdx.y * n;
  F += (int64_t)blockIdx.y * e.nf;
  cluster_grid<FORM != kGatherFree, FORM>(LOGTC, t, y, n, pm, e, tile, work, [] {});
  __syncthreads();
  const int z0 = blockIdx.x << (LOGTC - 1);  // first packed point
  for (int i = threadIdx.x; i < TC / 2; i += kClusterThreads) {
    const float2 v = reinterpret_cast<const float2 *>(tile)[i];
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(cluster_addr(s + pad16(z0 + i), 0)), "f"(v.x), "f"(v.y)
                 : "memory");
  }
  cluster_barrier();
  if (blockIdx.x != 0) return;
  smem_fft<float>(s, pitch, f.logL, 1, f.tw1);
  for (int64_t k = threadIdx.x; k <= e.K; k += kClusterThreads) {
    const float2 Zk = s[pad16((int)(k & (L - 1)))];
    const float2 Zm = cconj(s[pad16((int)((L - k) & (L - 1)))]);
    acc_output<float>(e, k, Zk, Zm, F);
  }
}
template <int FORM>
int nfft_cluster_small(int logL, const double *t, const float *y, int n, const PhaseMul &pm, const AccParams<float> &e,
                       const FftDev<float> &f, float2 *F, int nslab, cudaStream_t st) {
  static SetupFlag attr;
  if (!setup_done(&attr)) {
    CUNA_CK(cudaFuncSetAttribute(k_nfft_cluster_small<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)cluster_small_smem(kClusterLo - 1)));
    mark_setup_done(&attr);
  }
  k_nfft_cluster_small<FORM>
      <<<dim3(kClusterCtas, nslab), kClusterThreads, cluster_small_smem(logL), st>>>(t, y, n, pm, e, f, F);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}

template <int LOGL, bool MASKED>
int nfft_cluster_at(const double *t, const float *y, int n, const PhaseMul &pm, const AccParams<float> &e,
                    const FftDev<float> &f, float2 *F, int nslab, cudaStream_t st) {
  constexpr size_t sm = ClusterCfg<LOGL>::smem;
  static_assert(sm <= 226 * 1024, "shared memory of a CTA");
  static SetupFlag attr;
  if (!setup_done(&attr)) {
    CUNA_CK(cudaFuncSetAttribute(k_nfft_cluster<LOGL, MASKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    mark_setup_done(&attr);
  }
  k_nfft_cluster<LOGL, MASKED><<<dim3(kClusterCtas, nslab), kClusterThreads, sm, st>>>(t, y, n, pm, e, f, F);
  CUNA_CK(cudaGetLastError());
  return CUNA2_SUCCESS;
}
// nslab value rows y of n samples at the times t
template <bool MASKED>
int nfft_cluster(int logL, const double *t, const float *y, int n, const PhaseMul &pm, const AccParams<float> &e,
                 const FftDev<float> &f, float2 *F, int nslab, cudaStream_t st) {
  switch (logL) {
    case 13: return nfft_cluster_at<13, MASKED>(t, y, n, pm, e, f, F, nslab, st);
    case 14: return nfft_cluster_at<14, MASKED>(t, y, n, pm, e, f, F, nslab, st);
    case 15: return nfft_cluster_at<15, MASKED>(t, y, n, pm, e, f, F, nslab, st);
  }
  return fail(CUNA2_ERROR_UNSUPPORTED, "cluster transform of 2^%d points", logL);
}

}  // namespace
}  // namespace cuna
