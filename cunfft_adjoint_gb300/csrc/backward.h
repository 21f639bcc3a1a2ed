// backward.h -- launches of the accurate transform's vector-Jacobian product
// (backward.cu), called by the plans (accurate.cu).
#pragma once
#include <cuda_runtime.h>
#include "common.cuh"
#include "phase.cuh"
#include "runtime.h"

namespace cuna {

// Per-series constants of a batch of backward passes (up to kBwdSeries
// series per launch, passed by value): the phase multiplier of x = (t - t0)/T
// and ng / T, the chain-rule factor of dL/dt.
constexpr int kBwdSeries = 256;
struct BwdSeries {
  PhaseMul pm[kBwdSeries];
  double tscale[kBwdSeries];
};

// One group of ns series of n samples each: times, values, upstream gradients
// G (nf per series) and results (gy or gt may be NULL) of consecutive series
// lie one after the other.  z and r: ns packed complex grids of 2^g.logL
// points each (unused where one CTA holds the grid, `small`).
template <typename T> struct BwdArgs {
  typedef typename CxOf<T>::type C;
  const double *t;
  const T *y;
  const C *G;
  T *gy;
  double *gt;
  int64_t n, ng, nf;
  int ns, m;
  double tau;
  bool small;
  FftGeom g;
  C *z, *r;
  const BwdSeries *ser;
};
template <typename T> int backward_group(const BwdArgs<T> &a, cudaStream_t st);

}  // namespace cuna
