// tdm_pivots.cuh -- the Thomas pivots of one implicit-x system, one warp.
//
// v_i = u_i / (c_i - l_i v_{i-1}) is a chain of a division a row (about 190
// cycles) and the predictor waits for it: one thread a system took 14 us at
// 128 rows, 24 at 256, 89 at 1024.  The rows go to the 32 lanes in segments
// instead.  A lane starts kWarm rows ahead of its own from v = 0; the rows
// between contract the difference from the true v (by v_i l_i / u_i v_i per
// row, at most about 0.2 where the time step is within the explicit limits of
// the other directions) until the two are the same bits, and from there on
// they stay the same, the recurrence being a function of the value alone.
// Whether they met is checked: a lane's v at its first row must be the bits
// its neighbour ended with.  Lanes that differ run their rows again from the
// neighbour's value until none does, so the table is the one a single thread
// computes, whatever the coefficients.  6.6, 7.9 and 16 us at those sizes
// (the kernels that call it, their staging of the rows included).
#pragma once

#include <cuda_runtime.h>

namespace svof_tdm {

constexpr int kWarm = 24;

// rows 0 .. n-1 of the system with Laplacian rows lap[3 i + (0, 1, 2)] and
// prefactor pf: L[i] = tdm_l[i]; R[0] = tdm_c[0], R[i] = 1 / (c_i - l_i
// v_{i-1}), R[n-1] = the last row's or 0 where gtsv zeroes that row; V[i] =
// v_i.  All 32 lanes of the warp take part (n >= 3).
__device__ __forceinline__ void pivots(const double *lap, double pf, int n, double *__restrict__ L,
                                       double *__restrict__ R, double *__restrict__ V) {
  constexpr double kEps = 2.220446049250313080847e-16;  // DBL_EPSILON
  const int lane = threadIdx.x & 31;
  const double c0 = 1. - pf * lap[1];
  const double v0 = (-pf * lap[2]) / c0;
  const int rows = n - 2;  // rows 1 .. n-2
  const int seg = ((rows + 31) / 32) | 1;  // odd: the lanes' rows of lap fall on distinct banks
  const int a = 1 + lane * seg, b = min(a + seg, n - 1);
  double v = 0.;
  // the rows ahead (from row 1 on, its own start is the true one)
  int i = max(1, a - kWarm);
  if (1 == i) v = v0;
  for (; i < min(a, n - 1); i++) {
    const double l = -pf * lap[3 * i + 0];
    const double c = 1. - pf * lap[3 * i + 1];
    const double u = -pf * lap[3 * i + 2];
    const double val = 1. / (c - l * v);
    v = val * (u);
  }
  double start = v;
  bool todo = a < b;
  while (__any_sync(0xffffffffu, todo)) {
    if (todo) {
      v = start;
      for (i = a; i < b; i++) {
        const double l = -pf * lap[3 * i + 0];
        const double c = 1. - pf * lap[3 * i + 1];
        const double u = -pf * lap[3 * i + 2];
        const double val = 1. / (c - l * v);
        v = val * (u);
        L[i] = l;
        R[i] = val;
        V[i] = v;
      }
    }
    const double before = __shfl_up_sync(0xffffffffu, v, 1);
    todo = a < b && lane > 0 && __double_as_longlong(before) != __double_as_longlong(start);
    if (todo) start = before;
  }
  // the lane of row n - 2 has the last row too
  if (a < b && b == n - 1) {
    const double l = -pf * lap[3 * (n - 1) + 0];
    const double c = 1. - pf * lap[3 * (n - 1) + 1];
    const double val = c - l * v;
    L[n - 1] = l;
    R[n - 1] = fabs(val) > kEps ? 1. / val : 0.;
  }
  if (0 == lane) {
    L[0] = -pf * lap[0];
    R[0] = c0;
    V[0] = v0;
  }
}

}  // namespace svof_tdm
