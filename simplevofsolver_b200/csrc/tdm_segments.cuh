// tdm_segments.cuh -- Thomas recurrences of the implicit-x systems, one warp
// a line, by segments.
//
// A recurrence v_i = f_i(v_{i-1}) is a chain of a division (pivots, about 190
// cycles a row) or of three roundings (sweeps, about 60 with their loads) a
// row, and one thread a line leaves the rest of its warp, and often of its SM,
// waiting.  The rows go to the 32 lanes in segments instead.  A lane starts
// kWarm rows ahead of its own from 0; where the system is well dominated by
// its diagonal (implicit x within the explicit limits of the other directions)
// those rows contract the difference from the true value until the two are
// the same bits, and from there on they stay the same, each row being a
// function of the value before it alone.  Whether they met is checked: the
// value a lane entered its first row with must be the bits its neighbour
// ended with.  Lanes that differ run their rows again from the neighbour's
// value until none does, so the results are those of a single thread,
// whatever the coefficients; poorly dominated systems just take more rounds.
#pragma once

#include <cuda_runtime.h>

namespace svof_tdm {

constexpr int kWarm = 24;

// the pivots: rows 0 .. n-1 of the system with Laplacian rows lap[3 i + (0, 1, 2)] and
// prefactor pf: L[i] = tdm_l[i]; R[0] = tdm_c[0], R[i] = 1 / (c_i - l_i
// v_{i-1}), R[n-1] = the last row's or 0 where gtsv zeroes that row; V[i] =
// v_i.  All 32 lanes of the warp take part (n >= 3).  One thread a system:
// 14 us a launch at 128 rows, 24 at 256, 89 at 1024; now 6.6, 7.9 and 16 (the
// kernels that call it, their staging of the rows included).
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

// gtsv of one line (src/tdm.c:17-50) on the table above: x[0 .. n-1] holds the
// right-hand side and takes the solution, q[0 .. n-1] is scratch; both and the
// table in shared memory.  All 32 lanes of the warp take part (n >= 3).
__device__ __forceinline__ void line_solve(const double *L, const double *R, const double *V, int n, double *x,
                                           double *q) {
  const int lane = threadIdx.x & 31;
  const int seg = ((n - 2 + 31) / 32) | 1;  // odd: the lanes' rows on distinct banks
  // ---- forward, x -> q: rows 1 .. n-2 by segments
  {
    const int a = 1 + lane * seg, b = min(a + seg, n - 1);
    const double q0 = x[0] / R[0];
    int i = max(1, a - kWarm);
    double v = (1 == i) ? q0 : 0.;
    const int e = min(a, n - 1);
#pragma unroll 4
    for (; i < e; i++) v = R[i] * (x[i] - L[i] * v);
    double start = v;
    bool todo = a < b;
    while (__any_sync(0xffffffffu, todo)) {
      if (todo) {
        v = start;
#pragma unroll 4
        for (i = a; i < b; i++) {
          v = R[i] * (x[i] - L[i] * v);
          q[i] = v;
        }
      }
      const double before = __shfl_up_sync(0xffffffffu, v, 1);
      todo = a < b && lane > 0 && __double_as_longlong(before) != __double_as_longlong(start);
      if (todo) start = before;
    }
    if (0 == lane) q[0] = q0;
    if (a < b && b == n - 1) {
      const double r = R[n - 1];
      q[n - 1] = (0. != r) ? r * (x[n - 1] - L[n - 1] * v) : 0.;
    }
  }
  __syncwarp();
  // ---- backward, q -> x: rows n-2 .. 0 by segments from the top
  {
    const int seg_b = ((n - 1 + 31) / 32) | 1;
    const int a = n - 2 - lane * seg_b, b = max(a - seg_b, -1);  // rows a, a - 1 .. b + 1
    const double qn = q[n - 1];
    int i = min(n - 2, a + kWarm);
    double v = (n - 2 == i) ? qn : 0.;
    const int e = max(a, -1);
#pragma unroll 4
    for (; i > e; i--) v = q[i] - V[i] * v;
    double start = v;
    bool todo = a > b;
    while (__any_sync(0xffffffffu, todo)) {
      if (todo) {
        v = start;
#pragma unroll 4
        for (i = a; i > b; i--) {
          v = q[i] - V[i] * v;
          x[i] = v;
        }
      }
      const double before = __shfl_up_sync(0xffffffffu, v, 1);
      todo = a > b && lane > 0 && __double_as_longlong(before) != __double_as_longlong(start);
      if (todo) start = before;
    }
    if (0 == lane) x[n - 1] = qn;
  }
  __syncwarp();
}

}  // namespace svof_tdm
