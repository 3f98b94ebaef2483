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

// How often a line's segments have to be run again, from the table alone: a
// difference ahead of a segment shrinks by |R_i L_i| a row forward and by |V_i|
// a row backward; the rows it takes to fall below eps, beyond the `warm` ahead
// of each segment, run through one more segment a round.  The rounds of the
// boundary below row a = 1 + s seg (n rows; forward as far as row 1, backward
// as far as row n - 2, where the true value is known), at most `limit`.
__host__ __device__ inline int boundary_rounds(const double *L, const double *R, const double *V, int n, int seg, int s,
                                               int warm, double eps, bool backward, int limit) {
  constexpr int B = 8;  // rows whose loads are in flight together
  const int a = 1 + s * seg;
  if (a >= n - 1) return 0;
  const int have = backward ? n - 1 - a : a - 1;
  const int most = warm + (limit - 1) * seg + 1, last = have < most ? have : most;
  double p = 1.;
  int rows = 0;
  while (rows < last && p > eps) {
    double c[B];
#pragma unroll
    for (int k = 0; k < B; k++) {
      const int q = rows + k < last ? rows + k : last - 1;
      c[k] = backward ? V[a + q] : R[a - 1 - q] * L[a - 1 - q];
    }
#pragma unroll
    for (int k = 0; k < B; k++) {
      if (rows < last && p > eps) {
        p *= fabs(c[k]);
        rows++;
      }
    }
  }
  return rows <= warm ? 0 : (rows - warm + seg - 1) / seg;
}

__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_int(a) == __float_as_int(b); }

// gtsv of one line (src/tdm.c:17-50) on the table above: x[0 .. n-1] holds the
// right-hand side and takes the solution, q[0 .. n-1] is scratch; both and the
// table in shared memory.  All 32 lanes of the warp take part (n >= 3).
// WARM: rows ahead (float needs fewer)
template <class T, int WARM = kWarm>
__device__ __forceinline__ void line_solve(const T *__restrict__ L, const T *__restrict__ R, const T *__restrict__ V,
                                           int n, T *__restrict__ x, T *__restrict__ q) {
  const int lane = threadIdx.x & 31;
  const int seg = ((n - 2 + 31) / 32) | 1;  // odd: the lanes' rows on distinct banks
  // ---- forward, x -> q: rows 1 .. n-2 by segments
  {
    const int a = 1 + lane * seg, b = min(a + seg, n - 1);
    const T q0 = x[0] / R[0];
    int i = max(1, a - WARM);
    T v = (1 == i) ? q0 : T(0.);
    const int e = min(a, n - 1);
#pragma unroll 4
    for (; i < e; i++) v = R[i] * (x[i] - L[i] * v);
    T start = v;
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
      const T before = __shfl_up_sync(0xffffffffu, v, 1);
      todo = a < b && lane > 0 && !same_bits(before, start);
      if (todo) start = before;
    }
    if (0 == lane) q[0] = q0;
    if (a < b && b == n - 1) {
      const T r = R[n - 1];
      q[n - 1] = (T(0.) != r) ? r * (x[n - 1] - L[n - 1] * v) : T(0.);
    }
  }
  __syncwarp();
  // ---- backward, q -> x: rows n-2 .. 0 by segments from the top
  {
    const int seg_b = ((n - 1 + 31) / 32) | 1;
    const int a = n - 2 - lane * seg_b, b = max(a - seg_b, -1);  // rows a, a - 1 .. b + 1
    const T qn = q[n - 1];
    int i = min(n - 2, a + WARM);
    T v = (n - 2 == i) ? qn : T(0.);
    const int e = max(a, -1);
#pragma unroll 4
    for (; i > e; i--) v = q[i] - V[i] * v;
    T start = v;
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
      const T before = __shfl_up_sync(0xffffffffu, v, 1);
      todo = a > b && lane > 0 && !same_bits(before, start);
      if (todo) start = before;
    }
    if (0 == lane) x[n - 1] = qn;
  }
  __syncwarp();
}

// The same for a line by the calling thread alone, in place
template <class T>
__device__ __forceinline__ void line_solve_thread(const T *__restrict__ L, const T *__restrict__ R,
                                                  const T *__restrict__ V, int n, T *__restrict__ x) {
  T v = x[0] / R[0];
  x[0] = v;
#pragma unroll 4
  for (int i = 1; i < n - 1; i++) {
    v = R[i] * (x[i] - L[i] * v);
    x[i] = v;
  }
  const T r = R[n - 1];
  x[n - 1] = v = (T(0.) != r) ? r * (x[n - 1] - L[n - 1] * v) : T(0.);
#pragma unroll 4
  for (int i = n - 2; i >= 0; i--) {
    v = x[i] - V[i] * v;
    x[i] = v;
  }
}

// The same for 32 / LPL lines of a warp at once, LPL lanes a line, in place:
// x[0 .. n-1] is the line of the calling lane (its group's), src its right-hand
// side in global memory, read again only by lanes that have to repeat their
// rows.  seg: rows a lane, odd, LPL seg >= n - 2.  Fewer, longer segments
// spend less on the rows ahead; rows go in batches, operands first, since a
// lane's stores are to the array it loads from.
template <class T, int LPL, int WARM, class R>
__device__ __forceinline__ void group_solve(const T *__restrict__ L, const T *__restrict__ Rv,
                                            const T *__restrict__ V, int n, int seg, T *x, const R *src) {
  constexpr int B = 8;
  const int s = threadIdx.x & (LPL - 1);
  const int a = 1 + s * seg, b = min(a + seg, n - 1);
  const bool has = a < b;
  T v, start, sb, before;
  // rows a .. b-1 forward from v, stored
  auto forward = [&]() {
    int i = a;
    for (; i + B <= b; i += B) {
      T y[B], r[B], l[B];
#pragma unroll
      for (int k = 0; k < B; k++) {
        y[k] = x[i + k];
        r[k] = Rv[i + k];
        l[k] = L[i + k];
      }
#pragma unroll
      for (int k = 0; k < B; k++) {
        v = r[k] * (y[k] - l[k] * v);
        x[i + k] = v;
      }
    }
    for (; i < b; i++) {
      v = Rv[i] * (x[i] - L[i] * v);
      x[i] = v;
    }
  };
  auto backward = [&]() {
    int i = b - 1;
    for (; i - B + 1 >= a; i -= B) {
      T y[B], w[B];
#pragma unroll
      for (int k = 0; k < B; k++) {
        y[k] = x[i - k];
        w[k] = V[i - k];
      }
#pragma unroll
      for (int k = 0; k < B; k++) {
        v = y[k] - w[k] * v;
        x[i - k] = v;
      }
    }
    for (; i >= a; i--) {
      v = x[i] - V[i] * v;
      x[i] = v;
    }
  };
  // ---- forward
  const T q0 = x[0] / Rv[0];
  {
    int i = max(1, a - WARM);
    v = (1 == i) ? q0 : T(0.);
    const int e = min(a, n - 1);
#pragma unroll 8
    for (; i < e; i++) v = Rv[i] * (x[i] - L[i] * v);
  }
  __syncwarp();  // the rows ahead are read before their lanes write them
  start = v;
  if (has) forward();
  while (true) {
    before = __shfl_up_sync(0xffffffffu, v, 1, LPL);
    const bool again = has && s > 0 && !same_bits(before, start);
    if (!__any_sync(0xffffffffu, again)) break;
    if (again) {
      for (int i = a; i < b; i++) x[i] = T(src[i]);
      v = start = before;
      forward();
    }
  }
  if (0 == s) x[0] = q0;
  if (has && b == n - 1) {
    const T r = Rv[n - 1];
    x[n - 1] = (T(0.) != r) ? r * (x[n - 1] - L[n - 1] * v) : T(0.);
  }
  __syncwarp();
  // ---- backward
  {
    int i = min(n - 2, b - 1 + WARM);
    v = (n - 2 == i) ? x[n - 1] : T(0.);
    if (has) {
#pragma unroll 8
      for (; i >= b; i--) v = x[i] - V[i] * v;
    }
  }
  __syncwarp();
  sb = v;
  if (has) backward();
  while (true) {
    before = __shfl_down_sync(0xffffffffu, v, 1, LPL);
    const bool again = has && b != n - 1 && !same_bits(before, sb);
    if (!__any_sync(0xffffffffu, again)) break;
    if (again) {
      // the forward values of these rows again, then back from the
      // neighbour's value
      for (int i = a; i < b; i++) x[i] = T(src[i]);
      v = start;
      forward();
      v = sb = before;
      backward();
    }
  }
  if (0 == s) x[0] = x[0] - V[0] * v;
  __syncwarp();
}

}  // namespace svof_tdm
