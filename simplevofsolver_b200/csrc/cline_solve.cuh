// cline_solve.cuh -- complex Neumann Thomas solves along x of the spectral
// Poisson paths (2D stretched x: one line per ky; 3D: one per (ky, kz)),
// gtsv component-wise (src/tdm.c:17-50, dft.c:364-395).  Lines are contiguous:
// S[line][i], complex.
//
// The matrix depends on the grid alone, so gtsv's pivots are a table, made
// once per solver by k_cline_table with gtsv's own expressions (tab[line][i]:
// row 0 the diagonal c_0, rows 1 .. n-2 val_i = 1 / (c_i - l_i v_{i-1}), row
// n-1 the last row's 1 / val, or 0 where gtsv zeroes that row); v_i = val_i
// u_i is formed again from it.  The sweeps then have no division in their
// chains (one rounding of x - l q and one of the product a row), every value
// the one gtsv computes.
//
// k_cline_solve: one warp owns LPB whole lines in shared memory, lanes 2 l and
// 2 l + 1 sweep the real and imaginary parts of line l; forward values stay
// on chip, so the spectrum is read and written once (32 bytes a point and 8 +
// 8 of the table, where chunks that go back to memory between the sweeps move
// 80).  The tables pass through a ring of kSlots chunks of kChunk rows that
// cp.async fills ahead of the sweeps (read straight from memory a batch ahead
// instead, the sweeps waited for them: 2.3 ms a launch at 512^3).
// Bound: the instructions a lone warp issues around its chain of five dependent
// roundings a row (about 128 cycles a row both ways, 8.2 each rounding), over
// the lines an SM can hold: hence one warp a block, operands loaded in
// batches, and few rounds (k3_poisson.cu says where the streaming kernel takes
// over).
#pragma once

#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include "fft_device.cuh"
#include "smem_limit.cuh"

namespace svof_cline {

constexpr double kEps = 2.220446049250313080847e-16;  // DBL_EPSILON
constexpr int kBatch = 8;                 // rows whose operands are loaded ahead of their chain
constexpr int kChunk = 32, kSlots = 4;    // the tables' ring: rows a slot (a warp's lanes), slots
// (pitch even: rows load in pairs; 34 doubles: the lines' pairs on distinct banks)
constexpr int kPitch = kChunk + 2;
// Operands are fetched a batch ahead, past the end of what a chunk holds by up
// to kBatch rows (and never used there): kPad bytes before and behind.
constexpr size_t kPad = 2 * sizeof(double) * kBatch;
// bytes of the ring: LPB lines and pl / pu
__host__ __device__ constexpr size_t cline_ring(int lpb) {
  return kPad + sizeof(double) * kSlots * (lpb + 1) * kPitch;
}

// the pivots of every line: diagonal -pl - pu + lambda, lambda = evy[line %
// nky] (+ evz[line / nky]), the first and last rows Neumann.  One line per
// thread, chunks of kTabChunk rows through shared memory so that the table is
// written in runs.  Lines (other than line 0, singular by construction) that
// meet a pivot of magnitude at most DBL_EPSILON are counted in *nsmall.
constexpr int kTabLines = 64, kTabChunk = 16;
static __global__ void __launch_bounds__(kTabLines)
    k_cline_table(double *__restrict__ tab, const double *__restrict__ pl, const double *__restrict__ pu,
                  const double *__restrict__ evy, const double *__restrict__ evz, int nky, long nlines, int nx,
                  unsigned long long *__restrict__ nsmall) {
  __shared__ double st[kTabLines][kTabChunk + 1];
  const int t = threadIdx.x;
  const long l0 = (long)blockIdx.x * kTabLines, line = l0 + t;
  const bool live = line < nlines;
  double lam = 0.;
  if (live) lam = evz ? evy[line % nky] + evz[line / nky] : evy[line];
  double v = 0.;
  bool small = false;
  for (int p0 = 0; p0 < nx; p0 += kTabChunk) {
    const int pw = min(kTabChunk, nx - p0);
    if (live) {
      for (int s = 0; s < pw; s++) {
        const int i = p0 + s;
        const double l = pl[i], u = pu[i];
        double c = -l - u + lam;
        if (0 == i) c += l;
        if (nx - 1 == i) c += u;
        double r;
        if (0 == i) {
          small |= !(fabs(c) > kEps);
          v = u / c;
          r = c;
        } else {
          const double piv = c - l * v;
          const bool ok = fabs(piv) > kEps;
          small |= !ok;
          r = (i < nx - 1 || ok) ? 1. / piv : 0.;
          v = r * (u);
        }
        st[t][s] = r;
      }
    }
    __syncthreads();
    for (int e = t; e < kTabLines * pw; e += kTabLines) {
      const int ll = e / pw, q = e - ll * pw;
      if (l0 + ll < nlines) tab[(l0 + ll) * nx + p0 + q] = st[ll][q];
    }
    __syncthreads();
  }
  if (nsmall && live && small && 0 != line) atomicAdd(nsmall, 1ull);
}

// kBatch rows of one component of a line: its values, the table's and pl / pu
// (s a multiple of kBatch: the last two come in pairs)
template <class R>
struct Batch {
  double y[kBatch];
  double2 r[kBatch / 2], lu[kBatch / 2];
  __device__ __forceinline__ void fetch(const R *q, const double *rr, const double *ll, int s) {
#pragma unroll
    for (int k = 0; k < kBatch; k++) y[k] = (double)q[2 * (s + k)];
#pragma unroll
    for (int k = 0; k < kBatch / 2; k++) {
      r[k] = reinterpret_cast<const double2 *>(rr + s)[k];
      lu[k] = reinterpret_cast<const double2 *>(ll + s)[k];
    }
  }
  __device__ __forceinline__ double forward(R *q, int s, double x) const {
#pragma unroll
    for (int k = 0; k < kBatch / 2; k++) {
      x = r[k].x * (y[2 * k] - lu[k].x * x);
      q[2 * (s + 2 * k)] = R(x);
      x = r[k].y * (y[2 * k + 1] - lu[k].y * x);
      q[2 * (s + 2 * k + 1)] = R(x);
    }
    return x;
  }
  __device__ __forceinline__ double backward(R *q, int s, double x) const {
#pragma unroll
    for (int k = kBatch / 2 - 1; k >= 0; k--) {
      x = y[2 * k + 1] - (double)R(r[k].y * (lu[k].y)) * x;
      q[2 * (s + 2 * k + 1)] = R(x);
      x = y[2 * k] - (double)R(r[k].x * (lu[k].x)) * x;
      q[2 * (s + 2 * k)] = R(x);
    }
    return x;
  }
};

// R: the spectrum's type (float: the defect-corrected form's passes, FP64
// arithmetic on FP32 storage); gauge0: line 0 takes the value 0 at its last
// row (see k3_poisson.cu); *small_pivots += *nsmall when both are given
template <class R, int LPB>
__global__ void __launch_bounds__(32) k_cline_solve(R *__restrict__ spec, const double *__restrict__ tab,
                                                    const double *__restrict__ pl, const double *__restrict__ pu,
                                                    long nlines, int nx, int gauge0,
                                                    unsigned long long *__restrict__ small_pivots,
                                                    const unsigned long long *__restrict__ nsmall) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  using C2 = typename svof_fft_dev::Cplx<R>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int n = nx, pitch = nx | 1;  // odd: the lanes' lines fall on distinct banks
  double(*ring)[LPB + 1][kPitch] = reinterpret_cast<double(*)[LPB + 1][kPitch]>(smraw + kPad);  // [kSlots]
  C2 *sq = reinterpret_cast<C2 *>(smraw + cline_ring(LPB));
  const int lane = threadIdx.x;
  const long l0 = (long)blockIdx.x * LPB;
  const int nl = (int)min((long)LPB, nlines - l0);
  C2 *sp = reinterpret_cast<C2 *>(spec) + l0 * n;
  const double *tb = tab + l0 * n;
  const int nch = (n + kChunk - 1) / kChunk;
  // rows of chunk c of the lines' tables and of pl (pu): lane = row
  auto load_ring = [&](int c, const double *lu) {
    const int i = c * kChunk + lane;
    if (i < n) {
      double(*d)[kPitch] = ring[c & (kSlots - 1)];
#pragma unroll
      for (int ll = 0; ll < LPB; ll++)
        if (ll < nl) __pipeline_memcpy_async(&d[ll][lane], tb + (long)ll * n + i, sizeof(double));
      __pipeline_memcpy_async(&d[LPB][lane], lu + i, sizeof(double));
    }
  };
  for (int ll = 0; ll < nl; ll++)
    for (int i = lane; i < n; i += 32) __pipeline_memcpy_async(sq + ll * pitch + i, sp + (long)ll * n + i, sizeof(C2));
  for (int c = 0; c < kSlots - 1; c++) {
    if (c < nch) load_ring(c, pl);
    __pipeline_commit();
  }
  const int ll = lane >> 1;
  const bool sweeps = ll < nl;
  const int rl = sweeps ? ll : 0;
  R *q = reinterpret_cast<R *>(sq + rl * pitch) + (lane & 1);  // element i at q[2 i]
  double x = 0., c0 = 1.;
  for (int c = 0; c < nch; c++) {
    if (c + kSlots - 1 < nch) load_ring(c + kSlots - 1, pl);
    __pipeline_commit();
    __pipeline_wait_prior(kSlots - 1);
    __syncwarp();
    if (sweeps) {
      const double *r = ring[c & (kSlots - 1)][rl], *l = ring[c & (kSlots - 1)][LPB];
      const int i0 = c * kChunk, rows = min(kChunk, n - i0);
      R *qc = q + 2 * i0;
      const int e = (c == nch - 1) ? rows - 1 : rows;
      int s = 0;
      auto one = [&]() {
        x = r[s] * ((double)qc[2 * s] - l[s] * x);
        qc[2 * s] = R(x);
        s++;
      };
      if (0 == c) {
        c0 = r[0];
        x = (double)qc[0] / c0;
        qc[0] = R(x);
        for (s = 1; s < min(kBatch, e);) one();
      }
      // batches in pairs A, B: each one's operands on their way during the
      // other one's chain
      if (s + kBatch <= e) {
        Batch<R> A, B;
        A.fetch(qc, r, l, s);
        while (true) {
          B.fetch(qc, r, l, s + kBatch);
          x = A.forward(qc, s, x);
          s += kBatch;
          if (s + kBatch > e) break;
          A.fetch(qc, r, l, s + kBatch);
          x = B.forward(qc, s, x);
          s += kBatch;
          if (s + kBatch > e) break;
        }
      }
      while (s < e) one();
      if (c == nch - 1) {
        const double rv = r[e];
        x = (0. != rv && !(gauge0 && 0 == l0 + ll)) ? rv * ((double)qc[2 * e] - l[e] * x) : 0.;
        qc[2 * e] = R(x);
      }
    }
    __syncwarp();
  }
  // backward: x is the last row as it was stored (rounded to R).  The ring
  // still holds the last kSlots chunks' tables; pu takes pl's place
  __pipeline_wait_prior(0);
  __syncwarp();
  for (int c = max(0, nch - kSlots); c < nch; c++) {
    const int i = c * kChunk + lane;
    if (i < n) ring[c & (kSlots - 1)][LPB][lane] = __ldg(pu + i);
  }
  __syncwarp();
  if (sweeps) x = (double)q[2 * (n - 1)];
  for (int c = nch - 1; c >= 0; c--) {
    // chunk c + 1's slot is free
    if (c < nch - 1 && c - (kSlots - 1) >= 0) load_ring(c - (kSlots - 1), pu);
    __pipeline_commit();
    __pipeline_wait_prior(kSlots - 1);
    __syncwarp();
    const int i0 = c * kChunk, rows = min(kChunk, n - i0);
    if (sweeps) {
      const double *r = ring[c & (kSlots - 1)][rl], *u = ring[c & (kSlots - 1)][LPB];
      R *qc = q + 2 * i0;
      int s = (c == nch - 1) ? rows - 1 : rows;  // rows [0, s) to do
      const int e = (0 == c) ? 1 : 0;                  // row 0 has its own quotient
      auto one = [&]() {
        s--;
        x = (double)qc[2 * s] - (double)R(r[s] * (u[s])) * x;
        qc[2 * s] = R(x);
      };
      while (s > e && 0 != s % kBatch) one();
      if (s - kBatch >= e) {
        Batch<R> A, B;
        A.fetch(qc, r, u, s - kBatch);
        while (true) {
          s -= kBatch;
          B.fetch(qc, r, u, s - kBatch);
          x = A.backward(qc, s, x);
          if (s - kBatch < e) break;
          s -= kBatch;
          A.fetch(qc, r, u, s - kBatch);
          x = B.backward(qc, s, x);
          if (s - kBatch < e) break;
        }
      }
      while (s > e) one();
      if (0 == c) {
        x = (double)qc[0] - (double)R(u[0] / c0) * x;
        qc[0] = R(x);
      }
    }
    __syncwarp();
    if (lane < rows) {
#pragma unroll
      for (int m = 0; m < LPB; m++)
        if (m < nl) sp[(long)m * n + i0 + lane] = sq[m * pitch + i0 + lane];
    }
  }
  if (small_pivots && 0 == blockIdx.x && 0 == lane && *nsmall) atomicAdd(small_pivots, *nsmall);
}

// Lines per block: one while the chip has a warp slot for each, then as many
// as share a warp well within 32 KB (two at a time gain the most there is at
// 16 to 24 lines an SM; 128^3, 56 lines an SM: 32 / 20 / 18 us a launch with
// 2 / 4 / 8; 256^3, 223: 180 / 119 / 123)
inline size_t cline_smem(int lpb, int nx, size_t es) { return cline_ring(lpb) + 2 * es * lpb * (nx | 1) + kPad; }
inline int cline_lpb(long nlines, int nx, size_t es) {
  int lpb = nlines <= 148L * 10 ? 1 : (nlines <= 148L * 24 ? 2 : 8);
  while (lpb > 1 && cline_smem(lpb, nx, es) > 32 * 1024) lpb >>= 1;
  return lpb;
}

template <class F>
inline auto cline_by_lpb(int lpb, F f) {
  if (1 == lpb) return f(std::integral_constant<int, 1>());
  if (2 == lpb) return f(std::integral_constant<int, 2>());
  if (4 == lpb) return f(std::integral_constant<int, 4>());
  return f(std::integral_constant<int, 8>());
}

// opt-in shared memory of the solve of `nlines` lines (once per device)
template <class R>
inline cudaError_t cline_prepare(long nlines, int nx) {
  return cline_by_lpb(cline_lpb(nlines, nx, sizeof(R)), [&](auto c) {
    constexpr int LPB = decltype(c)::value;
    cudaError_t e = raise_smem_limit(k_cline_solve<R, LPB>, cline_smem(LPB, nx, sizeof(R)));
    if (cudaSuccess != e) return e;
    return cudaFuncSetAttribute(k_cline_solve<R, LPB>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
}

}  // namespace svof_cline
