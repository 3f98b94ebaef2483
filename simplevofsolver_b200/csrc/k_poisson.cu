// k_poisson.cu -- pressure Poisson solve of the FP64 2D path.
//
// Uniform x grid (src/fluid/compute_potential/dct.c:373-421):
//   k_dct_fwd     divergence right-hand side of one row, FFTW_REDFT10 along x
//   k_dct_ysolve  periodic tri-diagonal system along y for every x wavenumber
//                 (Sherman-Morrison, src/tdm.c:78-99), one wavenumber per thread
//   k_dct_inv     FFTW_REDFT01 along x, psi row with halo and Neumann walls
// Stretched x grid (src/fluid/compute_potential/dft.c:406-468):
//   k_dft_fwd     right-hand side of a tile of columns, r2c along y
//   k_cline_solve (cline_solve.cuh) complex Neumann tri-diagonal system along
//                 x for every y wavenumber (src/tdm.c:17-50, component-wise)
//   k_dft_inv     c2r along y, psi columns with halo and walls
//
// The reference transposes between x- and y-pencils around every transform;
// on one device the spectral array is instead laid out so that each line
// solve reads it coalesced: DCT path [j][kx] (threads over kx walk j), DFT
// path [ky][i] (contiguous lines).  No transpose pass exists.
//
// The transforms are the radix-2 decimation-in-time FFT of the oracle
// (oracle/svof_fft.c) with the same butterflies and the same twiddle tables,
// so with FMA contraction disabled they agree with it bit for bit.  Lengths
// must be powers of two (the DCT path's row transforms: 4 .. 4096 points, the
// DFT path's column transforms: 4 .. 8192).
#include <type_traits>

#include "cline_solve.cuh"
#include "fft_device.cuh"
#include "smem_limit.cuh"
#include "svof_internal.cuh"

namespace svof {

using svof_fft_dev::bitrev;

// assign_input, dct.c:285-315 / dft.c:315-345
__device__ __forceinline__ double poisson_rhs(const double *__restrict__ ux, const double *__restrict__ uy,
                                              const Grid2 &g, int i, int j, double prefactor) {
  const int nx = g.nx;
  const double dx = g.dxf[i - 1];
  const double ux_xm = ux[ix_ux(nx, i, j)];
  const double ux_xp = ux[ix_ux(nx, i + 1, j)];
  const double uy_ym = uy[ix_cc(nx, i, j)];
  const double uy_yp = uy[ix_cc(nx, i, j + 1)];
  return prefactor * (+(ux_xp - ux_xm) / dx + (uy_yp - uy_ym) / g.dy);
}

// the right-hand side of the forward solve (assign_input): the divergence of
// the predicted velocity times the substep's prefactor
struct DivRhs {
  const double *ux, *uy;
  Grid2 g;
  double prefactor;
  __device__ __forceinline__ double operator()(int i, int j) const { return poisson_rhs(ux, uy, g, i, j, prefactor); }
};

// a right-hand side given as an array [j-1][i-1] divided by the cell widths
// dxf (the adjoint's solve with the grid-metric weights of the x grid)
struct ArrayRhs {
  const double *r;
  const double *dxf;
  int nx;
  __device__ __forceinline__ double operator()(int i, int j) const {
    return r[(size_t)(j - 1) * nx + (i - 1)] / dxf[i - 1];
  }
};

// ---------------------------------------------------------------- DCT path
// A block owns DctShape<L2N>::ROWS consecutive rows j (N = nx = 2^L2N points
// each; THREADS threads, pairs of (row, butterfly group) across the lanes)
// and runs their transforms as the register-blocked passes of fft_device.cuh:
// the same butterflies, twiddles and stage order as the oracle, three stages
// per pass between shared-memory round trips.  Dynamic shared memory: re / im
// (ROWS fft_ld(L2N) each), the rows' input (ROWS N) and, for the inverse, the
// rows' output (ROWS N).
// ROWS: one row up to 256 points (those grids have few rows: one block per
// row keeps the SMs busy), then 2048 / N; THREADS: the first pass's pairs,
// 32 .. 256
template <int L2N>
struct DctShape {
  static constexpr int N = 1 << L2N;
  static constexpr int ROWS = (L2N <= 8 || (2048 >> L2N) < 1) ? 1 : (2048 >> L2N);
  static constexpr int PAIRS = ROWS * (N >> (L2N < 3 ? L2N : 3));
  static constexpr int THREADS = PAIRS < 32 ? 32 : (PAIRS > 256 ? 256 : (PAIRS + 31) / 32 * 32);
  static constexpr int LD = svof_fft_dev::fft_ld(L2N);
  static constexpr size_t SMEM_FWD = sizeof(double) * ROWS * (2 * (size_t)LD + N);
  static constexpr size_t SMEM_INV = sizeof(double) * ROWS * (2 * (size_t)LD + 2 * N);
};

// rows j0 .. j0 + ROWS - 1 of the right-hand side, FFTW_REDFT10 along x into
// spec (Makhoul: v_m = x_{2m}, v_{n-1-m} = x_{2m+1}, an FFT of v, then
// 2 Re(w_k V_k) with the pre/post twiddles cs)
template <int L2N, class Rhs>
__device__ __forceinline__ void dct_fwd_rows(const Rhs &rhs, double *__restrict__ spec,
                                             const double *__restrict__ tw, const double *__restrict__ cs, int ny) {
  using S = DctShape<L2N>;
  constexpr int N = S::N, ROWS = S::ROWS, LD = S::LD;
  extern __shared__ double dsm[];
  double *re = dsm, *im = re + ROWS * LD, *rr = im + ROWS * LD;  // rr [ROWS][N]
  const int j0 = 1 + blockIdx.x * ROWS;
  const int nr = min(ROWS, ny - j0 + 1);
  // the rows' right-hand sides, read in order (coalesced)
  for (int w = threadIdx.x; w < ROWS * N; w += S::THREADS) {
    const int c = w >> L2N, i = w & (N - 1);
    rr[w] = (c < nr) ? rhs(i + 1, j0 + c) : 0.;
  }
  __syncthreads();
  // point p of the bit-reversed FFT input holds v_m, m = bitrev(p)
  auto first = [&](int c, int base, auto gc, auto hc, double *xr, double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int m = bitrev(base + q * H, L2N);
      const int src = (m < N / 2) ? 2 * m : 2 * (N - 1 - m) + 1;
      xr[q] = rr[c * N + src];
      xi[q] = 0.;
    }
  };
  auto last = [&](int c, int base, auto gc, auto hc, const double *xr, const double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
    if (c >= nr) return;
    double *out = spec + (size_t)(j0 + c - 1) * N;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int k = base + q * H;
      const double2 w = __ldg(reinterpret_cast<const double2 *>(cs) + k);
      out[k] = 2.0 * (w.x * xr[q] + w.y * xi[q]);
    }
  };
  svof_fft_dev::fft_lines<double, L2N, ROWS, 1, S::THREADS>(re, im, tw, first, last);
}

template <int L2N>
__global__ void __launch_bounds__(DctShape<L2N>::THREADS) k_dct_fwd(const double *__restrict__ ux, const double *__restrict__ uy,
                                                        double *__restrict__ spec, const double *__restrict__ tw,
                                                        const double *__restrict__ cs, const double *__restrict__ dtp,
                                                        double gam, Grid2 g) {
  pdl_enter();
  const double dt = *dtp;
  const double prefactor = 1. / (gam * dt) / (2. * (1 << L2N));
  dct_fwd_rows<L2N>(DivRhs{ux, uy, g, prefactor}, spec, tw, cs, g.ny);
}

template <int L2N>
__global__ void __launch_bounds__(DctShape<L2N>::THREADS) k_dct_fwd_rhs(const double *__restrict__ r, double *__restrict__ spec,
                                                            const double *__restrict__ tw,
                                                            const double *__restrict__ cs, Grid2 g) {
  dct_fwd_rows<L2N>(ArrayRhs{r, g.dxf, g.nx}, spec, tw, cs, g.ny);
}

// periodic tri-diagonal solve along y per wavenumber k (src/tdm.c:78-99 with
// gtsv :17-50).  The k-dependent, time-independent quantities the reference
// recomputes on every call are tables: vt[j][k] (gtsv's v), rvt[j][k]
// (gtsv's val = 1 / (c - l v[j-1]), j = 1 .. n-3), lastf[k] (1 / val of the
// last row, 0 where the reference zeroes that row), q1t[j][k] and den[k]
// (Sherman-Morrison).  A block owns kt consecutive wavenumbers; all its
// threads stage the lines and their tables in shared memory ([j][t],
// coalesced), then one thread per line runs the recurrences on shared memory
// only, and all threads apply the Sherman-Morrison correction on the way out.
__global__ void k_dct_ysolve(double *__restrict__ spec, const double *__restrict__ vt,
                             const double *__restrict__ rvt, const double *__restrict__ q1t,
                             const double *__restrict__ ck, const double *__restrict__ lastf,
                             const double *__restrict__ den, double lap, int nx, int ny, int kt) {
  pdl_enter();
  extern __shared__ double sm[];
  double *sq = sm;                       // [ny][kt] line data
  double *sv = sm + (size_t)ny * kt;     // [ny][kt] v
  double *sr = sm + 2 * (size_t)ny * kt; // [ny][kt] val
  __shared__ double sl[64];
  const int k0 = blockIdx.x * kt;
  const int n = ny;
  const int nk = min(kt, nx - k0);
  for (int w = threadIdx.x; w < n * kt; w += blockDim.x) {
    const int j = w / kt, t = w - j * kt;
    const size_t g = (size_t)j * nx + k0 + t;
    const bool ok = t < nk;
    sq[w] = ok ? spec[g] : 0.;
    sv[w] = ok ? vt[g] : 0.;
    sr[w] = ok ? rvt[g] : 0.;
  }
  __syncthreads();
  const int t = threadIdx.x;
  if (t < nk) {
    const int k = k0 + t;
    const double l = lap, u = lap, c = ck[k];
    const double lf = lastf[k];
    const double d = den[k];
    double *q = sq + t;
    const double *v = sv + t, *r = sr + t;
#define Q(jj) q[(size_t)(jj) * kt]
#define V(jj) v[(size_t)(jj) * kt]
#define RV(jj) r[(size_t)(jj) * kt]
    // gtsv of size n-1 on rows 0 .. n-2.  The interior rows go in batches of
    // YB: the batch's loads first, then the dependent chain on registers,
    // then its stores (the same expressions in the same order as one row at
    // a time, which the remainder rows use).
    constexpr int YB = 8;
    double qprev = Q(0) / c;
    Q(0) = qprev;
    int i = 1;
    for (; i + YB <= n - 2; i += YB) {
      double xv[YB], rv[YB];
#pragma unroll
      for (int k = 0; k < YB; k++) {
        xv[k] = Q(i + k);
        rv[k] = RV(i + k);
      }
#pragma unroll
      for (int k = 0; k < YB; k++) {
        qprev = rv[k] * (xv[k] - l * qprev);
        xv[k] = qprev;
      }
#pragma unroll
      for (int k = 0; k < YB; k++) Q(i + k) = xv[k];
    }
    for (; i < n - 2; i++) {
      qprev = RV(i) * (Q(i) - l * qprev);
      Q(i) = qprev;
    }
    Q(n - 2) = (0. != lf) ? lf * (Q(n - 2) - l * qprev) : 0.;
    double qn = Q(n - 2);
    i = n - 3;
    for (; i - YB + 1 >= 0; i -= YB) {
      double xv[YB], vv[YB];
#pragma unroll
      for (int k = 0; k < YB; k++) {
        xv[k] = Q(i - k);
        vv[k] = V(i - k);
      }
#pragma unroll
      for (int k = 0; k < YB; k++) {
        qn = xv[k] - vv[k] * qn;
        xv[k] = qn;
      }
#pragma unroll
      for (int k = 0; k < YB; k++) Q(i - k) = xv[k];
    }
    for (; i >= 0; i--) {
      qn = Q(i) - V(i) * qn;
      Q(i) = qn;
    }
    // Sherman-Morrison correction
    const double num = Q(n - 1) - u * qn - l * Q(n - 2);
    const double qlast = fabs(d) < kDblEpsilon ? 0. : num / d;
    Q(n - 1) = qlast;
    sl[t] = qlast;
#undef Q
#undef V
#undef RV
  }
  __syncthreads();
  for (int w = threadIdx.x; w < n * kt; w += blockDim.x) {
    const int j = w / kt, tt = w - j * kt;
    if (tt < nk) {
      const size_t g = (size_t)j * nx + k0 + tt;
      spec[g] = (j < n - 1) ? sq[w] + sl[tt] * q1t[g] : sq[w];
    }
  }
}

// rows j0 .. j0 + ROWS - 1: REDFT01 then extract_output +
// fluid_update_boundaries_psi (the pre-twiddle pairs spectrum k and n - k;
// FFT point p is output position 2p below n/2, 2(n-1-p)+1 above)
template <int L2N>
__global__ void __launch_bounds__(DctShape<L2N>::THREADS) k_dct_inv(const double *__restrict__ spec, double *__restrict__ psi,
                                                        const double *__restrict__ tw, const double *__restrict__ cs,
                                                        Grid2 g) {
  pdl_enter();
  using S = DctShape<L2N>;
  constexpr int N = S::N, ROWS = S::ROWS, LD = S::LD;
  extern __shared__ double dsm[];
  double *re = dsm, *im = re + ROWS * LD, *in = im + ROWS * LD, *ro = in + ROWS * N;  // in, ro [ROWS][N]
  __shared__ double wold[4];  // old wall values of rows 1 and ny (left, right)
  const int nx = g.nx, ny = g.ny;
  const int j0 = 1 + blockIdx.x * ROWS;
  const int nr = min(ROWS, ny - j0 + 1);
  // old wall values of the rows that feed the halo, read before any write
  if (threadIdx.x < 4) {
    const int row = (threadIdx.x < 2) ? 1 : ny, side = threadIdx.x & 1;
    if (row >= j0 && row < j0 + nr) wold[threadIdx.x] = psi[ix_cc(nx, side ? nx + 1 : 0, row)];
  }
  // the spectrum rows, read in order (coalesced)
  for (int w = threadIdx.x; w < ROWS * N; w += S::THREADS) {
    const int c = w >> L2N;
    in[w] = (c < nr) ? spec[(size_t)(j0 - 1) * N + w] : 0.;
  }
  __syncthreads();
  auto first = [&](int c, int base, auto gc, auto hc, double *xr, double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int m = bitrev(base + q * H, L2N);
      const double a = in[c * N + m];
      const double b = (0 == m) ? 0. : in[c * N + N - m];
      const double2 w = __ldg(reinterpret_cast<const double2 *>(cs) + m);
      xr[q] = w.x * a + w.y * b;
      xi[q] = w.y * a - w.x * b;
    }
  };
  auto last = [&](int c, int base, auto gc, auto hc, const double *xr, const double *) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int p = base + q * H;
      const int o = (p < N / 2) ? 2 * p : 2 * (N - 1 - p) + 1;
      ro[c * N + o] = xr[q];
    }
  };
  svof_fft_dev::fft_lines<double, L2N, ROWS, 1, S::THREADS>(re, im, tw, first, last);
  __syncthreads();
  // psi rows with their halo images, written in order (coalesced)
  for (int w = threadIdx.x; w < nr * N; w += S::THREADS) {
    const int c = w >> L2N, i = (w & (N - 1)) + 1, j = j0 + c;
    const double y = ro[w];
    psi[ix_cc(nx, i, j)] = y;
    if (ny == j) psi[ix_cc(nx, i, 0)] = y;
    if (1 == j) psi[ix_cc(nx, i, ny + 1)] = y;
  }
  // Neumann walls, psi.c:7-20 (the wall takes its neighbour), and the halo
  // rows' wall cells, which take the walls' old values
  for (int c = threadIdx.x; c < nr; c += S::THREADS) {
    const int j = j0 + c;
    psi[ix_cc(nx, 0, j)] = ro[c * N];
    psi[ix_cc(nx, nx + 1, j)] = ro[c * N + N - 1];
    if (ny == j) {
      psi[ix_cc(nx, 0, 0)] = wold[2];
      psi[ix_cc(nx, nx + 1, 0)] = wold[3];
    }
    if (1 == j) {
      psi[ix_cc(nx, 0, ny + 1)] = wold[0];
      psi[ix_cc(nx, nx + 1, ny + 1)] = wold[1];
    }
  }
}

// ---- launch plans of the DCT row transforms, by length
namespace {
template <class F>
auto by_log2n(int l2n, F f) {
  switch (l2n) {
    case 2: return f(std::integral_constant<int, 2>());
    case 3: return f(std::integral_constant<int, 3>());
    case 4: return f(std::integral_constant<int, 4>());
    case 5: return f(std::integral_constant<int, 5>());
    case 6: return f(std::integral_constant<int, 6>());
    case 7: return f(std::integral_constant<int, 7>());
    case 8: return f(std::integral_constant<int, 8>());
    case 9: return f(std::integral_constant<int, 9>());
    case 10: return f(std::integral_constant<int, 10>());
    case 11: return f(std::integral_constant<int, 11>());
    default: return f(std::integral_constant<int, 12>());
  }
}
}  // namespace

bool dct_length_ok(int log2n) { return log2n >= kDctMinL2N && log2n <= kDctMaxL2N; }
int dct_rows(int log2n) {
  return by_log2n(log2n, [](auto c) { return DctShape<decltype(c)::value>::ROWS; });
}
int dct_threads(int log2n) {
  return by_log2n(log2n, [](auto c) { return DctShape<decltype(c)::value>::THREADS; });
}
size_t dct_smem(int log2n, bool inverse) {
  return by_log2n(log2n, [&](auto c) {
    using S = DctShape<decltype(c)::value>;
    return inverse ? S::SMEM_INV : S::SMEM_FWD;
  });
}
DctFwdKernel dct_fwd_kernel(int log2n) {
  return by_log2n(log2n, [](auto c) { return (DctFwdKernel)&k_dct_fwd<decltype(c)::value>; });
}
DctFwdRhsKernel dct_fwd_rhs_kernel(int log2n) {
  return by_log2n(log2n, [](auto c) { return (DctFwdRhsKernel)&k_dct_fwd_rhs<decltype(c)::value>; });
}
DctInvKernel dct_inv_kernel(int log2n) {
  return by_log2n(log2n, [](auto c) { return (DctInvKernel)&k_dct_inv<decltype(c)::value>; });
}
cudaError_t dct_prepare(int log2n) {
  if (!dct_length_ok(log2n)) return cudaErrorInvalidValue;
  cudaError_t e = raise_smem_limit(dct_fwd_kernel(log2n), dct_smem(log2n, false));
  if (cudaSuccess == e) e = raise_smem_limit(dct_fwd_rhs_kernel(log2n), dct_smem(log2n, false));
  if (cudaSuccess == e) e = raise_smem_limit(dct_inv_kernel(log2n), dct_smem(log2n, true));
  return e;
}

// ---------------------------------------------------------------- DFT path
// The spectrum is S[ky][i], complex, i fastest: the transforms read and write
// runs of consecutive i, the x solves (cline_solve.cuh) contiguous lines.  A
// block owns DftShape<L2N>::COLS consecutive columns i (N = ny = 2^L2N points
// each) and runs their transforms as the register-blocked passes of
// fft_device.cuh; the first pass evaluates the right-hand side (or reads the
// spectrum), the last one writes the results.  COLS: 4 (a 32-byte sector of a
// row) up to 1024 points, so that a 128-wide grid still makes 32 blocks and
// three blocks of a 1024-point one fit an SM; 2 and 1 columns above, for the
// same reason.  us a launch, forward and inverse, against tiles of up to 16
// columns with one stage per barrier: 128 x 256 10.5 / 7.3 against 33 / 26,
// 1501 x 2048 99 / 60 against 169 / 159 (x solves 9.8 against 15.5, 82 against
// 313).
template <int L2N>
struct DftShape {
  static constexpr int N = 1 << L2N;
  static constexpr int COLS = L2N <= 10 ? 4 : (L2N == 11 ? 2 : 1);
  static constexpr int PAIRS = COLS * (N >> (L2N < 3 ? L2N : 3));
  static constexpr int THREADS = PAIRS < 32 ? 32 : (PAIRS > 256 ? 256 : (PAIRS + 31) / 32 * 32);
  static constexpr int LD = svof_fft_dev::fft_ld(L2N);
  static constexpr size_t SMEM = sizeof(double) * COLS * 2 * (size_t)LD;
};

// columns i0 .. i0 + COLS - 1 of the right-hand side, r2c along y into spec
template <int L2N, class Rhs>
__device__ __forceinline__ void dft_fwd_cols(const Rhs &rhs, double *__restrict__ spec, const double *__restrict__ tw,
                                             int nx) {
  using S = DftShape<L2N>;
  constexpr int N = S::N, COLS = S::COLS, LD = S::LD;
  extern __shared__ double dsm[];
  double *re = dsm, *im = re + COLS * LD;
  const int i0 = 1 + blockIdx.x * COLS;
  const int nc = min(COLS, nx - i0 + 1);
  double2 *out = reinterpret_cast<double2 *>(spec) + (i0 - 1);
  auto first = [&](int c, int base, auto gc, auto hc, double *xr, double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
#pragma unroll
    for (int q = 0; q < G; q++) {
      xr[q] = (c < nc) ? rhs(i0 + c, bitrev(base + q * H, L2N) + 1) : 0.;
      xi[q] = 0.;
    }
  };
  auto last = [&](int c, int base, auto gc, auto hc, const double *xr, const double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
    if (c >= nc) return;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int k = base + q * H;
      if (k <= N / 2) out[(size_t)k * nx + c] = make_double2(xr[q], xi[q]);
    }
  };
  svof_fft_dev::fft_lines<double, L2N, COLS, 1, S::THREADS>(re, im, tw, first, last);
}

template <int L2N>
__global__ void __launch_bounds__(DftShape<L2N>::THREADS)
    k_dft_fwd(const double *__restrict__ ux, const double *__restrict__ uy, double *__restrict__ spec,
              const double *__restrict__ tw, const double *__restrict__ dtp, double gam, Grid2 g) {
  pdl_enter();
  const double dt = *dtp;
  const double prefactor = 1. / (gam * dt) / (1. * (1 << L2N));
  dft_fwd_cols<L2N>(DivRhs{ux, uy, g, prefactor}, spec, tw, g.nx);
}

template <int L2N>
__global__ void __launch_bounds__(DftShape<L2N>::THREADS)
    k_dft_fwd_rhs(const double *__restrict__ r, double *__restrict__ spec, const double *__restrict__ tw, Grid2 g) {
  dft_fwd_cols<L2N>(ArrayRhs{r, g.dxf, g.nx}, spec, tw, g.nx);
}

// c2r along y of COLS columns, extract_output and the psi boundaries
template <int L2N>
__global__ void __launch_bounds__(DftShape<L2N>::THREADS)
    k_dft_inv(const double *__restrict__ spec, double *__restrict__ psi, const double *__restrict__ tw, Grid2 g) {
  pdl_enter();
  using S = DftShape<L2N>;
  constexpr int N = S::N, COLS = S::COLS, LD = S::LD;
  extern __shared__ double dsm[];
  double *re = dsm, *im = re + COLS * LD;
  const int nx = g.nx;
  const int i0 = 1 + blockIdx.x * COLS;
  const int nc = min(COLS, nx - i0 + 1);
  const double2 *in = reinterpret_cast<const double2 *>(spec) + (i0 - 1);
  // Hermitian extension as FFTW's c2r reads it: Im of X_0 and X_{n/2} ignored
  auto first = [&](int c, int base, auto gc, auto hc, double *xr, double *xi) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int m = bitrev(base + q * H, L2N);
      double2 v = make_double2(0., 0.);
      if (c < nc) v = in[(size_t)(2 * m <= N ? m : N - m) * nx + c];
      xr[q] = v.x;
      xi[q] = (0 == m || 2 * m == N) ? 0. : (2 * m < N ? v.y : -v.y);
    }
  };
  auto last = [&](int c, int base, auto gc, auto hc, const double *xr, const double *) {
    constexpr int G = decltype(gc)::value, H = decltype(hc)::value;
    if (c >= nc) return;
#pragma unroll
    for (int q = 0; q < G; q++) {
      const int j = base + q * H + 1;
      psi[ix_cc(nx, i0 + c, j)] = xr[q];
      if (N == j) psi[ix_cc(nx, i0 + c, 0)] = xr[q];
      if (1 == j) psi[ix_cc(nx, i0 + c, N + 1)] = xr[q];
    }
  };
  svof_fft_dev::fft_lines<double, L2N, COLS, 1, S::THREADS>(re, im, tw, first, last);
  // Neumann walls, psi.c:7-20 (the blocks at either end of x): the wall cell
  // takes its neighbour's new value, read back after the barrier, and hands
  // its old value to the halo row's wall cell
  const bool has_left = (1 == i0), has_right = (i0 + nc - 1 == nx);
  if (!has_left && !has_right) return;
  __syncthreads();
  for (int w = threadIdx.x; w < 2 * N; w += S::THREADS) {
    const int side = w >> L2N, j = 1 + (w & (N - 1));
    if (side ? !has_right : !has_left) continue;
    const int iw = side ? nx + 1 : 0;
    const double old = psi[ix_cc(nx, iw, j)];
    psi[ix_cc(nx, iw, j)] = psi[ix_cc(nx, side ? nx : 1, j)];
    if (N == j) psi[ix_cc(nx, iw, 0)] = old;
    if (1 == j) psi[ix_cc(nx, iw, N + 1)] = old;
  }
}

// ---- launch plans of the DFT column transforms, by length
namespace {
template <class F>
auto dft_by_log2n(int l2n, F f) {
  if (13 == l2n) return f(std::integral_constant<int, 13>());
  return by_log2n(l2n, f);
}
}  // namespace

bool dft_length_ok(int log2n) { return log2n >= kDctMinL2N && log2n <= kDftMaxL2N; }
int dft_cols(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return DftShape<decltype(c)::value>::COLS; });
}
int dft_threads(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return DftShape<decltype(c)::value>::THREADS; });
}
size_t dft_smem(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return DftShape<decltype(c)::value>::SMEM; });
}
DftFwdKernel dft_fwd_kernel(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return (DftFwdKernel)&k_dft_fwd<decltype(c)::value>; });
}
DftFwdRhsKernel dft_fwd_rhs_kernel(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return (DftFwdRhsKernel)&k_dft_fwd_rhs<decltype(c)::value>; });
}
DftInvKernel dft_inv_kernel(int log2n) {
  return dft_by_log2n(log2n, [](auto c) { return (DftInvKernel)&k_dft_inv<decltype(c)::value>; });
}
DftXSolveKernel dft_xsolve_kernel(long nlines, int nx) {
  return svof_cline::cline_by_lpb(svof_cline::cline_lpb(nlines, nx, sizeof(double)), [](auto c) {
    return (DftXSolveKernel)&svof_cline::k_cline_solve<double, decltype(c)::value>;
  });
}
int dft_xsolve_lines(long nlines, int nx) { return svof_cline::cline_lpb(nlines, nx, sizeof(double)); }
size_t dft_xsolve_smem(long nlines, int nx) {
  return svof_cline::cline_smem(dft_xsolve_lines(nlines, nx), nx, sizeof(double));
}
cudaError_t dft_prepare(int log2n, int nx) {
  if (!dft_length_ok(log2n)) return cudaErrorInvalidValue;
  cudaError_t e = raise_smem_limit(dft_fwd_kernel(log2n), dft_smem(log2n));
  if (cudaSuccess == e) e = raise_smem_limit(dft_fwd_rhs_kernel(log2n), dft_smem(log2n));
  if (cudaSuccess == e) e = raise_smem_limit(dft_inv_kernel(log2n), dft_smem(log2n));
  if (cudaSuccess == e) e = svof_cline::cline_prepare<double>((1L << log2n) / 2 + 1, nx);
  return e;
}
cudaError_t dft_pivots(cudaStream_t st, double *tab, const double *pl, const double *pu, const double *evals, int nx,
                       int nky) {
  using namespace svof_cline;
  k_cline_table<<<(nky + kTabLines - 1) / kTabLines, kTabLines, 0, st>>>(tab, pl, pu, evals, nullptr, nky, nky, nx,
                                                                        nullptr);
  return cudaGetLastError();
}

}  // namespace svof
