// The sparse and dense kernels of the algebraic coarse levels.
#include <algorithm>

#include "lpg_common.cuh"
#include "lpg_internal.hpp"

namespace lpg {

// ---------------------------------------------------------------- CSR (AMG levels)
// Eight lanes per row: AMG rows of the N=1 hierarchy hold ~7-30 nonzeros.
constexpr int kLanesPerRow = 8;

__global__ void __launch_bounds__(256)
csr_spmv_kernel(const int64_t Nrows, const int64_t* __restrict__ rs, const int32_t* __restrict__ cols,
                const double* __restrict__ vals, const double alpha, const double* __restrict__ x,
                const double beta, double* __restrict__ y) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kLanesPerRow;
  const int lane = threadIdx.x % kLanesPerRow;
  double acc = 0;
  if (row < Nrows)
    for (int64_t jj = rs[row] + lane; jj < rs[row + 1]; jj += kLanesPerRow) acc += vals[jj] * x[cols[jj]];
  for (int o = kLanesPerRow / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, kLanesPerRow);
  if (row < Nrows && lane == 0) y[row] = (beta != 0.0) ? alpha * acc + beta * y[row] : alpha * acc;
}

int csr_spmv(int64_t Nrows, const int64_t* rowStarts, const int32_t* cols, const double* vals, double alpha,
             const double* x, double beta, double* y, cudaStream_t s) {
  if (Nrows <= 0) return LPG_OK;
  const int64_t threads = Nrows * kLanesPerRow;
  csr_spmv_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(Nrows, rowStarts, cols, vals, alpha, x,
                                                                    beta, y);
  LPG_LAUNCH_CHECK("csr_spmv_kernel");
  return LPG_OK;
}

__global__ void csr_cheb_start_kernel(const int64_t N, const double invTheta, const double* __restrict__ diagInv,
                                      const double* __restrict__ b, double* __restrict__ r,
                                      double* __restrict__ d, double* __restrict__ x) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < N; n += (int64_t)gridDim.x * blockDim.x) {
    const double rr = diagInv[n] * b[n];
    r[n] = rr;
    d[n] = invTheta * rr;
    x[n] = invTheta * rr;
  }
}
int csr_cheb_start(int64_t N, double invTheta, const double* diagInv, const double* b, double* r, double* d,
                   double* x, cudaStream_t s) {
  if (N <= 0) return LPG_OK;
  csr_cheb_start_kernel<<<(unsigned)std::min<int64_t>((N + 255) / 256, 4096), 256, 0, s>>>(N, invTheta, diagInv, b,
                                                                                          r, d, x);
  LPG_LAUNCH_CHECK("csr_cheb_start_kernel");
  return LPG_OK;
}

// r = alpha r + D^{-1} (beta b - A x)
__global__ void __launch_bounds__(256)
csr_cheb_residual_kernel(const int64_t Nrows, const int64_t* __restrict__ rs, const int32_t* __restrict__ cols,
                         const double* __restrict__ vals, const double alpha, const double beta,
                         const double* __restrict__ diagInv, const double* __restrict__ b,
                         const double* __restrict__ x, double* __restrict__ r) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kLanesPerRow;
  const int lane = threadIdx.x % kLanesPerRow;
  double acc = 0;
  if (row < Nrows)
    for (int64_t jj = rs[row] + lane; jj < rs[row + 1]; jj += kLanesPerRow) acc += vals[jj] * x[cols[jj]];
  for (int o = kLanesPerRow / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, kLanesPerRow);
  if (row < Nrows && lane == 0) {
    const double res = ((beta != 0.0) ? beta * b[row] : 0.0) - acc;
    const double rk = (alpha != 0.0) ? alpha * r[row] : 0.0;
    r[row] = rk + diagInv[row] * res;
  }
}
int csr_cheb_residual(int64_t N, const int64_t* rowStarts, const int32_t* cols, const double* vals, double alpha,
                      double beta, const double* diagInv, const double* b, const double* x, double* r,
                      cudaStream_t s) {
  if (N <= 0) return LPG_OK;
  const int64_t threads = N * kLanesPerRow;
  csr_cheb_residual_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(N, rowStarts, cols, vals, alpha,
                                                                             beta, diagInv, b, x, r);
  LPG_LAUNCH_CHECK("csr_cheb_residual_kernel");
  return LPG_OK;
}

// d = a d + b r ; x += d   (SmoothChebyshevUpdate)
__global__ void csr_cheb_update_kernel(const int64_t N, const double a, const double b, const int lastIt,
                                       const double* __restrict__ r, double* __restrict__ d,
                                       double* __restrict__ x) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < N; n += (int64_t)gridDim.x * blockDim.x) {
    const double dk = (a != 0.0) ? d[n] : 0.0;
    const double dn = a * dk + b * r[n];
    if (!lastIt) d[n] = dn;
    x[n] += dn;
  }
}
int csr_cheb_update(int64_t N, double a, double b, int lastIt, const double* r, double* d, double* x,
                    cudaStream_t s) {
  if (N <= 0) return LPG_OK;
  csr_cheb_update_kernel<<<(unsigned)std::min<int64_t>((N + 255) / 256, 4096), 256, 0, s>>>(N, a, b, lastIt, r,
                                                                                           d, x);
  LPG_LAUNCH_CHECK("csr_cheb_update_kernel");
  return LPG_OK;
}

// The level cycle's passes: a matrix product and the vector updates of its rows in one kernel,
// the vectors that other rows still read written out of place. Each of these kernels is
// bound by latency, so fewer are faster: mixed FPCG solve, 32^3, N = 7 16.43 -> 15.97 ms.
// LANES threads a row, 32 where the rows hold more than 48 entries on average. 8 against 32, us:
// rows of 18 entries (29,791 of them) 9.6 against 22.6; of 69 (2,827) 8.1 against 7.6; the
// restrictions of smoothed aggregation, hundreds of entries a row, to 2,827 rows 12.0
// against 6.2, to 209 rows 23.0 against 8.1.
template <int LANES>
__device__ __forceinline__ double csr_row(const int64_t row, const int64_t n, const int64_t* __restrict__ rs,
                                          const int32_t* __restrict__ cols, const double* __restrict__ vals,
                                          const double* __restrict__ x) {
  double acc = 0;
  if (row < n)
    for (int64_t jj = rs[row] + threadIdx.x % LANES; jj < rs[row + 1]; jj += LANES) acc += vals[jj] * x[cols[jj]];
  for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, LANES);
  return acc;   // the row's first lane
}
// MODE 0: y = A x; 1: y = b - A x; 2: y += A x;
// 3: r = diagInv (b - A x), d = c1 r, y = x + d (the smoother's start on x);
// 4: r -= diagInv (A x), y = c0 x + c1 r, sol = z + y (a step with d = x; LAST: r, y not stored)
template <int LANES, int MODE, bool LAST>
__global__ void __launch_bounds__(256)
csr_pass_kernel(const int64_t n, const int64_t* __restrict__ rs, const int32_t* __restrict__ cols,
                const double* __restrict__ vals, const double* __restrict__ diagInv, const double c0, const double c1,
                const double* __restrict__ b, const double* __restrict__ x, double* __restrict__ r,
                double* __restrict__ y, const double* z, double* sol) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
  const double acc = csr_row<LANES>(row, n, rs, cols, vals, x);
  if (row >= n || threadIdx.x % LANES) return;
  if constexpr (MODE == 0) y[row] = acc;
  if constexpr (MODE == 1) y[row] = b[row] - acc;
  if constexpr (MODE == 2) y[row] += acc;
  if constexpr (MODE == 3) {
    const double rk = diagInv[row] * (b[row] - acc), d = c1 * rk;
    r[row] = rk;
    y[row] = d;
    sol[row] = x[row] + d;
  }
  if constexpr (MODE == 4) {
    const double rk = r[row] - diagInv[row] * acc, d = c0 * x[row] + c1 * rk;
    if (!LAST) {
      r[row] = rk;
      y[row] = d;
    }
    sol[row] = z[row] + d;
  }
}
template <int MODE, bool LAST = false>
static int csr_pass(const CsrView& A, const double* diagInv, double c0, double c1, const double* b, const double* x,
                    double* r, double* y, const double* z, double* sol, cudaStream_t s) {
  if (A.n <= 0) return LPG_OK;
  const unsigned blocks = (unsigned)((A.n * (A.longRows ? 32 : kLanesPerRow) + 255) / 256);
  if (A.longRows)
    csr_pass_kernel<32, MODE, LAST><<<blocks, 256, 0, s>>>(A.n, A.rowStarts, A.cols, A.vals, diagInv, c0, c1, b, x, r, y,
                                                          z, sol);
  else
    csr_pass_kernel<kLanesPerRow, MODE, LAST><<<blocks, 256, 0, s>>>(A.n, A.rowStarts, A.cols, A.vals, diagInv, c0, c1,
                                                                    b, x, r, y, z, sol);
  LPG_LAUNCH_CHECK("csr_pass_kernel");
  return LPG_OK;
}
int csr_product(const CsrView& A, const double* x, double* y, cudaStream_t s) {
  return csr_pass<0>(A, nullptr, 0, 0, nullptr, x, nullptr, y, nullptr, nullptr, s);
}
int csr_product_add(const CsrView& A, const double* x, double* y, cudaStream_t s) {
  return csr_pass<2>(A, nullptr, 0, 0, nullptr, x, nullptr, y, nullptr, nullptr, s);
}
int csr_residual(const CsrView& A, const double* b, const double* x, double* res, cudaStream_t s) {
  return csr_pass<1>(A, nullptr, 0, 0, b, x, nullptr, res, nullptr, nullptr, s);
}
int csr_cheb_restart(const CsrView& A, const double* diagInv, double invTheta, const double* b, const double* x,
                     double* r, double* d, double* xOut, cudaStream_t s) {
  return csr_pass<3>(A, diagInv, 0, invTheta, b, x, r, d, nullptr, xOut, s);
}
int csr_cheb_step(const CsrView& A, const double* diagInv, double a, double b, const double* d, double* r, double* dOut,
                  const double* x, double* xOut, cudaStream_t s) {
  return dOut ? csr_pass<4>(A, diagInv, a, b, nullptr, d, r, dOut, x, xOut, s)
              : csr_pass<4, true>(A, diagInv, a, b, nullptr, d, r, nullptr, x, xOut, s);
}

// ---------------------------------------------------------------- dense coarse solve
// One warp per row of the dense inverse (parAlmond okl/dGEMV.okl).
__global__ void __launch_bounds__(256)
gemv_kernel(const int64_t n, const double* __restrict__ A, const double* __restrict__ x, double* __restrict__ y) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  double acc = 0;
  for (int64_t j = lane; j < n; j += 32) acc += A[row * n + j] * x[j];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (lane == 0) y[row] = acc;
}
int gemv(int64_t n, const double* A, const double* x, double* y, cudaStream_t s) {
  if (n <= 0) return LPG_OK;
  gemv_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(n, A, x, y);
  LPG_LAUNCH_CHECK("gemv_kernel");
  return LPG_OK;
}

}  // namespace lpg
