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
