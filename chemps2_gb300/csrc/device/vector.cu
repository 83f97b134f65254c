// Vector kernels of the Davidson eigensolver (FP64, deterministic reductions).
#include "kernels.cuh"

#include <cmath>

namespace c2g {

namespace {

// ---------------------------------------------------------------- vector kernels

template <int MAXC>
__global__ void __launch_bounds__(kDotThreads) multi_dot_kernel(const double* __restrict__ A, int64_t lda, int ncol,
                                                                const double* __restrict__ x, int64_t n,
                                                                double* __restrict__ partial) {
  double acc[MAXC];
#pragma unroll
  for (int j = 0; j < MAXC; j++) acc[j] = 0.0;
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t start = chunk * blockIdx.x;
  const int64_t end = (start + chunk < n) ? start + chunk : n;
  for (int64_t i = start + threadIdx.x; i < end; i += blockDim.x) {
    const double xi = x[i];
#pragma unroll
    for (int j = 0; j < MAXC; j++)
      if (j < ncol) acc[j] = fma(A[i + lda * j], xi, acc[j]);
  }
  __shared__ double red[kDotThreads / 32][MAXC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < MAXC; j++) {
    if (j >= ncol) break;
    double v = acc[j];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][j] = v;
  }
  __syncthreads();
  if (threadIdx.x < ncol) {
    double v = 0.0;
    for (int w = 0; w < kDotThreads / 32; w++) v += red[w][threadIdx.x];
    partial[static_cast<int64_t>(blockIdx.x) * ncol + threadIdx.x] = v;
  }
}

__global__ void reduce_partials_kernel(const double* __restrict__ partial, int nblk, int ncol, double* __restrict__ out) {
  const int j = threadIdx.x;
  if (j >= ncol) return;
  double v = 0.0;
  for (int b = 0; b < nblk; b++) v += partial[static_cast<int64_t>(b) * ncol + j];
  out[j] = v;
}

__global__ void combine_kernel(double* __restrict__ out, double beta, const double* __restrict__ A, int64_t lda,
                               const double* __restrict__ coef, int ncol, int64_t n) {
  __shared__ double c[64];
  if (threadIdx.x < ncol) c[threadIdx.x] = coef[threadIdx.x];
  __syncthreads();
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double v = (beta == 0.0) ? 0.0 : beta * out[i];
    for (int j = 0; j < ncol; j++) v = fma(c[j], A[i + lda * j], v);
    out[i] = v;
  }
}

__global__ void scale_kernel(double* x, double s, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    x[i] *= s;
}

__global__ void axpy_kernel(double* y, double a, const double* x, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    y[i] = fma(a, x[i], y[i]);
}

__global__ void fill_kernel(double* x, double v, int64_t n) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    x[i] = v;
}

// dst[:, j] = sign_j * src[:, cols - 1 - j], one CTA per column. sign_j makes the entry of
// largest magnitude (the first one on ties) positive, which fixes the gauge of each
// eigenvector so that every executor produces the same singular vectors.
__global__ void reverse_columns_kernel(double* __restrict__ dst, const double* __restrict__ src, int rows, int cols) {
  const int j = blockIdx.x;
  if (j >= cols) return;
  const double* col = src + static_cast<int64_t>(rows) * (cols - 1 - j);
  double best = -1.0;
  int bi = 0;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) {
    const double a = fabs(col[i]);
    if (a > best) {
      best = a;
      bi = i;
    }
  }
  __shared__ double sb[256];
  __shared__ int si[256];
  sb[threadIdx.x] = best;
  si[threadIdx.x] = bi;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      const double b2 = sb[threadIdx.x + o];
      const int i2 = si[threadIdx.x + o];
      if (b2 > sb[threadIdx.x] || (b2 == sb[threadIdx.x] && i2 < si[threadIdx.x])) {
        sb[threadIdx.x] = b2;
        si[threadIdx.x] = i2;
      }
    }
    __syncthreads();
  }
  const double sgn = (col[si[0]] < 0.0) ? -1.0 : 1.0;
  double* out = dst + static_cast<int64_t>(rows) * j;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) out[i] = sgn * col[i];
}

// t -= evals[0] * u   (CheMPS2/Davidson.cpp:280-283)
__global__ void residual_kernel(double* t, const double* u, const double* evals, int64_t n) {
  const double lam = evals[0];
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    t[i] = fma(-lam, u[i], t[i]);
}

__device__ __forceinline__ double precond_den(double d, double cutoff) {
  return (fabs(d) > cutoff) ? d : cutoff;
}

// w = K^-1 u   (CheMPS2/Davidson.cpp:294-305)
__global__ void precond_w_kernel(double* w, const double* u, const double* diag, const double* evals, double cutoff,
                                 int64_t n) {
  const double shift = evals[0];
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    w[i] = u[i] / precond_den(diag[i] - shift, cutoff);
}

// t = -K^-1 (t + alpha u), alpha = -(w.t)/(w.u)   (CheMPS2/Davidson.cpp:306-316)
__global__ void precond_t_kernel(double* t, const double* u, const double* diag, const double* evals,
                                 const double* dots2, double cutoff, int64_t n) {
  const double shift = evals[0];
  const double alpha = -dots2[0] / dots2[1];
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double v = fma(alpha, u[i], t[i]);
    t[i] = -v / precond_den(diag[i] - shift, cutoff);
  }
}

__global__ void neg_kernel(double* c, int n) {
  if (threadIdx.x < n) c[threadIdx.x] = -c[threadIdx.x];
}

__global__ void inv_sqrt_scale_kernel(double* x, const double* sumsq, int64_t n) {
  const double s = 1.0 / sqrt(sumsq[0]);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    x[i] *= s;
}

__global__ void mxm_row_kernel(double* mxm, int ld, int row, const double* dots, int ncol) {
  const int c = threadIdx.x;
  if (c < ncol) {
    mxm[c + ld * row] = dots[c];
    mxm[row + ld * c] = dots[c];
  }
}

inline int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 8) b = 152 * 8;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace

cudaError_t launch_multi_dot(const double* A, int64_t lda, int ncol, const double* x, int64_t n, double* partial,
                             double* out, cudaStream_t stream) {
  if (ncol <= 0) return cudaSuccess;
  if (ncol > 32) return cudaErrorInvalidValue;
  if (ncol <= 4)
    multi_dot_kernel<4><<<kDotBlocks, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial);
  else if (ncol <= 8)
    multi_dot_kernel<8><<<kDotBlocks, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial);
  else
    multi_dot_kernel<32><<<kDotBlocks, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial);
  reduce_partials_kernel<<<1, 32, 0, stream>>>(partial, kDotBlocks, ncol, out);
  return cudaGetLastError();
}

cudaError_t launch_combine(double* out, double beta, const double* A, int64_t lda, const double* coef, int ncol,
                           int64_t n, cudaStream_t stream) {
  if (ncol > 64) return cudaErrorInvalidValue;
  if (n <= 0) return cudaSuccess;
  combine_kernel<<<grid_for(n), 256, 0, stream>>>(out, beta, A, lda, coef, ncol, n);
  return cudaGetLastError();
}

cudaError_t launch_norm2(const double* x, int64_t n, double* partial, double* out, cudaStream_t stream) {
  return launch_multi_dot(x, n, 1, x, n, partial, out, stream);
}

cudaError_t launch_scale(double* x, double s, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  scale_kernel<<<grid_for(n), 256, 0, stream>>>(x, s, n);
  return cudaGetLastError();
}

cudaError_t launch_axpy(double* y, double a, const double* x, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  axpy_kernel<<<grid_for(n), 256, 0, stream>>>(y, a, x, n);
  return cudaGetLastError();
}

cudaError_t launch_fill(double* x, double v, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  fill_kernel<<<grid_for(n), 256, 0, stream>>>(x, v, n);
  return cudaGetLastError();
}

cudaError_t launch_reverse_columns(double* dst, const double* src, int rows, int cols, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  reverse_columns_kernel<<<cols, 256, 0, stream>>>(dst, src, rows, cols);
  return cudaGetLastError();
}

cudaError_t launch_residual(double* t, const double* u, const double* evals, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  residual_kernel<<<grid_for(n), 256, 0, stream>>>(t, u, evals, n);
  return cudaGetLastError();
}

cudaError_t launch_precond_w(double* w, const double* u, const double* diag, const double* evals, double cutoff,
                             int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  precond_w_kernel<<<grid_for(n), 256, 0, stream>>>(w, u, diag, evals, cutoff, n);
  return cudaGetLastError();
}

cudaError_t launch_precond_t(double* t, const double* u, const double* diag, const double* evals,
                             const double* dots2, double cutoff, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  precond_t_kernel<<<grid_for(n), 256, 0, stream>>>(t, u, diag, evals, dots2, cutoff, n);
  return cudaGetLastError();
}

cudaError_t launch_neg(double* c, int n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  neg_kernel<<<1, 64, 0, stream>>>(c, n);
  return cudaGetLastError();
}

cudaError_t launch_inv_sqrt_scale(double* x, const double* sumsq, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  inv_sqrt_scale_kernel<<<grid_for(n), 256, 0, stream>>>(x, sumsq, n);
  return cudaGetLastError();
}

cudaError_t launch_mxm_row(double* mxm, int ld, int row, const double* dots, int ncol, cudaStream_t stream) {
  mxm_row_kernel<<<1, 64, 0, stream>>>(mxm, ld, row, dots, ncol);
  return cudaGetLastError();
}

}  // namespace c2g
