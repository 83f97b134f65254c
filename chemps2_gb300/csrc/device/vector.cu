// Vector kernels of the Davidson eigensolver (FP64, deterministic reductions).
#include "kernels.cuh"

#include <math_constants.h>

#include <cmath>

namespace c2g {

namespace {

// ---------------------------------------------------------------- vector kernels

// The vector work of a Davidson iteration is a few passes over vectors that a small chain
// holds in cache, so its cost there is launches: each kernel does all that one pass over
// its vectors allows, and the sums are finished by the last CTA to arrive (in CTA order, so
// they do not depend on the arrival) instead of a second kernel. An L = 8 iteration took 24
// launches and a 12 us serial sum for each of its six dot products; it takes 8.
//
// FP64 adds are what a sum costs on this GPU (1.6 a clock and SM): a warp's sums of C
// columns exchange halves of the columns, C - 1 adds a lane instead of 5 C.

// Sums acc[0 .. C) over the warp: afterwards acc[0] of lane l is column l % C's total.
template <int C>
__device__ __forceinline__ void warp_columns(double (&acc)[C]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = C / 2; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (int j = 0; j < h; j++) {
      const double send = up ? acc[j] : acc[j + h], keep = up ? acc[j + h] : acc[j];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
#pragma unroll
  for (int o = C; o < 32; o <<= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
}

// Sums the threads' acc[0 .. ncol) over the grid. True in the CTA that has them, where
// thread j < ncol gets column j's sum in `total`. partial: gridDim.x x ncol doubles;
// counter: zero between launches.
template <int C>
__device__ __forceinline__ bool grid_columns(double (&acc)[C], int ncol, double* partial, unsigned int* counter,
                                             double& total) {
  constexpr int kWarps = kDotThreads / 32;
  __shared__ double red[kWarps][C];
  __shared__ unsigned int last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  warp_columns<C>(acc);
  if (lane < C) red[warp][lane] = acc[0];
  __syncthreads();
  total = 0.0;
  if (tid < ncol)
    for (int w = 0; w < kWarps; w++) total += red[w][tid];
  if (gridDim.x == 1) return true;
  if (tid < ncol) __stcg(partial + static_cast<int64_t>(blockIdx.x) * ncol + tid, total);
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // a warp per column: 32 strided sums, then a tree
  for (int j = warp; j < ncol; j += kWarps) {
    double v = 0.0;
    for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) v += __ldcg(partial + static_cast<int64_t>(b) * ncol + j);
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[0][j] = v;
  }
  if (tid == 0) *counter = 0u;
  __syncthreads();
  if (tid < ncol) total = red[0][tid];
  return true;
}

// Where a kernel's sums go: out[j], and with mxm the row and column `row` of that matrix.
struct SumOut {
  double* out;
  double* mxm;
  int ld, row;
  __device__ __forceinline__ void put(int j, double v) const {
    if (out) out[j] = v;
    if (mxm) {
      mxm[j + ld * row] = v;
      mxm[row + ld * j] = v;
    }
  }
};

// out[j] = A[:, j] . x
template <int C>
__global__ void __launch_bounds__(kDotThreads) multi_dot_kernel(const double* __restrict__ A, int64_t lda, int ncol,
                                                                const double* __restrict__ x, int64_t n,
                                                                double* partial, unsigned int* counter, SumOut o) {
  double acc[C];
#pragma unroll
  for (int j = 0; j < C; j++) acc[j] = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads) {
    const double xi = x[i];
#pragma unroll
    for (int j = 0; j < C; j++)
      if (j < ncol) acc[j] = fma(A[i + lda * j], xi, acc[j]);
  }
  double v;
  if (grid_columns<C>(acc, ncol, partial, counter, v) && threadIdx.x < ncol) o.put(threadIdx.x, v);
}

// out[0] = the lowest diag[i] over x[i] != 0 (inf if there is none)
__global__ void __launch_bounds__(kDotThreads) lowest_entry_kernel(const double* __restrict__ diag,
                                                                   const double* __restrict__ x, int64_t n,
                                                                   double* partial, unsigned int* counter,
                                                                   double* out) {
  constexpr int kWarps = kDotThreads / 32;
  __shared__ double red[kWarps];
  __shared__ unsigned int last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double v = CUDART_INF;
  auto block = [&] {  // the CTA's lowest, in thread 0
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (tid == 0)
      for (int w = 1; w < kWarps; w++) v = fmin(v, red[w]);
  };
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + tid; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads)
    if (x[i] != 0.0) v = fmin(v, diag[i]);
  block();
  if (tid == 0) {
    __stcg(partial + blockIdx.x, v);
    __threadfence();
    last = atomicAdd(counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  v = CUDART_INF;
  for (int b = tid; b < static_cast<int>(gridDim.x); b += kDotThreads) v = fmin(v, __ldcg(partial + b));
  block();
  if (tid == 0) {
    out[0] = v;
    *counter = 0u;
  }
}

// t -= A coef, then out[j] = A[:, j] . t (kNorm: out[0] = t . t instead)
template <int C, bool kNorm>
__global__ void __launch_bounds__(kDotThreads) subtract_kernel(double* __restrict__ t, const double* __restrict__ A,
                                                               int64_t lda, const double* __restrict__ coef, int ncol,
                                                               int64_t n, double* partial, unsigned int* counter,
                                                               SumOut o) {
  constexpr int S = kNorm ? 1 : C;
  __shared__ double c[C];
  if (threadIdx.x < C) c[threadIdx.x] = static_cast<int>(threadIdx.x) < ncol ? coef[threadIdx.x] : 0.0;
  __syncthreads();
  double acc[S];
#pragma unroll
  for (int j = 0; j < S; j++) acc[j] = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads) {
    double a[C], v = t[i];
#pragma unroll
    for (int j = 0; j < C; j++) a[j] = j < ncol ? A[i + lda * j] : 0.0;
#pragma unroll
    for (int j = 0; j < C; j++)
      if (j < ncol) v = fma(-c[j], a[j], v);
    t[i] = v;
    if constexpr (kNorm) {
      acc[0] = fma(v, v, acc[0]);
    } else {
#pragma unroll
      for (int j = 0; j < C; j++)
        if (j < ncol) acc[j] = fma(a[j], v, acc[j]);
    }
  }
  double v;
  const int nsum = kNorm ? 1 : ncol;
  if (grid_columns<S>(acc, nsum, partial, counter, v) && static_cast<int>(threadIdx.x) < nsum) o.put(threadIdx.x, v);
}

// u = V coef, t = HV coef - evals[0] u, out[0] = t . t   (CheMPS2/Davidson.cpp:277-288)
__global__ void __launch_bounds__(kDotThreads) ritz_kernel(double* __restrict__ t, double* __restrict__ u,
                                                           const double* __restrict__ HV, const double* __restrict__ V,
                                                           int64_t lda, const double* __restrict__ coef, int ncol,
                                                           const double* __restrict__ evals, int64_t n,
                                                           double* partial, unsigned int* counter, SumOut o) {
  __shared__ double c[64];
  if (static_cast<int>(threadIdx.x) < ncol) c[threadIdx.x] = coef[threadIdx.x];
  __syncthreads();
  const double lam = evals[0];
  double acc[1] = {0.0};
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads) {
    double x = 0.0, y = 0.0;
#pragma unroll 4
    for (int j = 0; j < ncol; j++) {
      x = fma(c[j], V[i + lda * j], x);
      y = fma(c[j], HV[i + lda * j], y);
    }
    y = fma(-lam, x, y);
    u[i] = x;
    t[i] = y;
    acc[0] = fma(y, y, acc[0]);
  }
  double v;
  if (grid_columns<1>(acc, 1, partial, counter, v) && threadIdx.x == 0) o.put(0, v);
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

__device__ __forceinline__ double precond_den(double d, double cutoff) {
  return (fabs(d) > cutoff) ? d : cutoff;
}

// w . t and w . u of w = K^-1 u   (CheMPS2/Davidson.cpp:294-305)
__global__ void __launch_bounds__(kDotThreads) precond_dots_kernel(const double* __restrict__ t,
                                                                   const double* __restrict__ u,
                                                                   const double* __restrict__ diag,
                                                                   const double* __restrict__ evals, double cutoff,
                                                                   int64_t n, double* partial, unsigned int* counter,
                                                                   SumOut o) {
  const double shift = evals[0];
  double acc[2] = {0.0, 0.0};
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads) {
    const double x = u[i], w = x / precond_den(diag[i] - shift, cutoff);
    acc[0] = fma(w, t[i], acc[0]);
    acc[1] = fma(w, x, acc[1]);
  }
  double v;
  if (grid_columns<2>(acc, 2, partial, counter, v) && threadIdx.x < 2) o.put(threadIdx.x, v);
}

// t = -K^-1 (t + alpha u), alpha = -(w.t)/(w.u)   (CheMPS2/Davidson.cpp:306-316), then
// out[j] = A[:, j] . t
template <int C>
__global__ void __launch_bounds__(kDotThreads) precond_kernel(double* __restrict__ t, const double* __restrict__ u,
                                                              const double* __restrict__ diag,
                                                              const double* __restrict__ evals,
                                                              const double* __restrict__ dots2, double cutoff,
                                                              const double* __restrict__ A, int64_t lda, int ncol,
                                                              int64_t n, double* partial, unsigned int* counter,
                                                              SumOut o) {
  const double shift = evals[0];
  const double alpha = -dots2[0] / dots2[1];
  double acc[C];
#pragma unroll
  for (int j = 0; j < C; j++) acc[j] = 0.0;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kDotThreads) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * kDotThreads) {
    const double v = -fma(alpha, u[i], t[i]) / precond_den(diag[i] - shift, cutoff);
    t[i] = v;
#pragma unroll
    for (int j = 0; j < C; j++)
      if (j < ncol) acc[j] = fma(A[i + lda * j], v, acc[j]);
  }
  double v;
  if (grid_columns<C>(acc, ncol, partial, counter, v) && static_cast<int>(threadIdx.x) < ncol) o.put(threadIdx.x, v);
}

// dst = x / sqrt(sumsq)
__global__ void normalize_kernel(double* __restrict__ dst, const double* __restrict__ x,
                                 const double* __restrict__ sumsq, int64_t n) {
  const double s = 1.0 / sqrt(sumsq[0]);
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[i] = x[i] * s;
}

inline int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 8) b = 152 * 8;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace

namespace {

// CTAs of the summing kernels: one element a thread until the SMs are full
int dot_grid(int64_t n) {
  const int64_t b = (n + kDotThreads - 1) / kDotThreads;
  return static_cast<int>(b < 1 ? 1 : b > kDotBlocks ? kDotBlocks : b);
}

unsigned int* dot_counter(double* partial) { return reinterpret_cast<unsigned int*>(partial + kDotCounter); }

cudaError_t dots_into(const double* A, int64_t lda, int ncol, const double* x, int64_t n, double* partial, SumOut o,
                      cudaStream_t stream) {
  if (ncol <= 0) return cudaSuccess;
  if (ncol > 32) return cudaErrorInvalidValue;
  const int g = dot_grid(n);
  unsigned int* ctr = dot_counter(partial);
  if (ncol <= 1)
    multi_dot_kernel<1><<<g, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial, ctr, o);
  else if (ncol <= 4)
    multi_dot_kernel<4><<<g, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial, ctr, o);
  else if (ncol <= 8)
    multi_dot_kernel<8><<<g, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial, ctr, o);
  else if (ncol <= 16)
    multi_dot_kernel<16><<<g, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial, ctr, o);
  else
    multi_dot_kernel<32><<<g, kDotThreads, 0, stream>>>(A, lda, ncol, x, n, partial, ctr, o);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_multi_dot(const double* A, int64_t lda, int ncol, const double* x, int64_t n, double* partial,
                             double* out, cudaStream_t stream) {
  return dots_into(A, lda, ncol, x, n, partial, SumOut{out, nullptr, 0, 0}, stream);
}

cudaError_t launch_project_row(const double* A, int64_t lda, int ncol, const double* x, int64_t n, double* partial,
                               double* mxm, int ld, int row, cudaStream_t stream) {
  return dots_into(A, lda, ncol, x, n, partial, SumOut{nullptr, mxm, ld, row}, stream);
}

cudaError_t launch_lowest_entry(const double* diag, const double* x, int64_t n, double* partial, double* out,
                                cudaStream_t stream) {
  lowest_entry_kernel<<<dot_grid(n), kDotThreads, 0, stream>>>(diag, x, n, partial, dot_counter(partial), out);
  return cudaGetLastError();
}

cudaError_t launch_subtract(double* t, const double* A, int64_t lda, const double* coef, int ncol, int64_t n,
                            bool norm, double* partial, double* out, cudaStream_t stream) {
  if (ncol < 1 || ncol > 32) return cudaErrorInvalidValue;
  const int g = dot_grid(n);
  unsigned int* ctr = dot_counter(partial);
  const SumOut o{out, nullptr, 0, 0};
#define C2G_SUB(C)                                                                                             \
  if (norm)                                                                                                    \
    subtract_kernel<C, true><<<g, kDotThreads, 0, stream>>>(t, A, lda, coef, ncol, n, partial, ctr, o);        \
  else                                                                                                         \
    subtract_kernel<C, false><<<g, kDotThreads, 0, stream>>>(t, A, lda, coef, ncol, n, partial, ctr, o);
  if (ncol <= 4) {
    C2G_SUB(4)
  } else if (ncol <= 8) {
    C2G_SUB(8)
  } else if (ncol <= 16) {
    C2G_SUB(16)
  } else {
    C2G_SUB(32)
  }
#undef C2G_SUB
  return cudaGetLastError();
}

cudaError_t launch_ritz(double* t, double* u, const double* HV, const double* V, int64_t lda, const double* coef,
                        int ncol, const double* evals, int64_t n, double* partial, double* out, cudaStream_t stream) {
  if (ncol < 1 || ncol > 64) return cudaErrorInvalidValue;
  ritz_kernel<<<dot_grid(n), kDotThreads, 0, stream>>>(t, u, HV, V, lda, coef, ncol, evals, n, partial,
                                                       dot_counter(partial), SumOut{out, nullptr, 0, 0});
  return cudaGetLastError();
}

cudaError_t launch_precond_dots(const double* t, const double* u, const double* diag, const double* evals,
                                double cutoff, int64_t n, double* partial, double* dots2, cudaStream_t stream) {
  precond_dots_kernel<<<dot_grid(n), kDotThreads, 0, stream>>>(t, u, diag, evals, cutoff, n, partial,
                                                               dot_counter(partial), SumOut{dots2, nullptr, 0, 0});
  return cudaGetLastError();
}

cudaError_t launch_precond(double* t, const double* u, const double* diag, const double* evals, const double* dots2,
                           double cutoff, const double* A, int64_t lda, int ncol, int64_t n, double* partial,
                           double* out, cudaStream_t stream) {
  if (ncol < 0 || ncol > 32) return cudaErrorInvalidValue;
  const int g = dot_grid(n);
  unsigned int* ctr = dot_counter(partial);
  const SumOut o{out, nullptr, 0, 0};
#define C2G_PRE(C) \
  precond_kernel<C><<<g, kDotThreads, 0, stream>>>(t, u, diag, evals, dots2, cutoff, A, lda, ncol, n, partial, ctr, o)
  if (ncol <= 4) C2G_PRE(4);
  else if (ncol <= 8) C2G_PRE(8);
  else if (ncol <= 16) C2G_PRE(16);
  else C2G_PRE(32);
#undef C2G_PRE
  return cudaGetLastError();
}

cudaError_t launch_normalize(double* dst, const double* x, const double* sumsq, int64_t n, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  normalize_kernel<<<grid_for(n), 256, 0, stream>>>(dst, x, sumsq, n);
  return cudaGetLastError();
}

cudaError_t launch_combine(double* out, double beta, const double* A, int64_t lda, const double* coef, int ncol,
                           int64_t n, cudaStream_t stream) {
  if (ncol > 64) return cudaErrorInvalidValue;
  if (n <= 0) return cudaSuccess;
  combine_kernel<<<grid_for(n), 256, 0, stream>>>(out, beta, A, lda, coef, ncol, n);
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

}  // namespace c2g
