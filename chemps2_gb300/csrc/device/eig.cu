// Symmetric eigensolvers (FP64 results): the Rayleigh-Ritz problem of the Davidson solver
// (order <= 32, one CTA) and the Gram matrices of the truncation (order <= 128, one CTA each, or
// above order 32 a cluster of eight where they are few), all by cyclic Jacobi with the
// round-robin (Brent-Luk) ordering: n / 2 disjoint plane rotations a round, n - 1 rounds a
// sweep.
//
// What bounds them: a warp's FP64 instruction takes 65 clocks here, dependent or not, and an
// SM does 1.6 FP64 multiply-adds a clock (both measured); an FP32 one takes 6, and an SM
// does 128. Hence:
//   - the matrix is its packed lower triangle, updated in place by 2 x 2 blocks (planes
//     P < Q), a lane for each block, and two barriers a round;
//   - a rotation is three shears by tan(angle / 2) and sin(angle): three multiply-adds for a
//     pair of elements instead of four operations;
//   - the half tangent is taken in FP32 (its error leaves 1e-7 of the element it should
//     annihilate, which the next sweep meets) and its sine in FP64, from an FP32 reciprocal
//     and one third-order step: orthogonal to FP64 accuracy, no FP64 division or square root;
//   - a plane's own diagonal block is updated by differences whose rounding scales with the
//     angle, so that the off-diagonal part goes on falling to 1e-15 of the norm;
//   - the Rayleigh-Ritz sweeps run in FP32, on off-diagonal elements of 24 bits and diagonal
//     elements of 48 (two floats, so that the gap between two close eigenvalues survives).
//     Their eigenvectors, applied to those found so far, are orthonormalised in FP64 by
//     (V^T V)^(-1/2) = I + E/2 + 3/8 E^2 + 5/16 E^3 + O(E^4), E = I - V^T V (1e-6 to 1e-4, so
//     the remainder is below FP64 rounding), and A = V^T G V is formed anew. A pass brings
//     the off-diagonal part down by 1e5 to 1e6: two passes, then one FP64 sweep (or as
//     many as it takes) to 1e-14 of the norm. The Gram matrices take FP64 sweeps only (see
//     gram_eigen): the FP32 passes gave 0.35 / 0.66 ms at order 32 and 13 / 27 at 128 in the
//     table below, but round small eigenvalues to 1e-16 of the norm.
// Measured, 20 Gram matrices of Gaussian / graded (1 to 1e-18) spectrum, against FP64 sweeps
// of four operations on the full matrix: order 16 0.48 / 0.85 -> 0.17 / 0.29 ms, 32 2.34 / 3.99
// -> 0.53 / 0.92, 64 6.2 / 11.7 -> 2.9 / 5.6, 128 41 / 82 -> 21 / 47 (one CTA for each; up to 38
// matrices above order 32 take a cluster each, 1.1 to 4 times as fast), with errors of the
// eigenvalues and the orthogonality of 0.3 to 2.6e-15 (2 to 70e-15 before). Rayleigh-Ritz
// of order 16: 332 -> 121 us cold, 177 -> 92 us warm; 32: 982 -> 357 and 584 -> 269.
#include "kernels.cuh"

#include <cmath>

namespace c2g {

namespace {

constexpr int kRrMax = 32;
static_assert(kBatchedEigMax == kRrMax, "the small kernels share their size");

// element (i, j) of a packed symmetric matrix
__device__ __forceinline__ int tri(int i, int j) {
  return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}
__host__ __device__ constexpr int tri_size(int m) { return m * (m + 1) / 2; }
__host__ __device__ constexpr int even_up(int n) { return n + (n & 1); }

template <typename R>
struct Planes {  // the rotations of a round: tan(angle / 2) and sin(angle)
  R h[kBatchedEigLargeMax / 2], s[kBatchedEigLargeMax / 2];
  int p[kBatchedEigLargeMax / 2], q[kBatchedEigLargeMax / 2];
  R red[2][32];
  float tan[kBatchedEigLargeMax / 2];  // FP32: tan(angle)
  R low[kBatchedEigLargeMax];          // FP32: what the diagonal of A leaves of its 48 bits
  int turned;                          // FP32: a rotation of the sweep was above the fine threshold
};

// Conversions by the bits of the formats, where a conversion instruction takes as long as
// an FP64 operation: magnitudes below 2^-126 go to zero, d2f truncates, |x| < 2^127.
__device__ __forceinline__ float d2f(double x) {
  const unsigned hi = __double2hiint(x), lo = __double2loint(x), mag = hi & 0x7fffffffu;
  const unsigned f = ((mag - (896u << 20)) << 3) | (lo >> 29);
  return __uint_as_float(mag < (897u << 20) ? 0u : (hi & 0x80000000u) | f);
}
__device__ __forceinline__ double f2d(float x) {
  const unsigned b = __float_as_uint(x), mag = b & 0x7fffffffu;
  const unsigned hi = mag < 0x00800000u ? 0u : (b & 0x80000000u) | ((mag >> 3) + (896u << 20));
  return __hiloint2double(hi, mag < 0x00800000u ? 0u : mag << 29);
}

// The rotation that annihilates apq, d = aqq - app, as h = tan(angle / 2) in FP32 (t:
// tan(angle)). Entries of magnitude at most about 1.
__device__ __forceinline__ float half_tangent(float d, float apq, float& t) {
  const float tau = __fdividef(d, 2.0f * apq), u = fmaf(tau, tau, 1.0f);
  t = copysignf(__fdividef(1.0f, fabsf(tau) + u * rsqrtf(u)), tau);
  const float w = fmaf(t, t, 1.0f);
  const float h = __fdividef(t, 1.0f + w * rsqrtf(w));
  if (apq == 0.0f || !(fabsf(tau) < 1e18f)) {  // nothing to annihilate, or an angle below 1e-18
    t = 0.0f;
    return 0.0f;
  }
  return h;
}
// sin(angle) = 2 h / (1 + h^2): in FP64 with one third-order step from an FP32 reciprocal, so
// that the rotation is orthogonal to FP64 accuracy for the h it is given
__device__ __forceinline__ float sine(float h) { return __fdividef(2.0f * h, fmaf(h, h, 1.0f)); }
__device__ __forceinline__ double sine(double h, float hf) {
  const double u = fma(h, h, 1.0);
  const double r = f2d(__fdividef(1.0f, fmaf(hf, hf, 1.0f)));
  const double e = fma(-u, r, 1.0);
  return 2.0 * h * fma(r, fma(e, e, e), r);
}

// (x, y) <- (c x - s y, s x + c y) by three shears
template <typename R>
__device__ __forceinline__ void rotate(R h, R s, R& x, R& y) {
  x = fma(-h, y, x);
  y = fma(s, x, y);
  x = fma(-h, y, x);
}

// hi + lo += x (Knuth's two-sum)
__device__ __forceinline__ void add_low(float& hi, float& lo, float x) {
  x += lo;
  const float s = hi + x, b = s - hi;
  lo = (hi - (s - b)) + (x - b);
  hi = s;
}

// Pair t of round r of m players: pos(0) = 0, pos(k) = 1 + (k - 1 - r mod m - 1), and the
// pairs are (pos(t), pos(m - 1 - t))
__device__ __forceinline__ void round_pair(int t, int r, int m, int& p, int& q) {
  int a = 0, b = m - 2 - t - r;
  if (t > 0) {
    a = t - 1 - r;
    a += 1 + (a < 0 ? m - 1 : 0);
  }
  b += 1 + (b < 0 ? m - 1 : 0);
  p = min(a, b);
  q = max(a, b);
}

// A plane's own diagonal block, as updates: their rounding scales with the angle, not with
// the diagonal
__device__ __forceinline__ void turn_plane(double h, double s, double& app, double& aqp, double& aqq) {
  const double b = aqp, d = app - aqq;
  const double cs = fma(-h, s, 1.0) * s, ss = s * s, x = fma(ss, d, 2.0 * cs * b);
  aqp = fma(cs, d, fma(-2.0 * ss, b, b));
  app -= x;
  aqq += x;
}

// Jacobi sweeps on the packed m x m matrix A (m even, entries of magnitude <= 1 or so; an
// odd order is padded by a zero row), the rotations applied to the columns of V (rows
// 0 .. n - 1, column j at V + ld j). FP64: until off(A)^2 <= tol |A|^2. FP32: until off(A)^2 is
// tol times what it was (or 1e-30 |A|^2), and with `fine` until a sweep turns no plane by
// more than 1e-3 over an element above 1e-16, so that a cluster of small eigenvalues is
// resolved as well. All threads of the CTA.
template <typename R>
__device__ void jacobi_sweeps(R* A, R* V, int ld, int n, int m, Planes<R>& sh, R tol, int max_sweeps,
                              bool fine = false) {
  constexpr bool k32 = sizeof(R) == 4;
  R goal = R(0);
  constexpr unsigned kAll = 0xffffffffu;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int npair = m / 2, nblk = npair * (npair - 1) / 2;
  // this thread's first 2 x 2 block (planes P and P + k) and the steps to its next; the
  // columns of V start at the warps after the last one with a block
  const int P0 = tid % npair, k0 = 1 + tid / npair, dP = nt % npair, dk = nt / npair;
  const int busy = ((nblk + 31) & ~31) % nt;
  const int v0 = tid >= busy ? tid - busy : tid + nt - busy;
  const int i0 = v0 % n, W0 = v0 / n, dI = nt % n, dW = nt / n;
  for (int sweep = 0; sweep < max_sweeps; sweep++) {
    R off = R(0), tot = R(0);
    for (int i = warp; i < m; i += nw)
      for (int j = lane; j <= i; j += 32) {
        const R v = A[i * (i + 1) / 2 + j];
        if (i == j) tot += v * v;
        else off += v * v;
      }
    off *= R(2);
    tot += off;
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_down_sync(kAll, off, o);
      tot += __shfl_down_sync(kAll, tot, o);
    }
    if (lane == 0) {
      sh.red[0][warp] = off;
      sh.red[1][warp] = tot;
    }
    __syncthreads();
    off = tot = R(0);
    for (int w = 0; w < nw; w++) {
      off += sh.red[0][w];
      tot += sh.red[1][w];
    }
    if (sweep == 0) goal = k32 ? fmaxf(tol * off, 1e-30f * tot) : tol * tot;
    const bool again = k32 && fine && sweep > 0 && sh.turned;
    __syncthreads();
    if (!(off > goal) && !again) break;
    if (tid == 0) sh.turned = 0;
    for (int r = 0; r < m - 1; r++) {
      if (tid < npair) {
        int p, q;
        round_pair(tid, r, m, p, q);
        const R app = A[tri(p, p)], aqq = A[tri(q, q)], apq = A[tri(q, p)];
        float tan;
        if constexpr (k32) {
          const float h = half_tangent((aqq - app) + (sh.low[q] - sh.low[p]), apq, tan);
          sh.h[tid] = h;
          sh.s[tid] = sine(h);
          sh.tan[tid] = tan;
          if (fine && fabsf(tan) > 1e-3f && fabsf(apq) > 1e-16f) sh.turned = 1;
        } else {
          const float hf = half_tangent(d2f(aqq - app), d2f(apq), tan);
          const double h = f2d(hf);
          sh.h[tid] = h;
          sh.s[tid] = sine(h, hf);
        }
        sh.p[tid] = p;
        sh.q[tid] = q;
      }
      __syncthreads();
      if (nt - 1 - tid < npair) {  // the planes' own diagonal blocks
        const int P = nt - 1 - tid;
        const R h = sh.h[P], s = sh.s[P];
        if (s != R(0)) {
          const int p = sh.p[P], q = sh.q[P];
          if constexpr (k32) {
            // app - t apq and aqq + t apq as two floats; the element between them is gone
            const float x = sh.tan[P] * A[tri(q, p)];
            A[tri(q, p)] = 0.0f;
            add_low(A[tri(p, p)], sh.low[p], -x);
            add_low(A[tri(q, q)], sh.low[q], x);
          } else {
            turn_plane(h, s, A[tri(p, p)], A[tri(q, p)], A[tri(q, q)]);
          }
        }
      }
      // the 2 x 2 blocks of planes P and Q = P + k (mod npair), each pair of planes once
      for (int e = tid, P = P0, k = k0; e < nblk; e += nt) {
        const int Q = P + k < npair ? P + k : P + k - npair;
        const R hp = sh.h[P], sp = sh.s[P], hq = sh.h[Q], sq = sh.s[Q];
        if (sp != R(0) || sq != R(0)) {
          const int p = sh.p[P], q = sh.q[P], u = sh.p[Q], v = sh.q[Q];
          const int pu = tri(p, u), pv = tri(p, v), qu = tri(q, u), qv = tri(q, v);
          R a = A[pu], b = A[pv], c = A[qu], d = A[qv];
          rotate(hp, sp, a, c);
          rotate(hp, sp, b, d);
          rotate(hq, sq, a, b);
          rotate(hq, sq, c, d);
          A[pu] = a;
          A[pv] = b;
          A[qu] = c;
          A[qv] = d;
        }
        P += dP;
        k += dk;
        if (P >= npair) {
          P -= npair;
          k++;
        }
      }
      for (int i = i0, P = W0; P < npair;) {
        const R h = sh.h[P], s = sh.s[P];
        if (s != R(0)) {
          R* vp = V + ld * sh.p[P] + i;
          R* vq = V + ld * sh.q[P] + i;
          R x = *vp, y = *vq;
          rotate(h, s, x, y);
          *vp = x;
          *vq = y;
        }
        i += dI;
        P += dW;
        if (i >= n) {
          i -= n;
          P++;
        }
      }
      __syncthreads();
    }
  }
}

// f(i, j, sum_{k < n} l(i, k) r(k, j)) for i < rows, j < n (lower: rows = n, only i >= j),
// 2 x 2 elements a thread. Ends with a barrier.
template <bool kLower, typename FL, typename FR, typename FO>
__device__ __forceinline__ void cta_product(int rows, int n, FL l, FR r, FO f) {
  const int rb = (rows + 1) / 2, cb = (n + 1) / 2;
  for (int e = threadIdx.x; e < rb * cb; e += blockDim.x) {
    // a full product's rows are half the matrix apart, so that a warp's columns (l(i, k) =
    // X[k + ld i], ld odd) fall in different banks
    const int i0 = kLower ? 2 * (e % rb) : e % rb, j0 = 2 * (e / rb);
    if (kLower && j0 > i0) continue;
    const int i1 = min(kLower ? i0 + 1 : i0 + rb, rows - 1), j1 = min(j0 + 1, n - 1);
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    for (int k = 0; k < n; k++) {
      const double x = l(i0, k), y = l(i1, k), u = r(k, j0), v = r(k, j1);
      a = fma(x, u, a);
      b = fma(x, v, b);
      c = fma(y, u, c);
      d = fma(y, v, d);
    }
    f(i0, j0, a);
    if (j1 > j0 && (!kLower || j1 <= i0)) f(i0, j1, b);
    if (i1 > i0) {
      f(i1, j0, c);
      if (j1 > j0) f(i1, j1, d);
    }
  }
  __syncthreads();
}

// The leading dimension of V: odd, so that a warp reading a row meets no bank twice.
__host__ __device__ constexpr int v_ld(int n) { return n | 1; }

// V = W (n x n), with a zero column where m > n
__device__ __forceinline__ void load_v(int n, int m, double* V, const double* W) {
  for (int e = threadIdx.x; e < n * m; e += blockDim.x) V[e % n + v_ld(n) * (e / n)] = e < n * n ? W[e] : 0.0;
}

// V (n columns of n, orthonormal to 1e-4 or better) orthonormalised, A = V^T G V for the
// matrix G (n x n). W: n x n scratch.
__device__ void orthonormal_transform(int n, int m, const double* G, double* A, double* V, double* W) {
  __shared__ double diag[kBatchedEigLargeMax];
  const int tid = threadIdx.x, nt = blockDim.x, ld = v_ld(n);
  auto lower = [&](const double* X, int i, int j) { return i >= j ? X[i + n * j] : X[j + n * i]; };
  // E, then E^2 in W's lower triangle, then (V^T V)^(-1/2) above it
  cta_product<true>(
      n, n, [&](int i, int k) { return V[k + ld * i]; }, [&](int k, int j) { return V[k + ld * j]; },
      [&](int i, int j, double v) { A[tri(i, j)] = (i == j ? 1.0 : 0.0) - v; });
  cta_product<true>(
      n, n, [&](int i, int k) { return A[tri(i, k)]; }, [&](int k, int j) { return A[tri(k, j)]; },
      [&](int i, int j, double v) { W[i + n * j] = v; });
  cta_product<true>(
      n, n, [&](int i, int k) { return A[tri(i, k)]; }, [&](int k, int j) { return lower(W, k, j); },
      [&](int i, int j, double v) {
        const double x = (i == j ? 1.0 : 0.0) + fma(0.5, A[tri(i, j)], fma(0.375, W[i + n * j], 0.3125 * v));
        if (i == j) diag[i] = x;
        else W[j + n * i] = x;
      });
  for (int e = tid; e < n * n; e += nt) {
    const int i = e % n, j = e / n;
    if (j <= i) A[i * (i + 1) / 2 + j] = i == j ? diag[i] : W[j + n * i];
  }
  __syncthreads();
  cta_product<false>(
      n, n, [&](int i, int k) { return V[i + ld * k]; }, [&](int k, int j) { return A[tri(k, j)]; },
      [&](int i, int j, double v) { W[i + n * j] = v; });
  load_v(n, m, V, W);
  __syncthreads();
  cta_product<false>(
      n, n, [&](int i, int k) { return G[i + n * k]; }, [&](int k, int j) { return V[k + ld * j]; },
      [&](int i, int j, double v) { W[i + n * j] = v; });
  cta_product<true>(
      n, n, [&](int i, int k) { return V[k + ld * i]; }, [&](int k, int j) { return W[k + n * j]; },
      [&](int i, int j, double v) { A[tri(i, j)] = v; });
  if (m > n)
    for (int e = tid; e < m; e += nt) A[tri(n, e)] = 0.0;
  __syncthreads();
}

// An FP32 pass ends at off(A) 3e-6 times what it was, well above FP32's rounding of a
// rotated matrix.
constexpr float kTol32 = 1e-11f;
constexpr int kSweeps32 = 12;
constexpr int kPasses32 = 2;

// The eigenproblem of G (n x n). In: A = V0^T G V0 packed, W = V0 (n x n, orthonormal) or, with
// `unit`, V0 = 1 and W not set. Out: the eigenvectors V (n x m, leading
// dimension v_ld(n)) and A = V^T G V diagonal.
// During an FP32 pass V's memory holds the FP32 eigenvectors and matrix, and W the FP64
// eigenvectors, which are then multiplied by half their rows at a time through A's memory.
__device__ void eigen(int n, int m, bool unit, const double* G, double* A, double* V, double* W,
                      Planes<float>& shf, Planes<double>& sh) {
  const int tid = threadIdx.x, nt = blockDim.x;
  float* Vf = reinterpret_cast<float*>(V);
  float* Af = Vf + n * m;
  for (int pass = 0; pass < kPasses32; pass++) {
    for (int e = tid; e < tri_size(m); e += nt) Af[e] = static_cast<float>(A[e]);
    for (int e = tid; e < n * m; e += nt) Vf[e] = e % n == e / n ? 1.0f : 0.0f;
    for (int j = tid; j < m; j += nt) {
      const double d = A[tri(j, j)];
      shf.low[j] = static_cast<float>(d - static_cast<double>(static_cast<float>(d)));
    }
    __syncthreads();
    jacobi_sweeps<float>(Af, Vf, n, n, m, shf, kTol32, kSweeps32, pass > 0);
    if (unit && pass == 0) {
      for (int e = tid; e < n * n; e += nt) W[e] = Vf[e];
      __syncthreads();
    } else {
      for (int r0 = 0; r0 < n; r0 += m / 2) {
        const int rows = min(m / 2, n - r0);
        for (int e = tid; e < rows * n; e += nt) A[e] = W[r0 + e % rows + n * (e / rows)];
        __syncthreads();
        cta_product<false>(
            rows, n, [&](int i, int k) { return A[i + rows * k]; },
            [&](int k, int j) { return f2d(Vf[k + n * j]); },
            [&](int i, int j, double v) { W[r0 + i + n * j] = v; });
      }
    }
    load_v(n, m, V, W);
    __syncthreads();
    orthonormal_transform(n, m, G, A, V, W);
    if (pass + 1 < kPasses32) {
      for (int e = tid; e < n * n; e += nt) W[e] = V[e % n + v_ld(n) * (e / n)];
      __syncthreads();
    }
  }
  jacobi_sweeps<double>(A, V, v_ld(n), n, m, sh, 1e-28, 30);
}

// The power of two that brings the largest magnitude to [0.5, 1) (1 for a zero, infinite or
// NaN matrix). v: this thread's largest magnitude; all threads of the CTA.
__device__ double unit_scale(double v, double* red) {
  const int tid = threadIdx.x, nw = blockDim.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  v = 0.0;
  for (int w = 0; w < nw; w++) v = fmax(v, red[w]);
  __syncthreads();
  if (!(v > 0.0) || isinf(v)) return 1.0;
  return ldexp(1.0, -max(-1000, min(1000, ilogb(v) + 1)));
}

// The rank of diagonal entry j of A among the n in ascending order (ties by index; the
// index itself where an entry is NaN, so that the ranks are a permutation).
__device__ __forceinline__ int ascending_rank(const double* A, int n, int j) {
  const double lam = A[tri(j, j)];
  int rk = 0;
  bool nan = false;
  for (int k = 0; k < n; k++) {
    const double o = A[tri(k, k)];
    rk += (o < lam || (o == lam && k < j)) ? 1 : 0;
    nan |= isnan(o);
  }
  return nan ? j : rk;
}

// Eigenvalues ascending at base + offE, eigenvectors in descending order at base + offU,
// each with the sign that makes its largest-magnitude entry (the first one on ties)
// positive -- the layout launch_reverse_columns produces.
// Equal eigenvalues (the zeros of a sector with empty blocks) keep the order that a selection
// sort with exchanges leaves them in, since a cut may fall among them.
// diag(j): the eigenvalue times `scale`; vec(i, j): element i of its vector. The CTA writes
// every `parts`-th column from `part` on.
template <class Diag, class Vec>
__device__ void write_descending(const EigJob& jb, double* base, Diag diag, Vec vec, double scale, int* order,
                                 int part = 0, int parts = 1) {
  const int n = jb.n, tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
  if (tid < 32) {
    for (int i = lane; i < n; i += 32) order[i] = i;
    __syncwarp();
    for (int i = 0; i < n; i++) {
      double best = 0.0;
      int at = n;
      for (int j = i + lane; j < n; j += 32) {
        const double v = diag(order[j]);
        if (at == n || v < best) {
          best = v;
          at = j;
        }
      }
      for (int d = 16; d > 0; d >>= 1) {
        const double b2 = __shfl_xor_sync(0xffffffffu, best, d);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, d);
        if (a2 < n && (at == n || b2 < best || (b2 == best && a2 < at))) {
          best = b2;
          at = a2;
        }
      }
      at = __shfl_sync(0xffffffffu, at, 0);  // (lanes may differ on a NaN)
      __syncwarp();
      if (lane == 0) {
        const int t = order[i];
        order[i] = order[at];
        order[at] = t;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (part == 0)
    for (int j = tid; j < n; j += blockDim.x) base[jb.offE + j] = diag(order[j]) / scale;
  for (int o = parts * (tid >> 5) + part; o < n; o += parts * nw) {
    const int col = order[n - 1 - o];
    double best = -1.0, v = 0.0;
    int at = n;
    for (int i = lane; i < n; i += 32)
      if (const double x = vec(i, col); fabs(x) > best) {
        v = x;
        best = fabs(v);
        at = i;
      }
    for (int d = 16; d > 0; d >>= 1) {
      const double b2 = __shfl_xor_sync(0xffffffffu, best, d), v2 = __shfl_xor_sync(0xffffffffu, v, d);
      const int a2 = __shfl_xor_sync(0xffffffffu, at, d);
      if (b2 > best || (b2 == best && a2 < at)) {
        best = b2;
        v = v2;
        at = a2;
      }
    }
    const double sgn = v < 0.0 ? -1.0 : 1.0;
    for (int i = lane; i < n; i += 32) base[jb.offU + i + static_cast<int64_t>(n) * o] = sgn * vec(i, col);
  }
}

// The Rayleigh-Ritz eigenproblem (CheMPS2/Davidson.cpp:242-276, where the reference calls
// dsyev on the <= 32 x 32 projected matrix). Warm start (Davidson expansion): the matrix
// grew by one row and column since the previous call, whose eigenvectors E are still in
// evecs; the solver starts from diag(E, 1)^T M diag(E, 1), diagonal but for the last row and
// column, which takes two to three sweeps instead of six to ten.
constexpr int kRrThreads = 256;
__global__ void __launch_bounds__(kRrThreads, 1) rr_eig_kernel(const double* __restrict__ mat, int n, int ld,
                                                            double* __restrict__ evals, double* __restrict__ evecs,
                                                            int warm) {
  __shared__ double A[tri_size(kRrMax)], V[kRrMax * v_ld(kRrMax)], W[kRrMax * kRrMax], G[kRrMax * kRrMax];
  __shared__ Planes<double> sh;
  __shared__ Planes<float> shf;
  const int tid = threadIdx.x, m = even_up(n);
  double big = 0.0;
  for (int e = tid; e < n * n; e += kRrThreads) big = fmax(big, fabs(mat[e % n + ld * (e / n)]));
  const double sc = unit_scale(big, sh.red[0]), hs = 0.5 * sc;
  for (int e = tid; e < n * n; e += kRrThreads) {
    const int i = e % n, j = e / n;
    G[e] = hs * mat[i + ld * j] + hs * mat[j + ld * i];
    W[e] = (warm && i < n - 1 && j < n - 1) ? evecs[i + ld * j] : (i == j ? 1.0 : 0.0);
  }
  for (int e = tid; e < tri_size(m); e += kRrThreads) A[e] = 0.0;
  __syncthreads();
  if (warm) {
    cta_product<false>(
        n, n, [&](int i, int k) { return G[i + n * k]; }, [&](int k, int j) { return W[k + n * j]; }, [&](int i, int j, double v) { V[i + n * j] = v; });
    cta_product<true>(
        n, n, [&](int i, int k) { return W[k + n * i]; }, [&](int k, int j) { return V[k + n * j]; },
        [&](int i, int j, double v) { A[tri(i, j)] = v; });
  } else {
    for (int e = tid; e < n * n; e += kRrThreads)
      if (e % n >= e / n) A[tri(e % n, e / n)] = G[e];
    __syncthreads();
  }
  if (n > 1) {
    eigen(n, m, !warm, G, A, V, W, shf, sh);
  } else {
    if (tid == 0) V[0] = 1.0;
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += kRrThreads) {
    const int i = e % n, j = e / n;
    const int rk = ascending_rank(A, n, j);
    if (i == 0) evals[rk] = A[tri(j, j)] / sc;
    evecs[i + ld * rk] = V[i + v_ld(n) * j];
  }
}

// The Gram matrices of the truncation, one CTA each, by FP64 sweeps throughout: their rotations
// leave a graded matrix's small elements their own relative accuracy, while V^T G V would
// round them to 1e-16 of the norm. The sweeps end at an off-diagonal part of 1e-15 of the norm:
// vectors of eigenvalues below that (singular values below 3e-8 of the largest) may still be
// mixed with one another.
__device__ __forceinline__ void gram_eigen(const EigJob& jb, double* base, double* A, double* V, Planes<double>& sh,
                                           int* order) {
  const int n = jb.n, m = even_up(n), ld = v_ld(n), tid = threadIdx.x, nt = blockDim.x;
  const double* G = base + jb.offG;
  double big = 0.0;
  for (int e = tid; e < n * n; e += nt) big = fmax(big, fabs(G[e]));
  const double sc = unit_scale(big, sh.red[0]), hs = 0.5 * sc;
  for (int e = tid; e < m * m; e += nt) {
    const int i = e % m, j = e / m;
    if (j <= i) A[tri(i, j)] = i < n ? hs * G[i + n * j] + hs * G[j + n * i] : 0.0;
    if (i < n) V[i + ld * j] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  if (n > 1) jacobi_sweeps<double>(A, V, ld, n, m, sh, 1e-30, 30);
  write_descending(
      jb, base, [=](int j) { return A[tri(j, j)]; }, [=](int i, int j) { return V[i + ld * j]; }, sc, order);
}

// order <= kBatchedEigMax
constexpr int kEigSmallThreads = 512;
__global__ void __launch_bounds__(kEigSmallThreads, 1) batched_eig_kernel(const EigJob* __restrict__ jobs,
                                                                          double* __restrict__ base) {
  constexpr int kN = kBatchedEigMax;
  __shared__ double A[tri_size(kN)], V[kN * v_ld(kN)];
  __shared__ Planes<double> sh;
  __shared__ int order[kN];
  gram_eigen(jobs[blockIdx.x], base, A, V, sh, order);
}

// order kBatchedEigMax + 1 .. kBatchedEigLargeMax, many matrices: A and V in dynamic shared
// memory
constexpr int kEigLargeThreads = 512;
__host__ __device__ constexpr size_t eig_large_bytes(int n) {
  return sizeof(double) * (static_cast<size_t>(tri_size(even_up(n))) + static_cast<size_t>(even_up(n)) * v_ld(n));
}
__global__ void __launch_bounds__(kEigLargeThreads) batched_eig_large_kernel(const EigJob* __restrict__ jobs,
                                                                             double* __restrict__ base) {
  extern __shared__ double dyn[];
  __shared__ Planes<double> sh;
  __shared__ int order[kBatchedEigLargeMax];
  const EigJob jb = jobs[blockIdx.x];
  gram_eigen(jb, base, dyn, dyn + tri_size(even_up(jb.n)), sh, order);
}

// The same orders, few matrices: a cluster of kCl CTAs for each, the
// same sweeps. In one CTA a round at order 128 is 49000 FP64 operations at 1.6 a clock
// (15 us) while nearly all SMs have nothing to do, as a state has few sectors of this size.
// Element e of the packed A is in CTA e mod kCl (in two copies: a round reads one and writes
// all of the other, so that it needs one cluster barrier), V's rows are dealt out in
// ranges, and every CTA finds all rotations of a round itself. V is turned between the
// arrival at the barrier and the wait. Now a round's chain bounds it (rotations from remote
// elements, blocks, barrier: 1 to 5 us).
constexpr int kCl = 8, kClThreads = 256;
// The line is by the number of matrices alone, where two CTAs of the clusters come to an SM: up
// to it the cluster loses at most 5 % (order 33), at 60 matrices one CTA each at most 5 % (order
// 128). ms for one CTA -> cluster, Gaussian spectrum: 6 matrices order 33 0.61 -> 0.52, 48 1.22
// -> 0.77, 64 2.85 -> 1.21, 96 9.0 -> 2.7, 128 20.3 -> 5.1; 38 matrices 0.55 -> 0.58, 1.23 -> 1.10,
// 2.86 -> 1.79, 9.0 -> 5.3, 20.9 -> 11.7; 60 matrices 0.55 -> 1.16, 1.24 -> 1.97, 2.85 -> 3.24, 8.6 ->
// 9.4, 20.6 -> 19.5. (512 threads: 4.8 ms for one of order 128 instead of 5.2, but half as many
// at a time; four CTAs: 7.9 ms.)
constexpr int kClMaxJobs = 38;
constexpr int kClA = (tri_size(kBatchedEigLargeMax) + kCl - 1) / kCl;
constexpr int kClRows = (kBatchedEigLargeMax + kCl - 1) / kCl, kClLd = kClRows + 1;

__device__ __forceinline__ uint32_t cl_addr(uint32_t a, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ double cl_load(uint32_t a, int rank) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(cl_addr(a, rank)) : "memory");
  return v;
}
__device__ __forceinline__ void cl_store(uint32_t a, int rank, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cl_addr(a, rank)), "d"(v) : "memory");
}
// (the barrier's instructions are for whole warps)
__device__ __forceinline__ void cl_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cl_sync() {
  cl_arrive();
  cl_wait();
}

__global__ void __cluster_dims__(kCl, 1, 1) __launch_bounds__(kClThreads, 1)
    batched_eig_cluster_kernel(const EigJob* __restrict__ jobs, double* __restrict__ base) {
  __shared__ double A[2][kClA], V[kBatchedEigLargeMax * kClLd];
  __shared__ double H[2][kBatchedEigLargeMax / 2], S[2][kBatchedEigLargeMax / 2];  // by parity of the round
  __shared__ int Pl[2][kBatchedEigLargeMax / 2], Ql[2][kBatchedEigLargeMax / 2];
  __shared__ double red[2][32], part[2], lam[kBatchedEigLargeMax];
  __shared__ int order[kBatchedEigLargeMax];
  const EigJob jb = jobs[blockIdx.x / kCl];
  const int rank = blockIdx.x % kCl;  // in the cluster too: clusters are runs of kCl CTAs
  const int n = jb.n, m = even_up(n), npair = m / 2, nel = tri_size(m), nblk = npair * (npair - 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + kCl - 1) / kCl, row0 = rank * per, nrow = max(0, min(per, n - row0));
  const uint32_t a0 = static_cast<uint32_t>(__cvta_generic_to_shared(&A[0][0]));
  auto at = [&](int b, int e) { return a0 + static_cast<uint32_t>(8 * (b * kClA + e / kCl)); };
  auto get = [&](int b, int e) { return cl_load(at(b, e), e % kCl); };
  auto put = [&](int b, int e, double v) { cl_store(at(b, e), e % kCl, v); };

  const double* G = base + jb.offG;
  double big = 0.0;
  for (int e = tid; e < n * n; e += kClThreads) big = fmax(big, fabs(G[e]));
  const double sc = unit_scale(big, red[0]), hs = 0.5 * sc;
  for (int e = tid; e < m * m; e += kClThreads) {
    const int i = e % m, j = e / m, x = tri(i, j);
    if (j <= i && x % kCl == rank) A[0][x / kCl] = i < n ? hs * G[i + n * j] + hs * G[j + n * i] : 0.0;
  }
  for (int e = tid; e < m * kClLd; e += kClThreads) V[e] = row0 + e % kClLd == e / kClLd ? 1.0 : 0.0;
  cl_sync();

  // this thread's 2 x 2 block (planes bP < bQ of a cycle, each pair once) and the first of
  // its elements of V with the steps to the next
  static_assert(kBatchedEigLargeMax / 2 * (kBatchedEigLargeMax / 2 - 1) / 2 <= kCl * kClThreads, "a block a thread");
  const int blk = rank + kCl * tid, bP = blk % npair, bQ0 = bP + 1 + blk / npair;
  const int bQ = bQ0 < npair ? bQ0 : bQ0 - npair;
  const bool block = blk < nblk;
  const int rows = max(nrow, 1), i0 = tid % rows, W0 = nrow > 0 ? tid / rows : npair;
  const int dI = kClThreads % rows, dW = kClThreads / rows;

  int cur = 0, par = 0;
  double goal = 0.0;
  for (int sweep = 0; sweep < 30 && n > 1; sweep++) {
    // off(A)^2 and |A|^2: every CTA adds the same eight parts in the same order, so that all
    // of the cluster take the same way
    double off = 0.0, tot = 0.0;
    for (int s = tid; s * kCl + rank < nel; s += kClThreads) {
      const int e = s * kCl + rank;
      int i = static_cast<int>((sqrtf(8.0f * static_cast<float>(e) + 1.0f) - 1.0f) * 0.5f);
      while (tri_size(i + 1) <= e) i++;
      while (tri_size(i) > e) i--;
      const double v = A[cur][s];
      if (e - tri_size(i) == i) tot += v * v;
      else off += v * v;
    }
    off *= 2.0;
    tot += off;
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_down_sync(0xffffffffu, off, o);
      tot += __shfl_down_sync(0xffffffffu, tot, o);
    }
    if (lane == 0) {
      red[0][warp] = off;
      red[1][warp] = tot;
    }
    __syncthreads();
    if (tid < 2) {
      double v = 0.0;
      for (int w = 0; w < kClThreads / 32; w++) v += red[tid][w];
      part[tid] = v;
    }
    cl_sync();
    off = tot = 0.0;
    const uint32_t pa = static_cast<uint32_t>(__cvta_generic_to_shared(part));
    for (int c = 0; c < kCl; c++) {
      off += cl_load(pa, c);
      tot += cl_load(pa + 8, c);
    }
    if (sweep == 0) goal = 1e-30 * tot;
    if (!(off > goal)) break;
    for (int r = 0; r < m - 1; r++) {
      const int nxt = cur ^ 1;
      if (tid < npair) {
        int p, q;
        round_pair(tid, r, m, p, q);
        const double app = get(cur, tri(p, p)), aqq = get(cur, tri(q, q)), apq = get(cur, tri(q, p));
        float tan;
        const float hf = half_tangent(d2f(aqq - app), d2f(apq), tan);
        const double h = f2d(hf);
        H[par][tid] = h;
        S[par][tid] = sine(h, hf);
        Pl[par][tid] = p;
        Ql[par][tid] = q;
      }
      __syncthreads();
      if (const int P = rank + kCl * (kClThreads - 1 - tid); P < npair) {
        const int p = Pl[par][P], q = Ql[par][P], pp = tri(p, p), qp = tri(q, p), qq = tri(q, q);
        double a = get(cur, pp), b = get(cur, qp), d = get(cur, qq);
        turn_plane(H[par][P], S[par][P], a, b, d);
        put(nxt, pp, a);
        put(nxt, qp, b);
        put(nxt, qq, d);
      }
      if (block) {
        const int P = bP, Q = bQ;
        const double hp = H[par][P], sp = S[par][P], hq = H[par][Q], sq = S[par][Q];
        const int p = Pl[par][P], q = Ql[par][P], u = Pl[par][Q], v = Ql[par][Q];
        const int pu = tri(p, u), pv = tri(p, v), qu = tri(q, u), qv = tri(q, v);
        double a = get(cur, pu), b = get(cur, pv), c = get(cur, qu), d = get(cur, qv);
        rotate(hp, sp, a, c);
        rotate(hp, sp, b, d);
        rotate(hq, sq, a, b);
        rotate(hq, sq, c, d);
        put(nxt, pu, a);
        put(nxt, pv, b);
        put(nxt, qu, c);
        put(nxt, qv, d);
      }
      cl_arrive();
      for (int i = i0, P = W0; P < npair;) {
        const double h = H[par][P], s = S[par][P];
        if (s != 0.0) {
          double* vp = V + kClLd * Pl[par][P] + i;
          double* vq = V + kClLd * Ql[par][P] + i;
          double x = *vp, y = *vq;
          rotate(h, s, x, y);
          *vp = x;
          *vq = y;
        }
        i += dI;
        P += dW;
        if (i >= nrow) {
          i -= nrow;
          P++;
        }
      }
      cl_wait();
      // the next round's planes go to the other copy: V may still be turned by these
      cur = nxt;
      par ^= 1;
    }
  }
  for (int j = tid; j < n; j += kClThreads) lam[j] = get(cur, tri(j, j));
  cl_sync();  // all rows of V are final
  const uint32_t v0 = static_cast<uint32_t>(__cvta_generic_to_shared(V));
  write_descending(
      jb, base, [&](int j) { return lam[j]; },
      [&](int i, int j) { return cl_load(v0 + static_cast<uint32_t>(8 * (kClLd * j + i % per)), i / per); }, sc, order,
      rank, kCl);
  cl_sync();  // no CTA ends while another reads its rows
}

// Loewdin orthonormaliser of k <= 4 vectors: L = S^-1/2 from the k x k overlap S
// (CheMPS2/Davidson.cpp:367-381). Serial Jacobi, one thread.
__global__ void lowdin_kernel(const double* __restrict__ overlap, int k, double* __restrict__ lowdin) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double a[4][4], v[4][4];
  for (int i = 0; i < k; i++)
    for (int j = 0; j < k; j++) {
      a[i][j] = overlap[i + k * j];
      v[i][j] = (i == j) ? 1.0 : 0.0;
    }
  for (int sweep = 0; sweep < 50; sweep++) {
    double off = 0.0;
    for (int i = 0; i < k; i++)
      for (int j = 0; j < k; j++)
        if (i != j) off += a[i][j] * a[i][j];
    double tot = off;
    for (int i = 0; i < k; i++) tot += a[i][i] * a[i][i];
    if (!(off > 1e-32 * tot)) break;  // below rounding
    for (int p = 0; p < k; p++)
      for (int q = p + 1; q < k; q++) {
        if (a[p][q] == 0.0) continue;
        const double tau = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
        const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
        const double c = 1.0 / sqrt(1.0 + t * t), s = t * c;
        for (int j = 0; j < k; j++) {
          const double x = a[p][j], y = a[q][j];
          a[p][j] = c * x - s * y;
          a[q][j] = s * x + c * y;
        }
        for (int i = 0; i < k; i++) {
          const double x = a[i][p], y = a[i][q];
          a[i][p] = c * x - s * y;
          a[i][q] = s * x + c * y;
          const double vx = v[i][p], vy = v[i][q];
          v[i][p] = c * vx - s * vy;
          v[i][q] = s * vx + c * vy;
        }
      }
  }
  double f[4];
  for (int j = 0; j < k; j++) f[j] = pow(a[j][j], -0.5);
  for (int i = 0; i < k; i++)
    for (int j = 0; j < k; j++) {
      double s = 0.0;
      for (int l = 0; l < k; l++) s += v[i][l] * f[l] * v[j][l];
      lowdin[i + k * j] = s;
    }
}

}  // namespace

cudaError_t launch_small_eig(double* mat, int n, int ld, double* evals, double* evecs, cudaStream_t stream,
                             bool warm) {
  if (n < 1 || n > kRrMax || ld < n) return cudaErrorInvalidValue;
  rr_eig_kernel<<<1, kRrThreads, 0, stream>>>(mat, n, ld, evals, evecs, warm && n > 1 ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_batched_eig(const EigJob* jobs, int njobs, double* base, cudaStream_t stream) {
  if (njobs <= 0) return cudaSuccess;
  batched_eig_kernel<<<njobs, kEigSmallThreads, 0, stream>>>(jobs, base);
  return cudaGetLastError();
}

cudaError_t launch_batched_eig_large(const EigJob* jobs, int njobs, int nmax, double* base, cudaStream_t stream) {
  if (njobs <= 0) return cudaSuccess;
  if (nmax > kBatchedEigLargeMax) return cudaErrorInvalidValue;
  if (njobs <= kClMaxJobs) {
    batched_eig_cluster_kernel<<<kCl * njobs, kClThreads, 0, stream>>>(jobs, base);
    return cudaGetLastError();
  }
  const cudaError_t e = cudaFuncSetAttribute(batched_eig_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(eig_large_bytes(kBatchedEigLargeMax)));
  if (e != cudaSuccess) return e;
  batched_eig_large_kernel<<<njobs, kEigLargeThreads, eig_large_bytes(nmax), stream>>>(jobs, base);
  return cudaGetLastError();
}

cudaError_t launch_lowdin(const double* overlap, int k, double* lowdin, cudaStream_t stream) {
  if (k < 1 || k > 4) return cudaErrorInvalidValue;
  lowdin_kernel<<<1, 32, 0, stream>>>(overlap, k, lowdin);
  return cudaGetLastError();
}

}  // namespace c2g
