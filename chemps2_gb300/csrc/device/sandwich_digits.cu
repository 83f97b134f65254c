// Two-pass path of large groups in FP64 on the 5th-generation tensor cores: the passes of
// sandwich_gemm.cu with every product of two FP64 blocks formed from exact integer products
// of their digits (the splitting of K. Ozaki, T. Ogita, S. Oishi and S. Rump, "Error-free
// transformations of matrix multiplication", 2012).
//
// Why: an SM of this GPU does 1.6 FP64 multiply-adds a clock and the tensor cores 4096
// 16-bit ones, and sandwich_gemm.cu runs at the FP64 pipe's rate.
//
// A step is one product L (m x K) R (K x n) of at most 64 x 32 outputs and K <= 32. Each row
// of L and column of R is scaled by the power of two above its largest magnitude, 2^e, and
// every element becomes the integer X = v 2^(62 - e) to the nearest, |X| <= 2^62: eight digits
// to the base 256 in [-128, 127], exact in FP16. The tensor core sums d_i d_j over K and over
// the pairs of one diagonal c = i + j <= 7 in FP32: at most 8 x 64 products of at most 2^14, so
// below 2^24 and exact. Dropped are the diagonals c >= 8. The eight sums are put together in
// 96 bits and rounded to a double by integer instructions; one FP64 instruction adds that to
// the item sum, where the FP64 pipe rounds at each of the K terms. Products longer than 32 take
// several steps; a second one adds to the first one's sums in tensor memory where its elements
// fit the same scales, and else to its rounded ones.
//
// What is dropped is small beside M, the product of the row's and the column's scales (at most
// K 2^-59 M, 2^-62 M as a rule), and so beside an output of which a product is near M, but not
// beside one where L is large along K where R is small, and the other way round. So each
// element has a weight, the binary orders d that it is below its row's or column's largest,
// and an output is taken from the digits only where some k has d <= 1, 3 or 5 in L and d <= 5, 3
// or 1 in R (a product of 2^-8 M or more), or no product at all. Any other one is formed by the K
// FP64 multiply-adds of the FP64 pipe. rms errors in units of 2^-53 sum |l| |r|, digits / FP64
// pipe: operands of one size 0.12 to 0.18 / 0.46 to 0.49, spread over 2^40 0.8 to 1.1 / 1.0 to 2.3, L
// falling and R rising along K by 2, 6 and 20 decades 0.12 to 0.30, 0.18 to 0.47 and 0.29 to 0.48 / 0.44
// to 0.49. Outputs formed by multiply-adds: none of random operands; in swept states 0.2 to 6 %
// of pass 1's and 0.01 to 0.5 % of pass 2's (ab initio to Hubbard L = 16).
//
// L's digits are rows of shared memory digit by digit and so are R's columns, so that digit i
// of L meets digits 0 .. 7 - i of R in one MMA whose accumulator starts at column group i: 8
// MMAs of M = 128 for each 16 of K. Persistent 256-thread CTAs, two per SM (256 columns of
// tensor memory and 106 KB of shared memory each, so that one cuts digits and rounds sums while the
// other's MMAs run) take the 64 x 32 halves of the tile lists' tiles from an atomic counter.
// While the MMAs of a step run, all threads round the previous step's sums (copied from
// tensor memory to shared memory by the warps of the quadrants that hold them) and the next
// step's operands are on their way from memory. An operand that the step before had too is
// not cut again.
//
// What bounds it: a step's fixed chain, load - exponents - digits - MMA - collect, of 2.2 to
// 4.6 us an SM whatever its size, with the tensor pipe busy 16 to 23 % of the time and the issue
// slots 38 %. us a product and SM, FP64 pipe -> digits, pass 1 / pass 2:
// 17 x 17 x 17 3.1 -> 2.7 / 4.2 -> 3.6, 32 x 32 x 32 8.3 -> 3.3 / 10.0 -> 4.6, 47 x 47 x 47 27 -> 11.0 /
// 31 -> 11.7, 64 x 64 x 64 65 -> 14.8 / 73 -> 15.5. With seven digits and no weights the last three were
// 3.0 / 4.4, 9.1 / 10.6 and 12.2 / 13.7, but outputs without a product near M lost up to all of their
// digits. Below about 17 x 17 x 12 the FP64 pipe is the faster one (digits_pay in runtime.cpp).
//
// Every mbarrier wait is bounded: after kPolls polls a CTA records an error in the runtime's
// mapped error word, writes NaN to that tile and to all that it takes after it (so that split
// tiles still meet at their counters), and frees its tensor memory once its MMAs are done, or
// after a second bounded wait. A step with an infinite or NaN element, or with a scale that may take a result out of
// the normal range, is formed by multiply-adds as a whole.
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>
#include <cstddef>

#include "kernels.cuh"
#include "slots.cuh"
#include "tcgen05.cuh"

namespace c2g {

namespace {

constexpr int kDgThreads = 256;
constexpr int kDgIssuer = 5;  // the warp that issues the MMAs: of the last to cut digits, and
                              // without tile rows of tensor memory in a tile of 32 rows
constexpr int kDgCtasPerSm = 2;
constexpr int kDgDigits = 8, kDgDiagonals = kDgDigits;
constexpr int kDgRows = 64, kDgCols = 32, kDgK = 32;  // of a step
constexpr uint32_t kDgTmemCols = kDgDiagonals * kDgCols;
constexpr int kDgBatch = 32;                          // records held in shared memory

// Exponent fields of the scales that digits take: those of a row and a column add up to at least
// 1092 and at most 3060, so that every sum, a multiple of 2^-68 of the scales' product and at most
// 2^6 times that, is a normal number.
constexpr unsigned int kDgExpoMin = 546, kDgExpoMax = 1530;

// K-major rows without swizzle, 16 of K at a time: 8-row groups of 256 bytes, 128 bytes
// between the two 8-wide halves of K
constexpr int kDgRowBytes = 32;
constexpr int kDgLBytes = kDgDigits * kDgRows * kDgRowBytes;  // one half (16) of a step's K
constexpr int kDgRBytes = kDgDigits * kDgCols * kDgRowBytes;
// leading dimension of a row of sums: 16-byte accesses of eight rows meet every bank once
constexpr int kDgSumLd = kDgCols + 4;

// One product: op(L) (rows x K) op(R) (K x cols), already at its tile.
struct DgRecord {  // 64 bytes
  const double* l;
  const double* r;
  double* s;  // pass 1: where it goes, column-major with leading dimension lds
  double alpha;
  int32_t lld, rld;  // element (i, k) of an operand: trans ? p[k + ld i] : p[i + ld k]
  int32_t k, lds;
  int16_t rows, cols;
  int8_t ltrans, rtrans;
  int8_t pad[10];
};
static_assert(sizeof(DgRecord) == 64, "DgRecord");

// A step whose sums are not rounded yet: its product's record, its range of K (up to two
// steps') and whether that begins and ends the product.
struct DgStep {
  DgRecord x;
  int32_t k0, k1;
  bool first, last;
};

struct __align__(1024) DgSmem {
  unsigned char l[2 * kDgLBytes];
  unsigned char r[2 * kDgRBytes];
  int sums[kDgDiagonals / 2 * kDgRows * kDgSumLd];  // [diagonal pair][row][column] of the previous step
  DgRecord rec[kDgBatch];
  unsigned long long bar;
  // largest exponent fields of the rows of L, then of the columns of R: of the step in
  // flight, the one being staged and (zero) the next
  alignas(16) unsigned int expo[3][kDgRows + kDgCols];
  // weight words (dg_weight) of the rows of L, then of the columns of R, by groups of 8 of K
  uint4 weight[kDgRows + kDgCols];
  DgStep step[2];  // of the step in flight and the next
  uint32_t tmem_base;
  int slot, is_last;
  // each thread's own outputs: in pass 2 a product's sums over its first steps, in pass 1 what
  // is formed by multiply-adds
  double part[8][kDgThreads];
};

static_assert(offsetof(DgSmem, expo) % 16 == 0 && (kDgRows + kDgCols) % 4 == 0, "16-byte reads of expo");

// Instruction descriptor of kind::f16: D F32 (bits 4-5 = 1), A and B F16 (bits 7-9 and 10-12
// = 0), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28; M = 128.
__host__ __device__ constexpr uint32_t dg_idesc(int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}

// Eight consecutive k of one row of an operand, in registers.
struct DgUnit {
  double v[8];
};

__device__ __forceinline__ void dg_load(DgUnit& u, const double* p, int ld, bool t, int row, int k0, int n) {
  p += t ? k0 + static_cast<int64_t>(ld) * row : row + static_cast<int64_t>(ld) * k0;
  const int64_t step = t ? 1 : ld;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    u.v[k] = k < n ? *p : 0.0;
    p += step;
  }
}

__device__ __forceinline__ unsigned int dg_exponent(const DgUnit& u) {
  unsigned int e = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) e = max(e, static_cast<unsigned int>(__double2hiint(u.v[k])) & 0x7ff00000u);
  return e >> 20;
}

// X + sum_i 128 256^i of an element: its eight digits plus 128, as bytes; emax: the row's
// largest exponent field
__device__ __forceinline__ unsigned long long dg_fixed(double v, unsigned int emax) {
  const unsigned int hi = __double2hiint(v), lo = __double2loint(v);
  const unsigned int e = (hi >> 20) & 0x7ffu;
  const unsigned long long m =
      (static_cast<unsigned long long>((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;  // below 2^63
  const unsigned int sh = e == 0u ? 63u : min(emax - e, 63u);
  const unsigned long long x = ((m >> sh) + 1ull) >> 1;  // to the nearest, below 2^62
  const unsigned long long s = static_cast<long long>(static_cast<int>(hi)) >> 63;
  return (x ^ s) - s + 0x8080808080808080ull;
}

// How far a unit's elements are below the row's largest, in binary orders d: bit k of byte
// 0 is set where the element is not zero, of byte 1 where d <= 5, of byte 2 where d <= 3 and
// of byte 3 where d <= 1.
__device__ __forceinline__ uint32_t dg_weight(const DgUnit& u, unsigned int emax) {
  uint32_t w = 0u;
  emax = max(emax, 6u);  // in a row of subnormal elements all are far below it
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const unsigned int hi = __double2hiint(u.v[k]), lo = __double2loint(u.v[k]);
    const unsigned int d = min(emax - ((hi >> 20) & 0x7ffu), 6u);
    const uint32_t t = (0x01010101u << k) >> ((4u * d) & 24u);
    if (((hi & 0x7fffffffu) | lo) != 0u) w |= t;
  }
  return w;
}

// digit i of two such integers as FP16, low first: 1024 + byte in FP16, less 1152
template <int i>
__device__ __forceinline__ uint32_t dg_pair(unsigned long long a, unsigned long long b) {
  constexpr int byte = (7 - i) & 3;
  const uint32_t x = static_cast<uint32_t>(i < 4 ? a >> 32 : a), y = static_cast<uint32_t>(i < 4 ? b >> 32 : b);
  const uint32_t t = (__byte_perm(x, y, byte | (4 + byte) << 8) & 0x00ff00ffu) | 0x64006400u;
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&t), __floats2half2_rn(1152.0f, 1152.0f));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Stores the digits of a unit (row `row`, k group kg of 8) of an operand; kRows: the rows of
// a digit, half_bytes: the size of one half of K.
template <int kRows>
__device__ __forceinline__ void dg_store(const DgUnit& u, unsigned int emax, unsigned char* buf, int half_bytes,
                                         int row, int kg) {
  unsigned long long x[8];
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = dg_fixed(u.v[k], emax);
  unsigned char* at = buf + (kg >> 1) * half_bytes + (kg & 1) * 128 + (row >> 3) * 256 + (row & 7) * 16;
#define C2G_DIGIT(i)                                                                                       \
  *reinterpret_cast<uint4*>(at + i * kRows * kDgRowBytes) =                                                \
      make_uint4(dg_pair<i>(x[0], x[1]), dg_pair<i>(x[2], x[3]), dg_pair<i>(x[4], x[5]), dg_pair<i>(x[6], x[7]));
  C2G_DIGIT(0)
  C2G_DIGIT(1)
  C2G_DIGIT(2)
  C2G_DIGIT(3)
  C2G_DIGIT(4)
  C2G_DIGIT(5)
  C2G_DIGIT(6)
  C2G_DIGIT(7)
#undef C2G_DIGIT
}

// (hi 2^32 + lo) 2^k as a double to the nearest, by the bits (a conversion or an FP64
// instruction costs a warp 65 clocks); |hi| < 2^62, |lo| < 2^62, the result in the normal
// range. A negative one is off by a unit of lo before it is rounded.
__device__ __forceinline__ double rounded(long long hi, long long lo, int k) {
  hi += lo >> 32;
  const unsigned int s = static_cast<unsigned int>(hi >> 63);
  const unsigned int h2 = static_cast<unsigned int>(hi >> 32) ^ s, h1 = static_cast<unsigned int>(hi) ^ s,
                     h0 = static_cast<unsigned int>(lo) ^ s;
  // the 96 bits h, normalised
  const bool a = h2 == 0u, b = a && h1 == 0u;
  const unsigned int w2 = b ? h0 : a ? h1 : h2, w1 = b ? 0u : a ? h0 : h1, w0 = a ? 0u : h0;
  const int z = __clz(static_cast<int>(w2));
  const int f = 1086 + 32 + k - z - (b ? 64 : a ? 32 : 0);  // the exponent field
  const unsigned long long u =
      static_cast<unsigned long long>(__funnelshift_l(w1, w2, z)) << 32 | __funnelshift_l(w0, w1, z);
  const unsigned long long m = (u >> 11) + ((u >> 10) & 1u);  // 2^52 .. 2^53
  const unsigned long long v = (static_cast<unsigned long long>(f - 1) << 52) + m;
  const unsigned int top = static_cast<unsigned int>(v >> 32) | (s & 0x80000000u);
  return w2 == 0u ? 0.0 : __hiloint2double(top, static_cast<unsigned int>(v));
}

// Output (i, j) of a step by FP64 multiply-adds.
__device__ __forceinline__ double dg_direct(const DgStep& S, int i, int j) {
  const DgRecord& X = S.x;
  const int64_t ls = X.ltrans ? 1 : X.lld, rs = X.rtrans ? 1 : X.rld;
  const double* l = X.l + (X.ltrans ? static_cast<int64_t>(X.lld) * i : i) + ls * S.k0;
  const double* r = X.r + (X.rtrans ? static_cast<int64_t>(X.rld) * j : j) + rs * S.k0;
  double v = 0.0;
#pragma unroll 4
  for (int k = S.k1 - S.k0; k > 0; k--) {
    v = fma(*l, *r, v);
    l += ls;
    r += rs;
  }
  return v;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok));
  return ok != 0;
}

// 16 accumulator columns of this thread's lane, not yet waited for
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// (the registers pass through the wait, so no use of them moves before it)
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&a)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
               :
               : "memory");
}

// The running state of a CTA: the step in flight on the tensor cores and the sums so far.
// kPolls: of a wait.
template <long long kPolls>
struct DgEngine {
  DgSmem& sm;
  uint32_t tmem;
  uint32_t phase = 0u;
  bool flying = false, ok = true;
  int held = 0, cur = 1;  // exponent tables of the step in flight and of the one being staged
  int at = 0;             // record of the step in flight
  // pass 2: the sums so far, columns col .. of the thread's row
  double acc[8];

  __device__ __forceinline__ DgEngine(DgSmem& s) : sm(s), tmem(s.tmem_base) { clear(); }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] = 0.0;
  }
  // A tile of up to 32 rows: 32 rows x 8 groups of 4 columns; of up to 64: 64 x 4 groups of 8.
  __device__ __forceinline__ static int row_of(bool big) { return threadIdx.x & (big ? 63 : 31); }
  __device__ __forceinline__ static int col_of(bool big) {
    return big ? (threadIdx.x >> 6) * 8 : (threadIdx.x >> 5) * 4;
  }

  // Issues the MMAs of the staged step of 16 `halves` of K (one thread), `onto` the sums
  // there. Digit i of L meets digits 0 .. 7 - i of R.
  __device__ __forceinline__ void issue(int halves, bool onto) {
    tc_fence_after();
    const uint64_t a0 = smem_desc(smem_u32(sm.l), 128, 256), b0 = smem_desc(smem_u32(sm.r), 128, 256);
    for (int h = 0; h < halves; h++) {
      const uint64_t a = a0 + static_cast<uint64_t>(h * (kDgLBytes >> 4));
      const uint64_t b = b0 + static_cast<uint64_t>(h * (kDgRBytes >> 4));
#pragma unroll
      for (int i = 0; i < kDgDigits; i++)
        tc_mma(tmem + i * kDgCols, a + static_cast<uint64_t>((i * kDgRows * kDgRowBytes) >> 4), b,
               dg_idesc((kDgDiagonals - i) * kDgCols), (h == 0 && i == 0 && !onto) ? 0u : 1u);
    }
    tc_commit(&sm.bar);
  }

  __device__ __forceinline__ void wait() {
    if (!mbar_wait(&sm.bar, phase, kPolls)) ok = false;
    phase ^= 1u;
    tc_fence_after();
  }

  // False where the MMAs may still be running, but not asked after a wait of kTcSpinLimit polls:
  // what follows is not used then.
  __device__ __forceinline__ bool live() const { return kPolls > 0 || ok; }

  // Tensor memory -> shared memory: warp w holds rows 32 (w % 4) .. + 31 and columns
  // 16 (w / 4) .. + 15. Two diagonals make one integer, 256 i_c + i_(c+1), below 2^31.
  __device__ __forceinline__ void collect() {
    const int rows = sm.step[at].x.rows, cols = sm.step[at].x.cols;
    const int warp = threadIdx.x >> 5, quad = warp & 3, c0 = 16 * (warp >> 2);
    if (quad * 32 < rows && c0 < cols) {
      const uint32_t from = tmem + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(c0);
      int* to = sm.sums + (quad * 32 + (threadIdx.x & 31)) * kDgSumLd + c0;
#pragma unroll
      for (int c = 0; c < kDgDiagonals / 2; c++) {
        uint32_t a[16], b[16];
        tmem_ld16_async(from + 2 * c * kDgCols, a);
        tmem_ld16_async(from + (2 * c + 1) * kDgCols, b);
        tmem_wait_ld(a);
        tmem_wait_ld(b);
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          int v[4];
#pragma unroll
          for (int t = 0; t < 4; t++)
            v[t] = __float2int_rn(__uint_as_float(a[j + t])) * 256 + __float2int_rn(__uint_as_float(b[j + t]));
          *reinterpret_cast<int4*>(to + c * kDgRows * kDgSumLd + j) = make_int4(v[0], v[1], v[2], v[3]);
        }
      }
    }
    tc_fence_before();
  }

  // The value of diagonals p in units of 2^e / 2^2044: p0 2^-20 + p1 2^-36 + p2 2^-52 + p3 2^-68
  __device__ __forceinline__ static double value(int p0, int p1, int p2, int p3, unsigned int el, unsigned int er) {
    return rounded(static_cast<long long>(p0) * 65536 + p1, static_cast<long long>(p2) * 65536 + p3,
                   static_cast<int>(el + er) - 2044 - 68);
  }

  // The collected sums of a whole product, each rounded once: to memory, or times alpha into acc.
  template <int kOut, bool kEach>
  __device__ __forceinline__ void finish_whole(const DgStep& S) {
    const int r = row_of(kOut == 8), c0 = col_of(kOut == 8);
    const int* s = sm.sums + r * kDgSumLd + c0;
    const unsigned int* expo = sm.expo[held];
    const unsigned int el = expo[r];
    double* to = S.x.s + r + static_cast<int64_t>(S.x.lds) * c0;
#pragma unroll
    for (int q = 0; q < kOut; q += 4) {
      int p[4][4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const int4 t = *reinterpret_cast<const int4*>(s + c * kDgRows * kDgSumLd + q);
        p[0][c] = t.x;
        p[1][c] = t.y;
        p[2][c] = t.z;
        p[3][c] = t.w;
      }
      const uint4 e4 = *reinterpret_cast<const uint4*>(expo + kDgRows + c0 + q);
      const unsigned int er[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const double v = value(p[t][0], p[t][1], p[t][2], p[t][3], el, er[t]);
        if constexpr (kEach) {
          if (c0 + q + t < S.x.cols) *to = v;
          to += S.x.lds;
        } else {
          acc[q + t] = fma(S.x.alpha, v, acc[q + t]);
        }
      }
    }
  }

  static constexpr unsigned int kAllDirect = 1u << 16;  // all outputs of a step by multiply-adds
  // Of the staged step, the outputs (bits) of this thread that have a product near that of the
  // scales, and << 8 those that have one that is not zero.
  template <int kOut>
  __device__ __forceinline__ unsigned int weigh(int cols) const {
    if (col_of(kOut == 8) >= cols) return 0u;
    const uint4 l = sm.weight[row_of(kOut == 8)], *w = sm.weight + kDgRows + col_of(kOut == 8);
    unsigned int f = 0u;
#pragma unroll
    for (int k = 0; k < kOut; k++) {
      const unsigned int hit = (l.x & w[k].x) | (l.y & w[k].y) | (l.z & w[k].z) | (l.w & w[k].w);
      if (hit > 255u) f |= 1u << k;
      if (hit != 0u) f |= 256u << k;
    }
    return f;
  }
  // The same of any step, one output after another: a product's steps are added up in sm.part,
  // so that an item is rounded into acc once whatever its inner dimension, as on the FP64
  // pipe. f: the outputs that are formed by multiply-adds.
  template <bool kEach>
  __device__ __forceinline__ void finish_part(const DgStep& S, unsigned int f) {
    const bool big = S.x.rows > 32;
    const int r = row_of(big), c0 = col_of(big), n = min(big ? 8 : 4, S.x.cols - c0);
    const int* s = sm.sums + r * kDgSumLd + c0;
    const unsigned int* expo = sm.expo[held];
#pragma unroll 1
    for (int k = 0; k < n; k++) {
      double v;
      if (f >> k & 1u)
        v = dg_direct(S, r, c0 + k);
      else
        v = value(s[k], s[k + kDgRows * kDgSumLd], s[k + 2 * kDgRows * kDgSumLd], s[k + 3 * kDgRows * kDgSumLd],
                  expo[r], expo[kDgRows + c0 + k]);
      if (!S.first) v += sm.part[k][threadIdx.x];
      if (kEach && S.last) S.x.s[r + static_cast<int64_t>(S.x.lds) * (c0 + k)] = v;
      else sm.part[k][threadIdx.x] = v;
    }
    if (!kEach && S.last) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k < n) acc[k] = fma(S.x.alpha, sm.part[k][threadIdx.x], acc[k]);
    }
  }

  // A step's sums (collected), `weighed` by weigh or kAllDirect.
  template <bool kEach>
  __device__ __forceinline__ void finish(unsigned int weighed) {
    const DgStep& S = sm.step[at];
    const bool big = S.x.rows > 32;
    const int r = row_of(big), c0 = col_of(big);
    if (r >= S.x.rows || c0 >= S.x.cols) return;
    const unsigned int f = (weighed >= kAllDirect ? 255u : weighed >> 8 & ~weighed) &
                           ((1u << min(S.x.cols - c0, big ? 8 : 4)) - 1u);
    if (!S.first || !S.last) {
      finish_part<kEach>(S, f);
      return;
    }
    // the outputs that are formed by multiply-adds: zeros for their sums, and themselves afterwards
    for (unsigned int g = f; g != 0u; g &= g - 1u)
#pragma unroll
      for (int c = 0; c < kDgDiagonals / 2; c++)
        sm.sums[(c * kDgRows + r) * kDgSumLd + c0 + __ffs(static_cast<int>(g)) - 1] = 0;
    if (big) finish_whole<8, kEach>(S);
    else finish_whole<4, kEach>(S);
    if (f == 0u) return;
    for (unsigned int g = f; g != 0u; g &= g - 1u) {
      const int k = __ffs(static_cast<int>(g)) - 1;
      const double v = dg_direct(S, r, c0 + k);
      if constexpr (kEach) S.x.s[r + static_cast<int64_t>(S.x.lds) * (c0 + k)] = v;
      else sm.part[k][threadIdx.x] = v;
    }
    if constexpr (!kEach) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (f >> k & 1u) acc[k] = fma(S.x.alpha, sm.part[k][threadIdx.x], acc[k]);
    }
  }
};

// Streams the products of sm.rec through the engine. Src: count(); prepare(q), called by all
// threads before record q is read (it may refill sm.rec and hold barriers), returns its slot.
// kEach: every product goes to its place in memory; else the sums of all add up in the engine.
template <bool kEach, long long kPolls, class Src>
__device__ __forceinline__ bool dg_stream(DgEngine<kPolls>& E, Src& src) {
  DgSmem& sm = E.sm;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  // The digits are cut first by the warps that hold no tile rows of tensor memory (those of
  // quadrants 2 and 3), which need not copy sums meanwhile: warps 2, 3, 6, 7, 1, 5, 0, 4.
  const int utid = static_cast<int>((0x32571046u >> (4 * warp)) & 0xfu) * 32 + lane;

  int q = 0, k0 = 0, slot = 0;
  bool more = false;
  const int n = src.count();
  auto seek = [&]() {  // the first product with an inner dimension at or after q
    more = false;
    for (; q < n; q++) {
      slot = src.prepare(q);
      if (sm.rec[slot].k > 0) {
        k0 = 0;
        more = true;
        return;
      }
    }
  };
  // The step's units: rows of L, then rows of R, over its k groups; this thread's first and
  // second. Packed: row | k group << 8 | (of L) << 12 | valid << 13.
  DgUnit u0, u1;
  int w0 = 0, w1 = 0;
  bool same_l = false, same_r = false;  // the operand is that of the step before, already cut
  auto fetch = [&](DgUnit& u, int e) -> int {
    const DgRecord& X = sm.rec[slot];
    const int rows = X.rows, cols = X.cols, rem = X.k - k0, kgc = rem > 16 ? 4 : 2;
    const int lsh = rows > 32 ? 6 : 5, rsh = cols > 16 ? 5 : 4;
    const int nl = same_l ? 0 : kgc << lsh, nr = same_r ? 0 : kgc << rsh;
    if (e >= nl + nr) return 0;
    const bool is_l = e < nl;
    const int f = is_l ? e : e - nl, sh = is_l ? lsh : rsh, row = f & ((1 << sh) - 1), kg = f >> sh;
    if (row >= (is_l ? rows : cols)) return is_l ? 1 << 12 : 0;
    dg_load(u, is_l ? X.l : X.r, is_l ? X.lld : X.rld, is_l ? X.ltrans : X.rtrans, row, k0 + 8 * kg, rem - 8 * kg);
    return row | kg << 8 | (is_l ? 1 << 12 : 0) | 1 << 13;
  };
  auto cut = [&](const DgUnit& u, int w, const unsigned int* expo, bool short_k) {
    if (!(w & (1 << 13))) return;
    const int row = w & 0xff, kg = (w >> 8) & 0xf;
    if (w & (1 << 12)) {
      dg_store<kDgRows>(u, expo[row], sm.l, kDgLBytes, row, kg);
      uint32_t* weight = reinterpret_cast<uint32_t*>(&sm.weight[row]);
      weight[kg] = dg_weight(u, expo[row]);
      if (short_k) weight[kg + 2] = 0u;
    } else {
      dg_store<kDgCols>(u, expo[kDgRows + row], sm.r, kDgRBytes, row, kg);
      // the classes in reverse, so that d <= 1, 3, 5 of L meet d <= 5, 3, 1 of R
      reinterpret_cast<uint32_t*>(&sm.weight[kDgRows + row])[kg] =
          __byte_perm(dg_weight(u, expo[kDgRows + row]), 0u, 0x1230);
    }
  };

  unsigned int pweighed = 0u;  // of the step in flight
  seek();
  if (more) {
    w0 = fetch(u0, utid);
    w1 = fetch(u1, utid + kDgThreads);
  }
  while (more) {
    unsigned int* expo = sm.expo[E.cur];
    const unsigned int* before = sm.expo[E.held];
    // the rows' and columns' largest exponents, or those already there
    if (w0 & (1 << 13)) atomicMax(expo + (w0 & 0xff) + (w0 & (1 << 12) ? 0 : kDgRows), dg_exponent(u0));
    if (w1 & (1 << 13)) atomicMax(expo + (w1 & 0xff) + (w1 & (1 << 12) ? 0 : kDgRows), dg_exponent(u1));
    if (tid < kDgRows + kDgCols && (tid < kDgRows ? same_l : same_r)) expo[tid] = before[tid];
    __syncthreads();
    const int spare = 3 - E.held - E.cur;  // last read a step ago
    bool odd = false;  // a scale so small or large that a result may leave the normal range, an infinity or a NaN
    if (tid < kDgRows + kDgCols) {
      sm.expo[spare][tid] = 0u;
      const unsigned int x = expo[tid];
      odd = x != 0u && x - kDgExpoMin > kDgExpoMax - kDgExpoMin;
    }
    // The second 32 of K go onto the first ones' sums where their scales will do: the sums of
    // 64 products of a diagonal are exact as well, and pairs of them below 2^31.
    bool onto = false;
    if (k0 == kDgK && E.flying) onto = !__syncthreads_or(tid < kDgRows + kDgCols && expo[tid] > before[tid]);
    if (E.flying) {
      E.wait();
      if (!onto && E.live()) E.collect();
    }
    // the digits (the MMAs that read the buffers are done) and weights
    if (E.live()) {
      const bool short_k = sm.rec[slot].k - k0 <= 16;
      cut(u0, w0, onto ? before : expo, short_k);
      cut(u1, w1, onto ? before : expo, short_k);
    }
    fence_async_smem();
    odd = __syncthreads_or(!E.ok || odd);
    if (odd && __syncthreads_or(!E.ok)) return false;
    const DgRecord& X = sm.rec[slot];
    const int rem = X.k - k0;
    if (warp == kDgIssuer) {
      if (elect_one()) E.issue(rem > 16 ? 2 : 1, onto);
      __syncwarp();
    }
    const int rows = X.rows, cols = X.cols;
    const bool first = k0 == 0, last = rem <= kDgK;
    const unsigned int weighed = odd         ? E.kAllDirect
                                 : rows > 32 ? E.template weigh<8>(cols)
                                             : E.template weigh<4>(cols);
    if (tid == 0) {
      DgStep& S = sm.step[onto ? E.at : E.at ^ 1];
      S.k1 = k0 + min(rem, kDgK);
      S.last = last;
      if (!onto) {
        S.x = X;
        S.k0 = k0;
        S.first = first;
      }
    }
    // the next step's operands; an operand that this step staged as well is not read again
    same_l = same_r = false;
    if (!last) {
      k0 += kDgK;
    } else {
      const double *l = X.l, *r = X.r;
      const int lld = X.lld, rld = X.rld, k = X.k, trans = X.ltrans | X.rtrans << 8;
      q++;
      seek();
      if (more && first) {
        const DgRecord& N = sm.rec[slot];
        same_l = N.k == k && N.l == l && N.lld == lld && N.ltrans == (trans & 0xff) && N.rows == rows;
        same_r = N.k == k && N.r == r && N.rld == rld && N.rtrans == trans >> 8 && N.cols == cols;
      }
    }
    if (more) {
      w0 = fetch(u0, utid);
      w1 = fetch(u1, utid + kDgThreads);
    }
    if (E.flying && !onto) E.template finish<kEach>(pweighed);
    E.flying = true;
    if (!onto) {
      E.held = E.cur;
      E.at ^= 1;
    }
    E.cur = spare;
    pweighed = onto ? pweighed | weighed : weighed;
  }
  if (E.flying) {
    __syncthreads();  // the last sums have been read
    E.wait();
    if (E.live()) E.collect();
    if (__syncthreads_or(!E.ok)) return false;
    E.template finish<kEach>(pweighed);
    E.flying = false;
  }
  return true;
}

// Pass 1: a batch of job tiles, each in up to two column halves.
struct DgInterSource {
  int units;
  __device__ __forceinline__ int count() const { return units; }
  __device__ __forceinline__ int prepare(int q) const { return q; }
};

// Pass 2: the items of a tile half, their records made from the item list kDgBatch at a time.
struct DgSumSource {
  const SumItem* items;
  int item0, item1;
  const SlotPtrs& sp;
  DgSmem& sm;
  int row0, col0, rows, cols;
  int held = -1;  // first item held (uniform)
  __device__ __forceinline__ int count() const { return item1 - item0; }
  __device__ __forceinline__ int prepare(int q) {
    if (held < 0 || q >= held + kDgBatch) {  // q never goes back
      __syncthreads();
      const int n = min(kDgBatch, item1 - item0 - q);
      if (static_cast<int>(threadIdx.x) < n) {
        const SumItem I = items[item0 + q + threadIdx.x];
        DgRecord d{};
        d.k = I.k;
        if (I.k > 0) {
          d.l = resolve<double>(sp, I.l.ref) + (I.l.trans ? static_cast<int64_t>(I.l.ld) * row0 : row0);
          d.r = resolve<double>(sp, I.r.ref) + (I.r.trans ? col0 : static_cast<int64_t>(I.r.ld) * col0);
        }
        d.lld = I.l.ld;
        d.rld = I.r.ld;
        d.ltrans = I.l.trans != 0;
        d.rtrans = I.r.trans == 0;  // a row of R's digits is a column of op(R)
        d.alpha = I.alpha;
        d.rows = static_cast<int16_t>(rows);
        d.cols = static_cast<int16_t>(cols);
        sm.rec[threadIdx.x] = d;
      }
      held = q;
      __syncthreads();
    }
    return q - held;
  }
};

__device__ void dg_setup(DgSmem& sm) {
  if (threadIdx.x == 0) {
    mbar_init(&sm.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < 3 * (kDgRows + kDgCols); i += kDgThreads)
    sm.expo[i / (kDgRows + kDgCols)][i % (kDgRows + kDgCols)] = 0u;
  fence_async_smem();
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(kDgTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

__device__ void dg_teardown(uint32_t tmem_d) {
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kDgTmemCols) : "memory");
  }
}

// The next `take` of the work list.
__device__ __forceinline__ int dg_next(unsigned int* sched, int* slot, int take) {
  __syncthreads();  // the previous work's epilogue is done in every thread
  if (threadIdx.x == 0) *slot = static_cast<int>(atomicAdd(sched, static_cast<unsigned int>(take)));
  __syncthreads();
  return *slot;
}

template <long long kPolls>
__device__ __forceinline__ void dg_end(DgEngine<kPolls>& E, unsigned int* sched, int* err) {
  if (__syncthreads_or(!E.ok)) {
    if (threadIdx.x == 0 && err) atomicOr(err, 2);
    mbar_wait(&E.sm.bar, E.phase ^ 1u);  // the MMAs still in flight, bounded again
  }
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(sched + 1, 1u) == gridDim.x - 1) {
    sched[0] = 0u;
    sched[1] = 0u;
  }
  dg_teardown(E.tmem);
}

// The records of pass 1's job tiles first .. first + n - 1, the two column halves of each.
__device__ __forceinline__ void dg_inter_batch(DgSmem& sm, const InterJob* __restrict__ jobs,
                                               const GemmTile* __restrict__ tiles, int first, int n,
                                               const SlotPtrs& sp) {
  if (static_cast<int>(threadIdx.x) < 2 * n) {
    const GemmTile T = tiles[first + (threadIdx.x >> 1)];
    const InterJob J = jobs[T.idx];
    const int row0 = (T.pos >> 16) * 64, col0 = (T.pos & 0xffff) * 64 + (threadIdx.x & 1) * kDgCols;
    DgRecord d{};
    d.rows = static_cast<int16_t>(min(64, J.m - row0));
    d.cols = static_cast<int16_t>(min(kDgCols, J.n - col0));
    d.k = d.cols > 0 ? J.k : 0;
    if (d.cols > 0) {
      d.l = resolve<double>(sp, J.l.ref) + (J.l.trans ? static_cast<int64_t>(J.l.ld) * row0 : row0);
      d.r = resolve<double>(sp, J.r.ref) + (J.r.trans ? col0 : static_cast<int64_t>(J.r.ld) * col0);
      d.s = sp.inter + J.off + row0 + static_cast<int64_t>(J.m) * col0;
    }
    d.alpha = 1.0;
    d.lld = J.l.ld;
    d.rld = J.r.ld;
    d.lds = J.m;
    d.ltrans = J.l.trans != 0;
    d.rtrans = J.r.trans == 0;
    sm.rec[threadIdx.x] = d;
  }
  __syncthreads();
}

// The rest of pass 1 for a CTA that gave up a wait: NaN in place of the products of the batch of n
// job tiles that it has and of all that it takes after it.
__device__ __noinline__ void dg_inter_nothing(DgSmem& sm, int n, const InterJob* jobs, const GemmTile* tiles,
                                              int ntiles, int take, const SlotPtrs& sp, unsigned int* sched) {
  for (;;) {
    for (int q = 0; q < 2 * n; q++) {
      const DgRecord& X = sm.rec[q];
      if (X.k > 0)
        for (int e = threadIdx.x; e < X.rows * X.cols; e += kDgThreads)
          X.s[e % X.rows + static_cast<int64_t>(X.lds) * (e / X.rows)] = CUDART_NAN;
    }
    const int first = dg_next(sched, &sm.slot, take);
    if (first >= ntiles) return;
    n = min(take, ntiles - first);
    dg_inter_batch(sm, jobs, tiles, first, n, sp);
  }
}

// The same of pass 2, from tile half t on; its tiles still meet at their counters.
__device__ __noinline__ void dg_sum_nothing(DgSmem& sm, int t, const SumGroup* groups, const GemmTile* tiles,
                                            int ntiles, double* partials, unsigned int* counters, const SlotPtrs& sp,
                                            unsigned int* sched) {
  for (; t < 2 * ntiles; t = dg_next(sched, &sm.slot, 1)) {
    const GemmTile T = tiles[t >> 1];
    const SumGroup G = groups[T.idx];
    const int row0 = (T.pos >> 16) * 64, col0 = (T.pos & 0xffff) * 64, off = (t & 1) * kDgCols;
    const int tm = min(64, G.m - row0), width = min(64, G.n - col0);
    if (off >= width) continue;
    bool last = true;  // and the tile's other half goes with it
    if (T.nsplit > 1) {
      const int TM = 16 * ((T.shape & 3) + 1), TN = 16 * (((T.shape >> 2) & 3) + 1);
      double* part = partials + T.part + static_cast<int64_t>(T.split) * TM * TN + TM * off;
      for (int e = threadIdx.x; e < tm * min(kDgCols, width - off); e += kDgThreads)
        __stcg(part + e % tm + TM * (e / tm), CUDART_NAN);
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0)
        sm.is_last = atomicAdd(counters + T.counter, 1u) ==
                     static_cast<unsigned>(T.nsplit * ((width + kDgCols - 1) / kDgCols) - 1);
      __syncthreads();
      last = sm.is_last;
      if (last && threadIdx.x == 0) counters[T.counter] = 0u;
    }
    double* O = const_cast<double*>(resolve<double>(sp, G.out)) + row0 + static_cast<int64_t>(G.ldo) * col0;
    if (last)
      for (int e = threadIdx.x; e < tm * width; e += kDgThreads)
        O[e % tm + static_cast<int64_t>(G.ldo) * (e / tm)] = CUDART_NAN;
  }
}

// Pass 1, `take` job tiles at a time.
template <long long kPolls>
__global__ void __launch_bounds__(kDgThreads, kDgCtasPerSm)
    inter_digits_kernel(const InterJob* __restrict__ jobs, const GemmTile* __restrict__ tiles, int ntiles, int take,
                        SlotPtrs sp, unsigned int* sched, int* err) {
  extern __shared__ unsigned char dyn[];
  DgSmem& sm = *reinterpret_cast<DgSmem*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
  dg_setup(sm);
  DgEngine<kPolls> E(sm);
  for (;;) {
    const int first = dg_next(sched, &sm.slot, take);
    if (first >= ntiles) break;
    const int n = min(take, ntiles - first);
    dg_inter_batch(sm, jobs, tiles, first, n, sp);
    DgInterSource src{2 * n};
    if (!dg_stream<true>(E, src)) {
      dg_inter_nothing(sm, n, jobs, tiles, ntiles, take, sp, sched);
      break;
    }
  }
  dg_end(E, sched, err);
}

// Pass 2: the column halves of the tiles one after another; a tile at most 32 columns wide
// has one.
template <long long kPolls>
__global__ void __launch_bounds__(kDgThreads, kDgCtasPerSm)
    sum_digits_kernel(const SumGroup* __restrict__ groups, const SumItem* __restrict__ items,
                      const GemmTile* __restrict__ tiles, int ntiles, double* partials, unsigned int* counters,
                      SlotPtrs sp, unsigned int* sched, int* err) {
  extern __shared__ unsigned char dyn[];
  DgSmem& sm = *reinterpret_cast<DgSmem*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
  dg_setup(sm);
  DgEngine<kPolls> E(sm);
  for (;;) {
    const int t = dg_next(sched, &sm.slot, 1);
    if (t >= 2 * ntiles) break;
    const GemmTile T = tiles[t >> 1];
    const SumGroup G = groups[T.idx];
    const int row0 = (T.pos >> 16) * 64, tcol0 = (T.pos & 0xffff) * 64, off = (t & 1) * kDgCols, col0 = tcol0 + off;
    const int tm = min(64, G.m - row0), tn = min(kDgCols, G.n - col0);
    if (tn <= 0) continue;
    E.clear();
    DgSumSource src{items, T.item0, T.item1, sp, sm, row0, col0, tm, tn};
    if (!dg_stream<false>(E, src)) {
      dg_sum_nothing(sm, t, groups, tiles, ntiles, partials, counters, sp, sched);
      break;
    }
    const bool big = tm > 32, mine = E.row_of(big) < tm;
    const int r = E.row_of(big), c0 = E.col_of(big), nout = big ? 8 : 4;
    // items without an inner dimension: out += alpha op(R)
    if (mine)
      for (int it = T.item0; it < T.item1; it++) {
        const SumItem& I = items[it];
        if (I.k > 0) continue;
        const double* R = resolve<double>(sp, I.r.ref);
        const int64_t si = I.r.trans ? I.r.ld : 1, sj = I.r.trans ? 1 : I.r.ld;
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (k < nout && c0 + k < tn) E.acc[k] = fma(I.alpha, R[(row0 + r) * si + (col0 + c0 + k) * sj], E.acc[k]);
      }
    double* O = const_cast<double*>(resolve<double>(sp, G.out));
    const int64_t ldo = G.ldo;
    const bool accum = (G.flags & kAccumulate) != 0;
    if (T.nsplit == 1) {
      if (mine)
#pragma unroll
        for (int k = 0; k < 8; k++)
          if (k < nout && c0 + k < tn) {
            const int64_t idx = (row0 + r) + ldo * (col0 + c0 + k);
            O[idx] = accum ? O[idx] + E.acc[k] : E.acc[k];
          }
      continue;
    }
    // a split tile: the last unit (split x column half) to arrive adds the splits in order
    const int TM = 16 * ((T.shape & 3) + 1), TN = 16 * (((T.shape >> 2) & 3) + 1);
    double* part = partials + T.part;
    const int64_t te = static_cast<int64_t>(TM) * TN;
    if (mine)
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k < nout && c0 + k < tn) __stcg(part + T.split * te + r + TM * (off + c0 + k), E.acc[k]);
    const int width = min(64, G.n - tcol0);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
      sm.is_last = atomicAdd(counters + T.counter, 1u) ==
                   static_cast<unsigned>(T.nsplit * ((width + kDgCols - 1) / kDgCols) - 1);
    __syncthreads();
    if (!sm.is_last) continue;
    __threadfence();
    if (threadIdx.x == 0) counters[T.counter] = 0u;  // ready for the next launch
    for (int e = threadIdx.x; e < tm * width; e += kDgThreads) {
      const int i = e % tm, c = e / tm;
      double v = 0.0;
      for (int s = 0; s < T.nsplit; s++) v += __ldcg(part + s * te + i + TM * c);
      const int64_t idx = (row0 + i) + ldo * (tcol0 + c);
      O[idx] = accum ? O[idx] + v : v;
    }
  }
  dg_end(E, sched, err);
}

constexpr int kDgSmemBytes = static_cast<int>(sizeof(DgSmem)) + 1024;

int dg_grid(int units) {
  static const int sms = [] {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 152;
    return n;
  }();
  return std::min(units, kDgCtasPerSm * sms);
}

}  // namespace

cudaError_t launch_inter_digits(const InterJob* jobs, const GemmTile* tiles, int ntiles, const SlotPtrs& sp,
                                unsigned int* sched, int* err, cudaStream_t stream, bool give_up) {
  if (ntiles <= 0) return cudaSuccess;
  const auto kernel = give_up ? inter_digits_kernel<0> : inter_digits_kernel<kTcSpinLimit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDgSmemBytes);
  if (e != cudaSuccess) return e;
  const int grid = dg_grid(ntiles);
  // several batches a CTA, so that no CTA is left with a long one at the end
  const int take = std::max(1, std::min(kDgBatch / 2, ntiles / (4 * grid)));
  kernel<<<grid, kDgThreads, kDgSmemBytes, stream>>>(jobs, tiles, ntiles, take, sp, sched, err);
  return cudaGetLastError();
}

cudaError_t launch_sum_digits(const SumGroup* groups, const SumItem* items, const GemmTile* tiles, int ntiles,
                              double* partials, unsigned int* counters, const SlotPtrs& sp, unsigned int* sched,
                              int* err, cudaStream_t stream, bool give_up) {
  if (ntiles <= 0) return cudaSuccess;
  const auto kernel = give_up ? sum_digits_kernel<0> : sum_digits_kernel<kTcSpinLimit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDgSmemBytes);
  if (e != cudaSuccess) return e;
  kernel<<<dg_grid(2 * ntiles), kDgThreads, kDgSmemBytes, stream>>>(groups, items, tiles, ntiles, partials, counters,
                                                                  sp, sched, err);
  return cudaGetLastError();
}

}  // namespace c2g
