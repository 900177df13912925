// Complex FP64 GEMM on the 5th-generation tensor cores (tcgen05.mma kind::f16) by exact
// digit slicing (the Ozaki scheme), for the framework's FP64 contractions:
//   becp = conj(beta) psi^T and V_NL psi = beta^T (D becp)   (nonlocal_op.py:67-82)
//   the refinement's projections X^H Y and rotations U X      (solver/davidson.py:48-61)
//
//   C[i][j] = sum_k op(A)[i][k] op(B)[k][j],   complex128 in and out.
//
// GB300 runs FP64 FMA at 1.06 TFLOP/s (measured), 1/1800 of its FP16 tensor rate, so the
// contraction is done on integers instead.  With E the binary exponent of the largest
// |re|, |im| of a row of op(A) (a column of op(B)), every component x becomes the integer
//   q = round(x 2^(B - E)),  |q| <= 2^B,  B = 62 (S = 8 digits) or 55 (S = 7 digits),
// written in balanced base 256, q = sum_s d_s 256^(S-1-s), -128 <= d_s <= 128.  A digit is exact in
// FP16 and a product of two is at most 2^14.  The products d_s(a) d_t(b) of one level l = s + t share a
// weight and one FP32 accumulator in tensor memory; levels 0 .. S-1 are kept (S (S + 1) / 2 digit products per real
// product).  Every 128 k the accumulators are emptied into 64-bit integers, and the only rounding after that is
// the conversion to FP64.
//   Accuracy is that of fixed point, relative to max|A_i.| max|B_j.| of an output's row and column and not to the
// output or to its terms: where a large component of one meets a zero or a small one of the other, and only small
// ones meet, the result has fewer correct digits than an FP64 sum (K = 512, a 1 against a zero, the rest 10^-6
// against 1: 1e-13 of sum|a b| with 8 digits, 7e-12 with 7; 10^-3: 2e-16, 1e-14).  In units of the two maxima:
//   slicing, per term: 2^-61 (S = 8), 2^-54 (S = 7); what the dropped levels hold at most, digits aligned: 2^-56, 2^-50
//     per term, on data whose digits are not about sqrt(K) 2^-60, sqrt(K) 2^-54 in all;
//   accumulators: a level's sum over 128 k is below 2^24 and exact up to level 3, and beyond it unless digits are aligned
//     (256 (l + 1) products of 2^14 are 2^25 at most); then each MMA may drop units of that level, 2^-52 and
//     smaller ones (l >= 5) against a sum of at least 2^6.
// That is within the normwise error of an FP64 sum, 2^-53 |A_i.| |B_j.|, for S = 8 up to K of 10^5, and of the
// double-float form (2^-48) for S = 7.
// Rows or columns that hold an infinity or a NaN are summed in plain FP64 at the end.
//
// Three kernels (for up to 96 k the first two are one, k_oz_prep):
//   k_oz_max   exponent of every row / column (one pass over each operand);
//   k_oz_pack  digits into the operand layout of the MMA: per 16 k, real part then imaginary
//              part, S slices each, a slice being 128 (A) or 32 (B) rows of 16 k in no-swizzle
//              core matrices (8 rows x 16 bytes), so one stage of the GEMM is one contiguous block;
//   k_oz_gemm  a CTA owns 128 x 32 complex outputs: the 512 columns of tensor memory hold S
//              levels x 32 columns of the real and the imaginary accumulator.  The B slices
//              lie side by side along N, so slice s of A times B slices 0 .. S-1-s is one MMA of
//              N = 32 (S - s) columns that lands on levels s .. S-1: 8 MMAs per part pair
//              instead of 36.  One thread copies operands (cp.async.bulk), one issues MMAs, sixteen
//              warps empty the accumulators.  K is split across CTAs; the split sums are
//              added in a fixed order.
// MMA time bounds it: 32 MMAs per 16 k, about 2,500 cycles for 128 x 32 x 16 complex products
// (the narrow ones wait for shared-memory operands, 4 KB per slice of A), a ceiling near
// 64 TFLOP/s of complex FP64 work on 152 SMs.  Measured with the passes over the operands:
//   becp, P 256, 160 bands, nG 23,847   14.34 ms (FP64 SIMT)        -> 0.37 ms
//   apply of the same size              12.02 ms (FP64 SIMT)        -> 0.45 ms
//   conj(X) Y^T, 168 x 336 x 23,847      3.33 ms (double-float SIMT) -> 0.45 ms
#include <algorithm>

#include "common.cuh"
#include "mma16.cuh"
#include "ozgemm.cuh"
#include "ozlayout.hpp"

namespace addft {

namespace {

__device__ unsigned g_oz_error = 0;   // bit 0: a bounded wait ran out

constexpr int kRowsA = kOzRowsA, kRowsB = kOzRowsB, kStep = kOzStep, kDrain = kOzDrain;
constexpr int kOzWait = 1 << 24;
constexpr int kEpiWarps = 16;              // warps that empty the accumulators
constexpr int kEpiCols = kRowsB / (kEpiWarps / 4);   // columns of each
constexpr int kOzThreads = 32 * (kEpiWarps + 2);     // one for copies, one for MMAs
constexpr int kSms = kOzSms;
constexpr size_t kOzScratchCap = size_t(384) << 20;   // scratch asked for; more K, rows or batch go in pieces

template <int S>
struct Oz {
  static constexpr int kBits = S == 8 ? 62 : 8 * S - 1;
  static constexpr int kABytes = 2 * S * kRowsA * kStep * 2;   // one stage of A
  static constexpr int kBBytes = 2 * S * kRowsB * kStep * 2;
  // A in a ring of parts (re, im of a stage are two items), B in a ring of stages: 208 KB (S = 8).
  // Whole stages of both, twice buffered, left the copy of one stage to the MMAs of one: 2.6 us per
  // stage where the MMAs take 1.25.
  static constexpr int kAItem = kABytes / 2, kARing = 5, kBRing = 3;
  static constexpr size_t kSmem = (size_t)kARing * kAItem + kBRing * kBBytes + 1024;
};

// ---------------------------------------------------------------------------
// exponents: ex[row] = largest exponent field of |re|, |im| over k (0x7ff: not finite)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int expo(double2 v) {
  return max((__double2hiint(v.x) >> 20) & 0x7ff, (__double2hiint(v.y) >> 20) & 0x7ff);
}

// ROWMAJOR (k contiguous): a warp per row and k chunk; else a thread per row and k chunk
template <bool ROWMAJOR>
__global__ void __launch_bounds__(256)
k_oz_max(const double2 *__restrict__ X, long s_row, long s_k, size_t s_batch, int rows, int K, int kchunk,
         int *__restrict__ ex) {
  const int k0 = blockIdx.y * kchunk, k1 = min(K, k0 + kchunk);
  const double2 *Xb = X + blockIdx.z * s_batch;
  int m = 0;
  int row;
  if (ROWMAJOR) {
    row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row < rows)
      for (int k = k0 + (threadIdx.x & 31); k < k1; k += 32) m = max(m, expo(Xb[row * s_row + k * s_k]));
    m = __reduce_max_sync(0xffffffffu, m);
    if (threadIdx.x & 31) return;
  } else {
    row = blockIdx.x * 256 + threadIdx.x;
    if (row < rows)
      for (int k = k0; k < k1; ++k) m = max(m, expo(Xb[row * s_row + k * s_k]));
  }
  if (row < rows && m > 0) atomicMax(ex + (size_t)blockIdx.z * rows + row, m);
}

// ---------------------------------------------------------------------------
// digits
// ---------------------------------------------------------------------------
// x -> q = round(x 2^(bits - E)) of a row whose exponent field is em, plus 128 in every byte but
// the top one: byte s of the result minus 128 is then the balanced digit.
template <int S>
__device__ __forceinline__ uint64_t oz_bytes(double x, int em) {
  const uint64_t u = (uint64_t)__double_as_longlong(x);
  const int e = (int)(u >> 52) & 0x7ff;
  uint64_t m = u & 0xFFFFFFFFFFFFFull;
  if (e) m |= 1ull << 52;
  const int sh = Oz<S>::kBits - 53 - (max(em, 1) - max(e, 1));
  uint64_t q;
  if (sh >= 0) {
    q = m << sh;
  } else {
    const int r = min(-sh, 63);
    q = (m + (1ull << (r - 1))) >> r;
  }
  if ((int64_t)u < 0) q = 0 - q;
  constexpr uint64_t kBias = S == 8 ? 0x0080808080808080ull : 0x0000808080808080ull;
  return q + kBias;
}

// 8 k of one row: one 16-byte core-matrix row per part and slice
template <int S, int R>
__device__ __forceinline__ void oz_octet(const double2 *x, int em, int conj, unsigned char *dst) {
  constexpr int kSlice = R * kStep * 2;   // bytes of one slice
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    uint64_t q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const double2 v = x[j];
      // rows that are not finite are left to the FP64 sum of the GEMM's epilogue
      q[j] = oz_bytes<S>(em == 0x7ff ? 0.0 : (part ? (conj ? -v.y : v.y) : v.x), em);
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      uint32_t h[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = digit_pair<S>(q[2 * j], q[2 * j + 1], s);
      *reinterpret_cast<uint4 *>(dst + (size_t)(part * S + s) * kSlice) = make_uint4(h[0], h[1], h[2], h[3]);
    }
  }
}

// A CTA packs R rows x 2048 / R k: a coalesced read into shared memory, then a thread per row
// and 8 k writes one 16-byte core-matrix row per part and slice.
template <int S, int R>
__global__ void __launch_bounds__(256)
k_oz_pack(const double2 *__restrict__ X, long s_row, long s_k, size_t s_batch, int conj, int rows, int K, int nks,
          const int *__restrict__ ex, unsigned char *__restrict__ out, size_t out_batch) {
  constexpr int KT = 2048 / R;
  constexpr int kSlice = R * kStep * 2;   // bytes of one slice
  __shared__ double2 T[R * (KT + 1)];
  const int r0 = blockIdx.y * R, k0 = blockIdx.x * KT;
  const double2 *Xb = X + blockIdx.z * s_batch;
  const bool kfast = s_k == 1;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int i = threadIdx.x + 256 * t;
    const int r = kfast ? i / KT : i % R, k = kfast ? i % KT : i / R;
    double2 v = make_double2(0.0, 0.0);
    if (r0 + r < rows && k0 + k < K) v = Xb[(r0 + r) * s_row + (k0 + k) * s_k];
    T[r * (KT + 1) + k] = v;
  }
  __syncthreads();
  const int r = threadIdx.x % R, oct = threadIdx.x / R;
  const int step = k0 / kStep + oct / 2;
  // rows of a tile beyond the operand's stay unwritten: each only reaches its own, unused, outputs
  if (step >= nks || r0 + r >= rows) return;
  const int em = ex[(size_t)blockIdx.z * rows + r0 + r];
  unsigned char *dst = out + blockIdx.z * out_batch + ((size_t)blockIdx.y * nks + step) * (2 * S * kSlice) +
                       (r >> 3) * 256 + (oct & 1) * 128 + (r & 7) * 16;
  oz_octet<S, R>(T + r * (KT + 1) + oct * 8, em, conj, dst);
}

// Both operands of a product of few k (kPrepSteps stages) in one launch: a CTA holds 64 rows of A or 32 of B with all
// their k, finds the exponents and writes the digits.  The passes by themselves are a memset and four launches, and these
// small products are launches: rotations of 16 x 16 x 6,000 to 32 x 32 x 9,000 36 to 39 us with them (20 to 26
// in double-float arithmetic, which holds fewer bits), 24 to 26 so.  Bits are those of the passes.
constexpr int kPrepSteps = 6;      // 96 k: 99 KB of shared memory, two CTAs per SM
constexpr int kPrepA = 64, kPrepB = kRowsB;
inline size_t prep_smem(int nks) { return (size_t)kPrepA * (nks * kStep + 1) * sizeof(double2); }

struct PrepArgs {
  const double2 *X;
  long s_row, s_k;
  size_t s_batch;
  int conj, rows;
  int *ex;
  unsigned char *out;
  size_t out_batch;
};

template <int S, int R, int RB>   // RB rows per CTA, R per tile
__device__ __forceinline__ void oz_prep(const PrepArgs &a, int blk, int K, int nks, double2 *T) {
  constexpr int kPer = 256 / RB;   // threads per row
  __shared__ int mx[256];
  const int r0 = blk * RB, Kp = nks * kStep, pitch = Kp + 1;
  const double2 *Xb = a.X + blockIdx.y * a.s_batch;
  const bool kfast = a.s_k == 1;
  for (int i = threadIdx.x; i < RB * Kp; i += 256) {
    const int r = kfast ? i / Kp : i % RB, k = kfast ? i % Kp : i / RB;
    T[r * pitch + k] = r0 + r < a.rows && k < K ? Xb[(r0 + r) * a.s_row + k * a.s_k] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int r = threadIdx.x % RB, part = threadIdx.x / RB;
  int em = 0;
  for (int k = part; k < Kp; k += kPer) em = max(em, expo(T[r * pitch + k]));
  mx[threadIdx.x] = em;
  __syncthreads();
  for (int p = 0; p < kPer; ++p) em = max(em, mx[p * RB + r]);
  if (r0 + r >= a.rows) return;
  if (part == 0) a.ex[(size_t)blockIdx.y * a.rows + r0 + r] = em;
  const int rt = r0 % R + r;   // row in its tile
  unsigned char *tile = a.out + blockIdx.y * a.out_batch + (size_t)(r0 / R) * nks * (2 * S * R * kStep * 2);
  for (int oct = part; oct < 2 * nks; oct += kPer)
    oz_octet<S, R>(T + r * pitch + oct * 8, em, a.conj,
                   tile + (size_t)(oct / 2) * (2 * S * R * kStep * 2) + (rt >> 3) * 256 + (oct & 1) * 128 + (rt & 7) * 16);
}

template <int S>
__global__ void __launch_bounds__(256) k_oz_prep(PrepArgs a, PrepArgs b, int ctas_a, int K, int nks) {
  extern __shared__ __align__(16) double2 prep_smem_[];
  if ((int)blockIdx.x < ctas_a) oz_prep<S, kRowsA, kPrepA>(a, blockIdx.x, K, nks, prep_smem_);
  else oz_prep<S, kRowsB, kPrepB>(b, blockIdx.x - ctas_a, K, nks, prep_smem_);
}

// ---------------------------------------------------------------------------
// GEMM
// ---------------------------------------------------------------------------
struct OzArgs {
  const unsigned char *pa, *pb;   // packed operands
  size_t pa_batch, pb_batch;
  const int *ea, *eb;             // row exponents
  int rows, cols, tb, K, nks, nsplit, steps;   // tb: column tiles; steps: stages per split
  // output element (i, j): out[b * s_batch + split * s_split + i * s_row + j * s_col]
  double2 *out;
  size_t s_batch, s_split;
  long s_row, s_col;
  int accum;
  // the operands themselves, for rows and columns that are not finite
  const double2 *A, *B;
  long a_row, a_k, b_row, b_k;
  size_t a_batch, b_batch;
  int conj_a, conj_b;
};

// (hi 2^SH + lo) 2^n to nearest, ties to even, in integer arithmetic: on the FP64 pipe the
// conversions and scalings of one 128 x 32 tile took 19 us, the MMAs of 16 k take 1.2 us.
template <int SH>
__device__ __forceinline__ double oz_value(long long hi, long long lo, int n);

template <int SH>
__device__ __forceinline__ double oz_value(long long hi, long long lo, int n) {
  uint64_t L = (uint64_t)hi << SH;
  long long H = hi >> (64 - SH);
  const uint64_t L2 = L + (uint64_t)lo;
  H += (lo >> 63) + (L2 < L ? 1 : 0);
  L = L2;
  const bool neg = H < 0;
  if (neg) {
    L = 0 - L;
    H = ~H + (L == 0 ? 1 : 0);
  }
  if ((H | (long long)L) == 0) return 0.0;
  // top: the 64 bits from the leading one down, worth 2^(e - 63); rest: anything below
  int e;
  uint64_t top, rest;
  if (H != 0) {
    const int z = __clzll(H);
    top = z ? ((uint64_t)H << z) | (L >> (64 - z)) : (uint64_t)H;
    rest = L << z;
    e = 127 - z;
  } else {
    const int z = __clzll((long long)L);
    top = L << z;
    rest = 0;
    e = 63 - z;
  }
  const int be = e + n + 1023;
  if (be <= 0 || be >= 2046) {   // subnormal, underflow or overflow
    const double v = scale2((double)top * 5.42101086242752217e-20, 0);   // top 2^-64
    const int m = e + n + 1;
    const double r = scale2(scale2(v, m / 2), m - m / 2);
    return neg ? -r : r;
  }
  uint64_t u = ((uint64_t)be << 52) + ((top >> 11) & 0xFFFFFFFFFFFFFull);
  const uint64_t low = top & 0x7ff;
  u += (low > 0x400 || (low == 0x400 && (rest || (u & 1)))) ? 1 : 0;
  return __longlong_as_double((long long)(neg ? u | 0x8000000000000000ull : u));
}

// The FP64 sum of one output over k0 .. k1 - 1 (operands with infinities or NaNs).
__device__ __noinline__ double2 oz_plain(const OzArgs &g, int bt, int i, int j, int k0, int k1) {
  const double2 *a = g.A + bt * g.a_batch + i * g.a_row, *b = g.B + bt * g.b_batch + j * g.b_row;
  double2 s = make_double2(0.0, 0.0);
  for (int k = k0; k < k1; ++k) {
    double2 x = a[k * g.a_k], y = b[k * g.b_k];
    if (g.conj_a) x.y = -x.y;
    if (g.conj_b) y.y = -y.y;
    s.x += x.x * y.x - x.y * y.y;
    s.y += x.x * y.y + x.y * y.x;
  }
  return s;
}

template <int S>
__global__ void __launch_bounds__(kOzThreads, 1) k_oz_gemm(OzArgs g) {
  using P = Oz<S>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t fa[P::kARing], ea[P::kARing], fb[P::kBRing], eb[P::kBRing], accf, acce;
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // column tiles fastest: CTAs that run together share their rows' operand in L2
  const int rt = blockIdx.x / g.tb, ct = blockIdx.x - rt * g.tb;
  const int bt = blockIdx.y / g.nsplit, sp = blockIdx.y - bt * g.nsplit;
  const int s0 = sp * g.steps, s1 = min(g.nks, s0 + g.steps);
  const int nst = max(0, s1 - s0);
  const int nblk = (nst + kDrain - 1) / kDrain;
  if (tid == 0) {
    for (int i = 0; i < P::kARing; ++i) {
      bar_init(&fa[i], 1);
      bar_init(&ea[i], 1);
    }
    for (int i = 0; i < P::kBRing; ++i) {
      bar_init(&fb[i], 1);
      bar_init(&eb[i], 1);
    }
    bar_init(&accf, 1);
    bar_init(&acce, kEpiWarps);
  }
  if (warp == 0) tmem_alloc(&tslot, 512);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  const uint32_t sa = smem_addr(smem), sb = sa + P::kARing * P::kAItem;
  bool ok = true;

  if (warp == kEpiWarps) {
    if (lane == 0) {   // copies
      const unsigned char *pa = g.pa + bt * g.pa_batch + ((size_t)rt * g.nks + s0) * P::kABytes;
      const unsigned char *pb = g.pb + bt * g.pb_batch + ((size_t)ct * g.nks + s0) * P::kBBytes;
      // a tile with fewer rows copies only their core matrices, slice by slice
      const int rows8 = (min(kRowsA, g.rows - rt * kRowsA) + 7) & ~7;
      constexpr uint32_t kSlice = kRowsA * kStep * 2;
      int na = 0, nb = 0;   // items under way
      for (int a = 0; a < 2 * nst && ok; ++a) {
        const int s = a >> 1;
        if (!(a & 1)) {
          const int j = s % P::kBRing;
          if (s >= P::kBRing) ok = bar_wait<kOzWait>(&eb[j], (s / P::kBRing - 1) & 1);
          if (!ok) break;
          bar_expect(&fb[j], P::kBBytes);
          bulk_copy(sb + j * P::kBBytes, pb + (size_t)s * P::kBBytes, P::kBBytes, &fb[j]);
          nb = s + 1;
        }
        const int j = a % P::kARing;
        if (a >= P::kARing) ok = bar_wait<kOzWait>(&ea[j], (a / P::kARing - 1) & 1);
        if (!ok) break;
        const uint32_t dst = sa + j * P::kAItem;
        const unsigned char *src = pa + (size_t)a * P::kAItem;
        if (rows8 == kRowsA) {
          bar_expect(&fa[j], P::kAItem);
          bulk_copy(dst, src, P::kAItem, &fa[j]);
        } else {
          bar_expect(&fa[j], S * rows8 * kStep * 2);
          for (int i = 0; i < S; ++i) bulk_copy(dst + i * kSlice, src + i * kSlice, rows8 * kStep * 2, &fa[j]);
        }
        na = a + 1;
      }
      // nothing may still be landing in shared memory when the CTA ends
      for (int a = max(0, na - P::kARing); a < na; ++a) ok = bar_wait<kOzWait>(&fa[a % P::kARing], (a / P::kARing) & 1) && ok;
      for (int s = max(0, nb - P::kBRing); s < nb; ++s) ok = bar_wait<kOzWait>(&fb[s % P::kBRing], (s / P::kBRing) & 1) && ok;
      if (!ok) atomicOr(&g_oz_error, 1u);
    }
  } else if (warp == kEpiWarps + 1) {
    // MMAs
    const bool lead = elect_one();
    const uint32_t a_lo = desc_lo(sa), b_lo = desc_lo(sb);
    int ja = 0, jb = 0;
    uint32_t pa = 0, pb = 0;   // phases of the rings
    bool issued = false;
    for (int s = 0; s < nst && ok; ++s) {
      const int blk = s / kDrain;
      const bool first = s % kDrain == 0;
      if (first && blk > 0) ok = bar_wait<kOzWait>(&acce, (blk - 1) & 1);   // the accumulators have been read
      if (ok) ok = bar_wait<kOzWait>(&fb[jb], pb);
      const uint32_t b0 = b_lo + jb * (P::kBBytes >> 4);
#pragma unroll
      for (int ra = 0; ra < 2; ++ra) {   // part of A
        if (ok) ok = bar_wait<kOzWait>(&fa[ja], pa);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        issued = true;
        if (lead) {
          const uint32_t a0 = a_lo + ja * (P::kAItem >> 4);
#pragma unroll
          for (int rb = 0; rb < 2; ++rb) {   // part of B; re: rr, ii; im: ri, ir
            const uint32_t d = tmem + ((ra ^ rb) ? 256 : 0), bd = b0 + ((rb * S * kRowsB * kStep * 2) >> 4);
#pragma unroll
            for (int i = 0; i < S; ++i)
              mma_f16(d + 32 * i, a0 + ((i * kRowsA * kStep * 2) >> 4), bd, idesc_f16(32 * (S - i), ra && rb),
                      !(first && ra == 0 && i == 0));
          }
          mma_commit(&ea[ja]);
          if (ra == 1) {
            mma_commit(&eb[jb]);
            if (s % kDrain == kDrain - 1 || s == nst - 1) mma_commit(&accf);
          }
        }
        __syncwarp();
        if (++ja == P::kARing) {
          ja = 0;
          pa ^= 1;
        }
      }
      if (!ok) break;
      if (++jb == P::kBRing) {
        jb = 0;
        pb ^= 1;
      }
    }
    if (!ok) {   // every MMA issued has to be done before tensor memory is given back
      if (lead) atomicOr(&g_oz_error, 1u);
      if (issued) {
        if (lead) mma_commit(&accf);
        __syncwarp();
        bar_wait<kOzWait>(&accf, 0);
        bar_wait<kOzWait>(&accf, 1);
      }
    }
  } else {
    // epilogue: warp w reads tensor-memory lanes 32 (w % 4) .. and columns kEpiCols (w / 4) .. of
    // each level
    const int q = warp & 3, c0 = kEpiCols * (warp >> 2);
    long long hi[2][kEpiCols], lo[2][kEpiCols];   // [re, im]
#pragma unroll
    for (int c = 0; c < kEpiCols; ++c) hi[0][c] = hi[1][c] = lo[0][c] = lo[1][c] = 0;
    const uint32_t base = tmem + ((uint32_t)(32 * q) << 16) + c0;
    for (int blk = 0; blk < nblk && ok; ++blk) {
      ok = bar_wait<kOzWait>(&accf, blk & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int l = 0; l < S; ++l) {
        uint32_t v[2][kEpiCols];
        TMEM_LD8(base + 32 * l, v[0]);
        TMEM_LD8(base + 256 + 32 * l, v[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        const int w = l < 4 ? 1 << (8 * (3 - l)) : 1 << (8 * (S - 1 - l));
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int c = 0; c < kEpiCols; ++c) {
            const long long x = (long long)__float2int_rn(__uint_as_float(v[p][c])) * w;
            if (l < 4) hi[p][c] += x;
            else lo[p][c] += x;
          }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&acce);
    }
    if (!ok && lane == 0) atomicOr(&g_oz_error, 1u);
    const int row = rt * kRowsA + 32 * q + lane;
    if (ok && row < g.rows) {
      const int em = g.ea[(size_t)bt * g.rows + row];
      double2 *o = g.out + bt * g.s_batch + sp * g.s_split + row * g.s_row;
      auto put = [&](int col, double2 v) {
        double2 *p = o + col * g.s_col;
        if (g.accum) {
          const double2 w = *p;
          v.x += w.x;
          v.y += w.y;
        }
        *p = v;
      };
      unsigned plain = 0;   // columns left to the FP64 sum
#pragma unroll
      for (int c = 0; c < kEpiCols; ++c) {
        const int col = ct * kRowsB + c0 + c;
        if (col >= g.cols) break;
        const int en = g.eb[(size_t)bt * g.cols + col];
        if (em == 0x7ff || en == 0x7ff) {
          plain |= 1u << c;
          continue;
        }
        // q_a q_b = 256^(S - 1) (hi 256^(S - 4) + lo), x = q 2^(E - bits), E = field - 1022
        const int n = 8 * (S - 1) + max(em, 1) + max(en, 1) - 2 * 1022 - 2 * P::kBits;
        put(col, make_double2(oz_value<8 * (S - 4)>(hi[0][c], lo[0][c], n), oz_value<8 * (S - 4)>(hi[1][c], lo[1][c], n)));
      }
      for (; plain; plain &= plain - 1) {
        const int col = ct * kRowsB + c0 + __ffs(plain) - 1;
        put(col, oz_plain(g, bt, row, col, s0 * kStep, min(g.K, s1 * kStep)));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 512);
}

// C[i][j] (+)= sum_s part[s][j][i] in split order; part is column-major (rows fastest)
__global__ void __launch_bounds__(256)
k_oz_splits(const double2 *__restrict__ part, int nsplit, int rows, int cols, size_t part_batch, double2 *__restrict__ C,
            long s_row, long s_col, size_t s_batch, int accum) {
  const size_t n = (size_t)rows * cols;
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  // threads walk C along its contiguous index
  const int i = s_row == 1 ? (int)(t % rows) : (int)(t / cols), j = s_row == 1 ? (int)(t / rows) : (int)(t % cols);
  const double2 *p = part + blockIdx.y * part_batch + (size_t)j * rows + i;
  double2 s = p[0];
  for (int z = 1; z < nsplit; ++z) {
    const double2 v = p[(size_t)z * n];
    s.x += v.x;
    s.y += v.y;
  }
  double2 *c = C + blockIdx.y * s_batch + i * s_row + j * s_col;
  if (accum) {
    s.x += c->x;
    s.y += c->y;
  }
  *c = s;
}

// ---------------------------------------------------------------------------
// Small products in plain FP64, one launch
// ---------------------------------------------------------------------------
struct SmallArgs {
  OzMat A, B;
  double2 *C;
  long s_row, s_col;
  size_t s_batch;
  int M, N, K, accum;
};

__device__ __forceinline__ void cfma(double2 &s, double2 x, double2 y) {
  s.x += x.x * y.x - x.y * y.y;
  s.y += x.x * y.y + x.y * y.x;
}

__device__ __forceinline__ void small_put(const SmallArgs &g, int b, int i, int j, double2 v) {
  double2 *c = g.C + b * g.s_batch + i * g.s_row + j * g.s_col;
  if (g.accum) {
    v.x += c->x;
    v.y += c->y;
  }
  *c = v;
}

// long K: a CTA sums 2 x 2 outputs over one of nsplit ranges of K
__global__ void __launch_bounds__(128) k_small_dot(SmallArgs g, int nsplit, double2 *__restrict__ part) {
  const int j0 = 2 * blockIdx.x, i0 = 2 * blockIdx.y, b = blockIdx.z / nsplit, sp = blockIdx.z % nsplit;
  const int per = (g.K + nsplit - 1) / nsplit, k0 = sp * per, k1 = min(g.K, k0 + per);
  const double2 *a = (const double2 *)g.A.p + b * g.A.s_batch, *x = (const double2 *)g.B.p + b * g.B.s_batch;
  const double2 *ar[2], *xr[2];
  for (int r = 0; r < 2; ++r) {
    ar[r] = a + min(i0 + r, g.M - 1) * g.A.s_row;
    xr[r] = x + min(j0 + r, g.N - 1) * g.B.s_row;
  }
  double2 s[2][2];
  for (int r = 0; r < 2; ++r)
    for (int c = 0; c < 2; ++c) s[r][c] = make_double2(0.0, 0.0);
  const double ca = g.A.conj ? -1.0 : 1.0, cb = g.B.conj ? -1.0 : 1.0;
#pragma unroll 2
  for (int k = k0 + threadIdx.x; k < k1; k += 128) {
    double2 u[2], v[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      u[r] = ar[r][k * g.A.s_k];
      v[r] = xr[r][k * g.B.s_k];
      u[r].y *= ca;
      v[r].y *= cb;
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) cfma(s[r][c], u[r], v[c]);
  }
  __shared__ double red[4][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    double t = (q & 1) ? s[q >> 2][(q >> 1) & 1].y : s[q >> 2][(q >> 1) & 1].x;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) red[warp][q] = t;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const int i = i0 + (threadIdx.x >> 1), j = j0 + (threadIdx.x & 1), q = 2 * threadIdx.x;
    const double2 v = make_double2(red[0][q] + red[1][q] + red[2][q] + red[3][q],
                                   red[0][q + 1] + red[1][q + 1] + red[2][q + 1] + red[3][q + 1]);
    if (i < g.M && j < g.N) {
      if (nsplit > 1) part[((size_t)b * nsplit + sp) * g.M * g.N + (size_t)j * g.M + i] = v;
      else small_put(g, b, i, j, v);
    }
  }
}

// short K: a thread per output, lanes along the index C is contiguous in
__global__ void __launch_bounds__(128) k_small_outer(SmallArgs g, int j_fast) {
  const size_t n = (size_t)g.M * g.N;
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (t >= n) return;
  const int i = j_fast ? (int)(t / g.N) : (int)(t % g.M), j = j_fast ? (int)(t % g.N) : (int)(t / g.M);
  const double2 *a = (const double2 *)g.A.p + b * g.A.s_batch + i * g.A.s_row;
  const double2 *x = (const double2 *)g.B.p + b * g.B.s_batch + j * g.B.s_row;
  double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int k = 0; k < g.K; ++k) {
    double2 u = a[k * g.A.s_k], v = x[k * g.B.s_k];
    if (g.A.conj) u.y = -u.y;
    if (g.B.conj) v.y = -v.y;
    cfma(s, u, v);
  }
  small_put(g, b, i, j, s);
}

// CTAs of k_small_dot per output group so that the chip has about four per SM
int small_splits(int M, int N, int K, int batch) {
  const long groups = (long)((M + 1) / 2) * ((N + 1) / 2) * batch;
  return (int)std::max<long>(1, std::min<long>((K + 1023) / 1024, 4 * kSms / groups));
}
size_t small_bytes(int M, int N, int K, int batch) {
  if (M < 1 || N < 1 || K < 1 || batch < 1) return 0;
  const int ns = small_splits(M, N, K, batch);
  return ns > 1 ? (size_t)ns * M * N * batch * sizeof(double2) : 0;
}

// Estimated microseconds of the two forms (measured: plain FP64 16 us per 10^6 complex products
// beyond its launch; the digit slices 25 us for their small kernels, then 1.3 us per tile and 16 k
// over the SMs).
bool small_product(int M, int N, int K, int batch) {
  if (M < 1 || N < 1 || K < 1 || batch < 1) return true;
  const double work = (double)M * N * K * batch;
  if (work > 2e7) return false;
  auto tiles = [](int r, int c) { return (double)((r + kRowsA - 1) / kRowsA) * ((c + kRowsB - 1) / kRowsB); };
  const double t = std::min(tiles(M, N), tiles(N, M)) * batch * ((K + kStep - 1) / kStep);
  return 5.0 + 16e-6 * work < 25.0 + 1.3 * t / kSms;
}

addft_status small_run(int M, int N, int K, int batch, const OzMat &A, const OzMat &B, double2 *C, long s_row, long s_col,
                       size_t s_batch, bool accum, void *work, size_t bytes, cudaStream_t st) {
  const SmallArgs g = {A, B, C, s_row, s_col, s_batch, M, N, K, accum ? 1 : 0};
  const bool contig = A.s_k == 1 && B.s_k == 1;
  const size_t n = (size_t)M * N;
  if (K >= 64 && (contig || (double)M * N < 8192) && (M + 1) / 2 <= 65535) {
    int ns = small_splits(M, N, K, batch);
    if (!work || bytes < small_bytes(M, N, K, batch)) ns = 1;
    k_small_dot<<<dim3((N + 1) / 2, (M + 1) / 2, batch * ns), 128, 0, st>>>(g, ns, (double2 *)work);
    ADDFT_TRY(check_launch("k_small_dot"));
    if (ns == 1) return ADDFT_OK;
    k_oz_splits<<<dim3((unsigned)((n + 255) / 256), batch), 256, 0, st>>>((const double2 *)work, ns, M, N, n * ns, C, s_row,
                                                                         s_col, s_batch, accum ? 1 : 0);
    return check_launch("k_oz_splits");
  }
  k_small_outer<<<dim3((unsigned)((n + 127) / 128), batch), 128, 0, st>>>(g, s_col == 1 ? 1 : 0);
  return check_launch("k_small_outer");
}

addft_status oz_max(const OzMat &m, int rows, int K, int batch, int *ex, cudaStream_t st) {
  // enough blocks to stream the operand at memory rate
  if (m.s_k == 1) {
    const int rb = (rows + 7) / 8;
    const int want = std::max(1, std::min((K + 255) / 256, (8 * 152 + rb * batch - 1) / (rb * batch)));
    const int chunk = (K + want - 1) / want;
    k_oz_max<true><<<dim3(rb, (K + chunk - 1) / chunk, batch), 256, 0, st>>>(
        (const double2 *)m.p, m.s_row, m.s_k, m.s_batch, rows, K, chunk, ex);
  } else {
    const int rb = (rows + 255) / 256;
    const int want = std::max(1, std::min((K + 7) / 8, (8 * 152 + rb * batch - 1) / (rb * batch)));
    const int chunk = (K + want - 1) / want;
    k_oz_max<false><<<dim3(rb, (K + chunk - 1) / chunk, batch), 256, 0, st>>>(
        (const double2 *)m.p, m.s_row, m.s_k, m.s_batch, rows, K, chunk, ex);
  }
  return check_launch("k_oz_max");
}

template <int S, int R>
addft_status oz_pack(const OzMat &m, int rows, int K, int nks, int batch, const int *ex, unsigned char *out,
                     size_t out_batch, cudaStream_t st) {
  constexpr int KT = 2048 / R;
  k_oz_pack<S, R><<<dim3((nks * kStep + KT - 1) / KT, (rows + R - 1) / R, batch), 256, 0, st>>>(
      (const double2 *)m.p, m.s_row, m.s_k, m.s_batch, m.conj, rows, K, nks, ex, out, out_batch);
  return check_launch("k_oz_pack");
}

template <int S>
addft_status oz_run(int rows, int cols, int K, int batch, const OzMat &A, const OzMat &B, double2 *C, long s_row,
                    long s_col, size_t s_batch, bool accum, int max_split, void *work, size_t bytes, cudaStream_t st) {
  const OzLayout l = oz_layout(S, rows, cols, K, batch, max_split);
  ADDFT_REQUIRE(l.total <= bytes, ADDFT_INVALID_ARG, "oz_gemm: a piece of %d x %d x %d wants %zu B of %zu", rows, cols, K,
                l.total, bytes);
  char *w = (char *)work;
  int *ea = (int *)(w + l.o_ex), *eb = ea + (size_t)batch * rows;
  unsigned char *pa = (unsigned char *)w + l.o_pa, *pb = (unsigned char *)w + l.o_pb;
  if (l.nks <= kPrepSteps) {
    const PrepArgs a = {(const double2 *)A.p, A.s_row, A.s_k, A.s_batch, A.conj, rows, ea, pa, l.pa};
    const PrepArgs b = {(const double2 *)B.p, B.s_row, B.s_k, B.s_batch, B.conj, cols, eb, pb, l.pb};
    const int ca = (rows + kPrepA - 1) / kPrepA, cb = (cols + kPrepB - 1) / kPrepB;
    ADDFT_TRY(smem_optin(k_oz_prep<S>, prep_smem(l.nks)));
    k_oz_prep<S><<<dim3(ca + cb, batch), 256, prep_smem(l.nks), st>>>(a, b, ca, K, l.nks);
    ADDFT_TRY(check_launch("k_oz_prep"));
  } else {
    ADDFT_CUDA(cudaMemsetAsync(ea, 0, (size_t)batch * (rows + cols) * sizeof(int), st));
    ADDFT_TRY(oz_max(A, rows, K, batch, ea, st));
    ADDFT_TRY(oz_max(B, cols, K, batch, eb, st));
    ADDFT_TRY((oz_pack<S, kRowsA>(A, rows, K, l.nks, batch, ea, pa, l.pa, st)));
    ADDFT_TRY((oz_pack<S, kRowsB>(B, cols, K, l.nks, batch, eb, pb, l.pb, st)));
  }
  OzArgs g;
  g.pa = pa; g.pb = pb; g.pa_batch = l.pa; g.pb_batch = l.pb;
  g.ea = ea; g.eb = eb;
  g.rows = rows; g.cols = cols; g.tb = l.tb; g.K = K; g.nks = l.nks; g.nsplit = l.nsplit; g.steps = l.steps;
  double2 *part = (double2 *)(w + l.o_part);
  const size_t n = (size_t)rows * cols;
  if (l.nsplit > 1) {
    g.out = part; g.s_row = 1; g.s_col = rows; g.s_split = n; g.s_batch = n * l.nsplit; g.accum = 0;
  } else {
    g.out = C; g.s_row = s_row; g.s_col = s_col; g.s_split = 0; g.s_batch = s_batch; g.accum = accum ? 1 : 0;
  }
  g.A = (const double2 *)A.p; g.a_row = A.s_row; g.a_k = A.s_k; g.a_batch = A.s_batch; g.conj_a = A.conj;
  g.B = (const double2 *)B.p; g.b_row = B.s_row; g.b_k = B.s_k; g.b_batch = B.s_batch; g.conj_b = B.conj;
  ADDFT_TRY(smem_optin(k_oz_gemm<S>, Oz<S>::kSmem));
  k_oz_gemm<S><<<dim3(l.ta * l.tb, batch * l.nsplit), kOzThreads, Oz<S>::kSmem, st>>>(g);
  ADDFT_TRY(check_launch("k_oz_gemm"));
  if (l.nsplit > 1) {
    k_oz_splits<<<dim3((unsigned)((n + 255) / 256), batch), 256, 0, st>>>(part, l.nsplit, rows, cols, n * l.nsplit, C,
                                                                         s_row, s_col, s_batch, accum ? 1 : 0);
    ADDFT_TRY(check_launch("k_oz_splits"));
  }
  return ADDFT_OK;
}

// The 128-row side goes to the index that pads less, with 10 % in favour of the one C is
// contiguous along, whose stores are then coalesced.
bool oz_swap(int M, int N, bool m_contig, bool n_contig) {
  auto pad = [](int a, int b) {
    return (double)((a + kRowsA - 1) / kRowsA * kRowsA) * ((b + kRowsB - 1) / kRowsB * kRowsB);
  };
  return pad(N, M) * (n_contig ? 1.0 : 1.1) < pad(M, N) * (m_contig ? 1.0 : 1.1);
}

}  // namespace

size_t oz_work_bytes(int digits, int M, int N, int K, int batch) {
  if (small_product(M, N, K, batch)) return small_bytes(M, N, K, batch);
  const size_t need = std::max(oz_layout(digits, M, N, K, batch).total, oz_layout(digits, N, M, K, batch).total);
  return std::min(need, kOzScratchCap);
}

bool oz_fits(int digits, int M, int N, int K, int batch, const void *work, size_t bytes) {
  if (small_product(M, N, K, batch)) return true;
  OzPieces p;
  return work && ((uintptr_t)work & 255) == 0 && oz_pieces(digits, M, N, K, batch, bytes, p) &&
         oz_pieces(digits, N, M, K, batch, bytes, p);
}

addft_status oz_gemm(int digits, int M, int N, int K, int batch, const OzMat &A, const OzMat &B, void *C, long s_row,
                     long s_col, size_t s_batch, bool accum, void *work, size_t work_bytes, cudaStream_t st) {
  if (small_product(M, N, K, batch))
    return small_run(M, N, K, batch, A, B, (double2 *)C, s_row, s_col, s_batch, accum, work, work_bytes, st);
  const bool sw = oz_swap(M, N, s_row == 1, s_col == 1);
  const int r = sw ? N : M, c = sw ? M : N;
  const OzMat &ma = sw ? B : A, &mb = sw ? A : B;
  const long sr = sw ? s_col : s_row, sc = sw ? s_row : s_col;
  OzPieces p;
  ADDFT_REQUIRE(work && ((uintptr_t)work & 255) == 0 && oz_pieces(digits, r, c, K, batch, work_bytes, p),
                ADDFT_INVALID_ARG, "oz_gemm: work buffer of %zu B too small or not 256-byte aligned", work_bytes);
  auto at = [](const OzMat &m, int b, int row, int k) {
    OzMat o = m;
    o.p = (const double2 *)m.p + b * m.s_batch + row * m.s_row + k * m.s_k;
    return o;
  };
  return (addft_status)oz_each_piece(r, c, K, batch, p, [&](int b0, int r0, int c0, int k0, int nb, int nr, int nc, int nk) {
    const OzMat a = at(ma, b0, r0, k0), b = at(mb, b0, c0, k0);
    double2 *o = (double2 *)C + b0 * s_batch + r0 * sr + c0 * sc;
    return (int)(digits == 8 ? oz_run<8>(nr, nc, nk, nb, a, b, o, sr, sc, s_batch, accum || k0 > 0, p.nsplit, work, work_bytes, st)
                             : oz_run<7>(nr, nc, nk, nb, a, b, o, sr, sc, s_batch, accum || k0 > 0, p.nsplit, work, work_bytes, st));
  });
}

unsigned oz_status() {
  unsigned v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, g_oz_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(g_oz_error, &z, sizeof(z));
  return v;
}

}  // namespace addft
