// FP32 projector contractions of V_NL psi on the 5th-generation tensor cores
// (tcgen05.mma kind::tf32, accumulators in tensor memory), split-precision TF32:
// every product a b is formed as hi(a) hi(b) + hi(a) lo(b) + lo(a) hi(b) (becp: + lo(a) lo(b))
// with FP32 accumulation (hi = round-to-nearest TF32 of x, lo = TF32 of x - hi); 2e-7 to
// 6e-7 relative on random operands.
//
//   becp[k][p][b] = sum_G conj(proj[k][p][G]) psi[k][b][G]          (nonlocal_op.py:67-70)
//     D (128 x 2 NB) = P (128 x K) X^T: rows are hi and lo of 32 projectors and of the same
//     with each (re, im) pair replaced by (-im, re), columns hi and lo of NB bands; K runs
//     over (G, re/im).  Split-K over G across CTAs, deterministic partials.
//   out[k][b][G] (+)= sum_p beta[k][p][G] DB[k][p][b]                 (nonlocal_op.py:73-76)
//     D (128 x 128) = Bt (128 x K) Y^T: rows are 128 G of a tile, columns the real and
//     imaginary parts of 64 bands; K runs over (projector, re/im).
//
// Operands are written by the CTA's threads into shared memory in the canonical
// no-swizzle K-major layout (8-row x 16-byte core matrices; in the one-chunk apply
// LBO = 128 B between the two core matrices of one K = 8 step, SBO = 256 B between 8-row
// groups), since the hi/lo split has to happen in registers on the way.  One thread issues the MMAs; a
// commit to an mbarrier tells the producers when the operand buffer is free again, and
// the next step's global loads are in flight (in registers) while the MMAs run.
// Every mbarrier wait has an iteration limit: on expiry the kernel records an error
// (read with addft_tc05_status), waits (bounded) for its own MMAs, frees its tensor
// memory and returns.
#include <algorithm>

#include "common.cuh"
#include "mma16.cuh"
#include "ozgemm.cuh"

namespace addft {

namespace {

__device__ unsigned g_tc05_error = 0;   // bit 0: an mbarrier wait ran out

constexpr int kWaitLimit = 1 << 24;

// tcgen05 shared-memory matrix descriptor: start address, LBO, SBO (bytes >> 4), the
// fixed 0b001 at bits 46-48, base offset 0, no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

// instruction descriptor, kind::tf32: F32 accumulator, TF32 A and B, both K-major, N and M.
__host__ __device__ constexpr uint32_t idesc_tf32(int M, int N) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// the same from the descriptors' lower words (start address, LBO), SBO = 128 B
__device__ __forceinline__ void mma_tf32_lo(uint32_t dtmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  constexpr uint32_t hi = (128u >> 4) | (1u << 14);
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tmov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
      "setp.ne.b32 p, %5, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, p;\n\t}" ::"r"(dtmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(hi), "r"(acc)
      : "memory");
}

__device__ __forceinline__ uint32_t tf32_rna(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void split4(const float (&x)[4], uint4 &hi, uint4 &lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    h[i] = tf32_rna(x[i]);
    l[i] = tf32_rna(x[i] - __uint_as_float(h[i]));
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// byte offset of K-chunk kc (4 floats) of row r in a canonical tile of R rows, K = 8 per slice
__device__ __forceinline__ uint32_t coff(int R, int r, int k4) {
  const int slice = k4 >> 1, kc = k4 & 1;
  return (uint32_t)(slice * (R / 8) * 256 + (r >> 3) * 256 + kc * 128 + (r & 7) * 16);
}

#define TC05_LD32(taddr, r)                                                                                      \
  asm volatile(                                                                                                  \
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18," \
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"                                             \
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),          \
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),    \
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),  \
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])   \
      : "r"(taddr))

// ---------------------------------------------------------------------------
// becp
// ---------------------------------------------------------------------------
// A tile is 32 projectors x 16 RB bands over one chunk of G.  The M = 128 operand holds each
// projector four times, as rows hi, lo, i hi, i lo (i x = (-Im x, Re x)), the N operand each band
// twice, hi and lo; K is (G, re/im).  One MMA then gives every product of the split, lo lo included,
// in accumulators of its own, and an element is split, exchanged and stored once per tile.
//   Tensor memory adds with truncation, so an error grows with the number of MMAs in an accumulator (8:
// 1.9e-7 rms of random becp, 16: 3.4e-7, 235: 4.5e-6).  Two sets of accumulators take turns, one
// stage of 32 G (8 MMAs) each, and are added to FP32 sums in registers.
//   A warp reads 256 contiguous bytes of a row; a lane splits its G and writes the halves of the
// 16-byte chunks it shares with its neighbour.  The chunks of a row lie rows + 1 core-matrix rows
// apart, so the 16 lanes of a shared-memory phase write 8 different bank groups.  16 warps convert and drain, one issues the MMAs; bounded waits.
//   Bound by shared memory (the MMAs read A, 4 KB, and B per K = 8 step at 90 to 110 B per cycle, beside the
// operands' stores) with few projectors by the loads' latency: 168 bands x 256 projectors x 23,847 G 234
// us (mma.sync) -> 84, 64 x 32 x 142,609 60 -> 38 (23 with the loads taken out).  Keeping 4 stages of
// loads in flight, in registers or with cp.async, was no quicker (43, 39 us), nor were tiles of 64 projectors
// with one set of accumulators (85 us with its sums, and 6e-6 rms).
constexpr int kBWarps = 16;
constexpr int kBThreads = 32 * kBWarps + 32;
template <int RB>
struct BT {
  static constexpr int NB = 16 * RB, N = 2 * NB;
  static constexpr uint32_t kChunkA = 128 * 16 + 16, kChunkB = N * 16 + 16;   // bytes between 4-float K chunks
  static constexpr uint32_t kA = 16 * kChunkA, kB = 16 * kChunkB, kStage = kA + kB;
  static constexpr uint32_t kCols = 2 * N <= 64 ? 64 : 2 * N <= 128 ? 128 : 2 * N <= 256 ? 256 : 512;
  static constexpr int kPitch = NB + 1;
  static constexpr size_t kRed = (size_t)128 * kPitch * 4;
  static constexpr size_t kSmem = 2 * kStage + 128;
  static constexpr int kPre = RB <= 4 ? 2 : 1;          // stages of loads in registers
  static constexpr int kQ = (NB / 8 + 3) / 4;           // 8-band groups per draining warp
  static_assert(2 * N <= 512 && kSmem + 1024 <= 227 * 1024 && kRed <= kSmem, "tile");
};
}  // namespace

template <int RB>
__global__ void __launch_bounds__(kBThreads, 1)
k_becp_tc05(const float2 *__restrict__ proj, const float2 *__restrict__ psi, int nb, int nG, int nproj, int nsplit,
            float2 *__restrict__ out) {
  using T = BT<RB>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[2], accf[2], acce[2];   // operands written, MMAs done, sums taken
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p0 = blockIdx.y * 32, b0 = blockIdx.x * T::NB;
  const int nkz = gridDim.z / nsplit;
  const int k = blockIdx.z / nsplit, sp = blockIdx.z - k * nsplit;
  // stages sp, sp + nsplit, ...: CTAs that run together read neighbouring G
  const int nst = ((nG + 31) / 32 - sp + nsplit - 1) / nsplit;
  if (tid == 0)
    for (int i = 0; i < 2; ++i) {
      bar_init(&full[i], kBWarps);
      bar_init(&accf[i], 1);
      bar_init(&acce[i], kBWarps);
    }
  if (warp == kBWarps) tmem_alloc(&tslot, T::kCols);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot, sbase = smem_addr(smem);
  bool ok = true;
  float sum[T::kQ][8];
#pragma unroll
  for (int c = 0; c < T::kQ; ++c)
#pragma unroll
    for (int q = 0; q < 8; ++q) sum[c][q] = 0.f;

  if (warp == kBWarps) {
    const bool lead = elect_one();
    constexpr uint32_t idesc = idesc_tf32(128, T::N);
    const uint32_t a_lo = (sbase >> 4) | ((T::kChunkA >> 4) << 16);
    const uint32_t b_lo = ((sbase + T::kA) >> 4) | ((T::kChunkB >> 4) << 16);
    int s = 0;
    for (; s < nst; ++s) {
      const int j = s & 1;
      ok = bar_wait<kWaitLimit>(&full[j], (s >> 1) & 1);
      if (ok && s >= 2) ok = bar_wait<kWaitLimit>(&acce[j], ((s >> 1) - 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (lead) {
        const uint32_t o = j * (T::kStage >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          mma_tf32_lo(tmem + j * T::N, a_lo + o + (2 * kk * T::kChunkA) / 16, b_lo + o + (2 * kk * T::kChunkB) / 16,
                      idesc, kk > 0);
        mma_commit(&accf[j]);
      }
      __syncwarp();
    }
    if (!ok) {   // every MMA issued has to be done before tensor memory is given back
      if (lead) atomicOr(&g_tc05_error, 1u);
      for (int t = max(0, s - 2); t < s; ++t) bar_wait<kWaitLimit>(&accf[t & 1], (t >> 1) & 1);
    }
  } else {
    constexpr int NR = 2 + RB;   // rows of this warp: projectors warp, warp + 16, bands warp, warp + 16, ...
    // rows past the end repeat the last one: they feed outputs that nobody stores
    const float2 *Pk = proj + (size_t)k * nproj * nG, *Xk = psi + (size_t)k * nb * nG;
    int row[NR];
#pragma unroll
    for (int i = 0; i < 2; ++i) row[i] = min(p0 + warp + 16 * i, nproj - 1);
#pragma unroll
    for (int i = 0; i < RB; ++i) row[2 + i] = min(b0 + warp + 16 * i, nb - 1);
    float2 v[T::kPre][NR];
    auto load = [&](int s, float2 (&x)[NR]) {
      // the last stage may be short: its lanes past the end read the last G and are cleared when written
      const int g = min(32 * (sp + s * nsplit) + lane, nG - 1);
#pragma unroll
      for (int i = 0; i < NR; ++i) x[i] = (i < 2 ? Pk : Xk)[(long)row[i] * nG + g];
    };
    const uint32_t wa = sbase + (lane >> 1) * T::kChunkA + (lane & 1) * 8 + warp * 16;
    const uint32_t wb = sbase + T::kA + (lane >> 1) * T::kChunkB + (lane & 1) * 8 + warp * 16;
    // accumulators: part warp % 4 of the rows, 8-band groups warp / 4, warp / 4 + 4, ...
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * (warp >> 2);
    auto drain = [&](int j) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < T::kQ; ++c)
        if (8 * (warp >> 2) + 32 * c < T::NB) {
          uint32_t h[8], l[8];
          TMEM_LD8(tq + j * T::N + 32 * c, h);
          TMEM_LD8(tq + j * T::N + T::NB + 32 * c, l);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int q = 0; q < 8; ++q) sum[c][q] += __uint_as_float(h[q]) + __uint_as_float(l[q]);
        }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&acce[j]);
    };
    auto stage = [&](int s, float2 (&x)[NR]) {
      const int j = s & 1;
      if (s >= 2) {   // MMAs of stage s - 2: its operands' room and its accumulators
        ok = bar_wait<kWaitLimit>(&accf[j], ((s >> 1) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return;
      }
      const uint32_t o = j * T::kStage;
      if (32 * (sp + s * nsplit) + lane >= nG) {
#pragma unroll
        for (int i = 0; i < NR; ++i) x[i] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const uint32_t hx = tf32_rna(x[i].x), hy = tf32_rna(x[i].y);
        const uint32_t lx = tf32_rna(x[i].x - __uint_as_float(hx)), ly = tf32_rna(x[i].y - __uint_as_float(hy));
        if (i < 2) {   // rows hi, lo, i hi, i lo of 32 each
          const uint32_t d = wa + o + i * 256;
          sts64(d, hx, hy);
          sts64(d + 512, lx, ly);
          sts64(d + 1024, hy ^ 0x80000000u, hx);
          sts64(d + 1536, ly ^ 0x80000000u, lx);
        } else {
          const uint32_t d = wb + o + (i - 2) * 256;
          sts64(d, hx, hy);
          sts64(d + T::NB * 16, lx, ly);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&full[j]);
      if (s + T::kPre < nst) load(s + T::kPre, x);
      if (s >= 2) drain(j);
    };
#pragma unroll
    for (int i = 0; i < T::kPre; ++i)
      if (i < nst) load(i, v[i]);
    for (int s = 0; s < nst && ok; s += T::kPre)
#pragma unroll
      for (int i = 0; i < T::kPre; ++i)
        if (ok && s + i < nst) stage(s + i, v[i]);
    for (int s = max(0, nst - 2); s < nst && ok; ++s) {
      ok = bar_wait<kWaitLimit>(&accf[s & 1], (s >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) drain(s & 1);
    }
    if (!ok && lane == 0) atomicOr(&g_tc05_error, 1u);
  }
  ok = __syncthreads_and(ok) != 0;
  float *red = reinterpret_cast<float *>(smem);   // [part][projector][band]
  if (ok && warp < kBWarps) {
    float *r = red + (32 * (warp & 3) + lane) * T::kPitch + 8 * (warp >> 2);
#pragma unroll
    for (int c = 0; c < T::kQ; ++c)
      if (8 * (warp >> 2) + 32 * c < T::NB)
#pragma unroll
        for (int q = 0; q < 8; ++q) r[32 * c + q] = sum[c][q];
  }
  __syncthreads();
  if (warp == kBWarps) {
    tmem_free(tmem, T::kCols);
    return;
  }
  if (!ok) return;
  float2 *dst = out + ((size_t)sp * nkz + k) * nproj * nb;
  for (int e = tid; e < 32 * T::NB; e += 32 * kBWarps) {
    const int p = e / T::NB, b = e - p * T::NB;
    if (p0 + p >= nproj || b0 + b >= nb) continue;
    const float *r = red + p * T::kPitch + b;
    constexpr int q = 32 * T::kPitch;
    dst[(size_t)(p0 + p) * nb + b0 + b] = make_float2(r[0] + r[q], r[2 * q] + r[3 * q]);
  }
}

// Tile of a problem: 32 projectors, equal tiles of up to kMost bands.
void becp_tc05_tile(int nb, int *pt, int *bt) {
  constexpr int kMost = 96;
  const int n = (nb + kMost - 1) / kMost;
  *pt = 32;
  *bt = ((nb + n - 1) / n + 15) / 16 * 16;
}

template <int RB>
static addft_status becp_go(dim3 grid, int nb, int nG, int nproj, int nsplit, const float2 *proj, const float2 *psi,
                            float2 *out, cudaStream_t st) {
  ADDFT_TRY(smem_optin(k_becp_tc05<RB>, BT<RB>::kSmem));
  k_becp_tc05<RB><<<grid, kBThreads, BT<RB>::kSmem, st>>>(proj, psi, nb, nG, nproj, nsplit, out);
  return check_launch("k_becp_tc05");
}

addft_status launch_becp_tc05(int nk, int nb, int nG, int nproj, int nsplit, const float2 *proj, const float2 *psi,
                              float2 *out, cudaStream_t st) {
  int pt, bt;
  becp_tc05_tile(nb, &pt, &bt);
  const dim3 grid((nb + bt - 1) / bt, (nproj + pt - 1) / pt, nk * nsplit);
  switch (bt / 16) {
#define BECP_CASE(rb) \
  case rb: return becp_go<rb>(grid, nb, nG, nproj, nsplit, proj, psi, out, st);
    BECP_CASE(1) BECP_CASE(2) BECP_CASE(3) BECP_CASE(4) BECP_CASE(5) BECP_CASE(6)
#undef BECP_CASE
  }
  return ADDFT_INVALID_ARG;
}

// ---------------------------------------------------------------------------
// V_NL apply: out[k][b][G] (+)= sum_j A[k][j][G] X[k][j][b]   (A = beta, X = D becp)
// ---------------------------------------------------------------------------
namespace {
constexpr int kAG = 128;   // G per tile (M)
constexpr int kAB = 64;    // bands per tile (N = 128: real parts, then imaginary parts)
constexpr int kAJ = 32;    // projectors per K chunk (K = 64 floats = 8 MMA steps)
constexpr int kATile = 128 * 2 * kAJ * 4;   // bytes of one 128-row operand tile: 32 KB
constexpr size_t kApplySmem = 4 * (size_t)kATile + 1024;   // A hi, A lo, B hi, B lo
}  // namespace

template <bool ACCUM>
__global__ void __launch_bounds__(256, 1)
k_apply_tc05(const float2 *__restrict__ X, int xs_j, int xs_i, size_t xs_k, const float2 *__restrict__ A,
             size_t as_k, int nj, int ni, int nG, float2 *__restrict__ out, size_t os_k) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b0 = blockIdx.y * kAB, k = blockIdx.z;
  const float2 *Ak = A + (size_t)k * as_k;
  const float2 *Xk = X + (size_t)k * xs_k;
  float2 *ok_ = out + (size_t)k * os_k;
  if (tid == 0) bar_init(&bar);
  if (warp == 0) tmem_alloc(&tslot, 128);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  const uint32_t idesc = idesc_tf32(128, 128);
  const uint32_t ahi = smem_addr(smem), alo = ahi + kATile, bhi = alo + kATile, blo = bhi + kATile;
  const int nchunk = (nj + kAJ - 1) / kAJ;
  const int ntile = (nG + kAG - 1) / kAG;
  // operand rows: row r = tid % 128 of A (G) and B (band part), projector half ph = tid / 128
  const int r = tid & 127, ph = tid >> 7;
  constexpr int kH = kAJ / 2;   // projectors per thread and chunk
  // B row r: band b0 + (r & 63); r < 64: (Re X, -Im X) per projector, r >= 64: (Im X, Re X)
  const int bn = b0 + (r & 63);
  const bool bpart = r >= 64, bok = bn < ni;
  auto build_b = [&](int c) {
    float2 xv[kH];
#pragma unroll
    for (int jj = 0; jj < kH; ++jj) {
      const int j = c * kAJ + ph * kH + jj;
      xv[jj] = (bok && j < nj) ? Xk[(size_t)j * xs_j + (size_t)bn * xs_i] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < kH / 2; ++q) {   // two projectors per 4-float K chunk
      float v[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float2 x = xv[2 * q + h];
        v[2 * h] = bpart ? x.y : x.x;
        v[2 * h + 1] = bpart ? x.x : -x.y;
      }
      uint4 hi, lo;
      split4(v, hi, lo);
      sts128(bhi + coff(128, r, ph * (kH / 2) + q), hi);
      sts128(blo + coff(128, r, ph * (kH / 2) + q), lo);
    }
  };
  float2 av[kH];   // this thread's A values of the next (tile, chunk), loaded ahead
  auto load_a = [&](int t, int c) {
    const int g = t * kAG + r;
#pragma unroll
    for (int jj = 0; jj < kH; ++jj) {
      const int j = c * kAJ + ph * kH + jj;
      av[jj] = (g < nG && j < nj) ? Ak[(size_t)j * nG + g] : make_float2(0.f, 0.f);
    }
  };
  bool ok = true;
  int ncommit = 0;
  if (nchunk == 1) build_b(0);
  if (blockIdx.x < ntile) load_a(blockIdx.x, 0);
  // epilogue mapping: warp w reads D lanes 32 (w % 4) .. (rows = G), band half bh = w / 4
  const int bh = warp >> 2;
  for (int t = blockIdx.x; t < ntile && ok; t += gridDim.x) {
    for (int c = 0; c < nchunk && ok; ++c) {
      if (ncommit > 0) ok = __syncthreads_and(bar_wait<kWaitLimit>(&bar, (ncommit - 1) & 1)) != 0;   // operands free
      if (!ok) break;
      if (nchunk > 1) build_b(c);
#pragma unroll
      for (int q = 0; q < kH / 2; ++q) {
        float v[4] = {av[2 * q].x, av[2 * q].y, av[2 * q + 1].x, av[2 * q + 1].y};
        uint4 hi, lo;
        split4(v, hi, lo);
        sts128(ahi + coff(128, r, ph * (kH / 2) + q), hi);
        sts128(alo + coff(128, r, ph * (kH / 2) + q), lo);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int kk = 0; kk < kAJ * 2 / 8; ++kk) {
          const uint64_t ah = sdesc(ahi + kk * 16 * 256, 128, 256), al = sdesc(alo + kk * 16 * 256, 128, 256);
          const uint64_t bh_ = sdesc(bhi + kk * 16 * 256, 128, 256), bl = sdesc(blo + kk * 16 * 256, 128, 256);
          mma_tf32(tmem, ah, bh_, idesc, (c > 0 || kk > 0) ? 1u : 0u);
          mma_tf32(tmem, ah, bl, idesc, 1u);
          mma_tf32(tmem, al, bh_, idesc, 1u);
        }
        mma_commit(&bar);
      }
      ++ncommit;
      // next operands in flight while the MMAs run
      if (c + 1 < nchunk) load_a(t, c + 1);
      else if (t + (int)gridDim.x < ntile) load_a(t + gridDim.x, 0);
    }
    if (!ok) break;
    const int row = t * kAG + 32 * (warp & 3) + lane;   // D row (G) of this thread
    float2 w[32];   // old values, read before the accumulator is waited for
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int b = b0 + 32 * bh + j;
      w[j] = (ACCUM && b < ni && row < nG) ? ok_[(size_t)b * nG + row] : make_float2(0.f, 0.f);
    }
    ok = __syncthreads_and(bar_wait<kWaitLimit>(&bar, (ncommit - 1) & 1)) != 0;   // accumulator complete
    if (!ok) break;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t re[32], im[32];
    TC05_LD32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * bh), re);
    TC05_LD32(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(64 + 32 * bh), im);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (row < nG) {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int b = b0 + 32 * bh + j;
        if (b < ni)
          ok_[(size_t)b * nG + row] = make_float2(__uint_as_float(re[j]) + w[j].x, __uint_as_float(im[j]) + w[j].y);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  if (!ok) {
    if (tid == 0 && ncommit > 0) mma_commit(&bar);   // one more commit tracks every MMA issued
    bar_wait<kWaitLimit>(&bar, ncommit & 1);
    if (lane == 0) atomicOr(&g_tc05_error, 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 128);
}

// ---------------------------------------------------------------------------
// apply with more than one chunk of projectors
// ---------------------------------------------------------------------------
// k_deep_pack writes X, split and in operand layout, to scratch once.  A unit is 128 G x NB bands; K
// runs over all projectors in stages of 16.  16 warps split A (a lane holds one G and two
// projectors: coalesced loads, one 16-byte chunk, 8 lanes fill a core matrix), one lane copies X's
// stages, one warp issues the MMAs (three of N = 2 NB per K = 8 step).  Two sets of accumulators take
// turns, two stages each, and are added to FP32 sums in registers (tensor memory adds with
// truncation); a unit's sums are added to `out` while the next unit's first stages run.  Bounded
// waits.  Bound by shared memory (the MMAs' operands and the stores of them): 168 bands x 256
// projectors x 23,847 G 152 -> 68 us; splitting X in every tile instead of once cost 140.
namespace {
constexpr int kDJ = 16;                                  // projectors per stage
template <int NB>
struct DT {
  static constexpr int N = 2 * NB, kG = NB / 32;         // columns (re, im), band groups of 32 lanes
  static constexpr uint32_t kChunkA = 128 * 16, kChunkB = N * 16, kA = kDJ / 2 * kChunkA, kB = kDJ / 2 * kChunkB;
  static constexpr uint32_t kStage = 2 * kA + 2 * kB;    // A hi, A lo, B hi, B lo
  static constexpr uint32_t kCols = 2 * N <= 128 ? 128 : 2 * N <= 256 ? 256 : 512;
  static constexpr size_t kSmem = 2 * kStage + 128;
};
}  // namespace

// X of (k, band tile, stage): B hi, then B lo; zeros past the last projector and band
template <int NB>
__global__ void k_deep_pack(const float2 *__restrict__ X, int xs_j, int xs_i, size_t xs_k, int nj, int ni, int nst,
                            int nbt, unsigned char *__restrict__ out) {
  using T = DT<NB>;
  const int b = threadIdx.x, q = blockIdx.x, bt = blockIdx.y, k = blockIdx.z;   // q: pair of projectors
  const float2 *Xk = X + (size_t)k * xs_k + (size_t)(bt * NB + b) * xs_i;
  float x[4];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 v = 2 * q + h < nj && bt * NB + b < ni ? Xk[(size_t)(2 * q + h) * xs_j] : make_float2(0.f, 0.f);
    x[2 * h] = v.x;
    x[2 * h + 1] = v.y;
  }
  uint4 hi, lo;
  split4(x, hi, lo);
  constexpr uint32_t m = 0x80000000u;
  const int s = q / (kDJ / 2), c = q - s * (kDJ / 2);
  unsigned char *o = out + (((size_t)k * nbt + bt) * nst + s) * (2 * T::kB) + c * T::kChunkB + b * 16;
  *(uint4 *)o = make_uint4(hi.x, hi.y ^ m, hi.z, hi.w ^ m);                     // re: (re, -im)
  *(uint4 *)(o + T::kB) = make_uint4(lo.x, lo.y ^ m, lo.z, lo.w ^ m);
  *(uint4 *)(o + NB * 16) = make_uint4(hi.y, hi.x, hi.w, hi.z);                 // im: (im, re)
  *(uint4 *)(o + NB * 16 + T::kB) = make_uint4(lo.y, lo.x, lo.w, lo.z);
}

template <int NB, bool ACCUM>
__global__ void __launch_bounds__(kBThreads + 32, 1)
k_apply_deep(const unsigned char *__restrict__ X, const float2 *__restrict__ A, size_t as_k, int nk, int nj, int ni, int nG, float2 *__restrict__ out, size_t os_k) {
  using T = DT<NB>;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[2], free_[2], accf[2], acce[2];
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntile = (nG + 127) / 128, nbt = (ni + NB - 1) / NB, units = ntile * nbt * nk;
  const int nst = (nj + kDJ - 1) / kDJ;
  if (tid == 0)
    for (int i = 0; i < 2; ++i) {
      bar_init(&full[i], kBWarps + 1);
      bar_init(&free_[i], 1);
      bar_init(&accf[i], 1);
      bar_init(&acce[i], kBWarps);
    }
  if (warp == kBWarps) tmem_alloc(&tslot, T::kCols);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot, sbase = smem_addr(smem);
  bool ok = true;

  if (warp == kBWarps) {
    const bool lead = elect_one();
    constexpr uint32_t idesc = idesc_tf32(128, T::N);
    const uint32_t a_lo = (sbase >> 4) | ((T::kChunkA >> 4) << 16);
    const uint32_t b_lo = ((sbase + 2 * T::kA) >> 4) | ((T::kChunkB >> 4) << 16);
    int it = 0, bl = 0;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x)
      for (int s = 0; s < nst && ok; ++s) {
        const int j = it & 1, set = bl & 1;
        const bool first = (s & 1) == 0, last = (s & 1) || s == nst - 1;
        ok = bar_wait<kWaitLimit>(&full[j], (it >> 1) & 1);
        if (ok && first && bl >= 2) ok = bar_wait<kWaitLimit>(&acce[set], ((bl >> 1) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (lead) {
          const uint32_t ah = a_lo + j * (T::kStage >> 4), al = ah + (T::kA >> 4);
          const uint32_t bh = b_lo + j * (T::kStage >> 4), bl_ = bh + (T::kB >> 4), d = tmem + set * T::N;
#pragma unroll
          for (int kk = 0; kk < kDJ / 4; ++kk) {
            const uint32_t oa = 2 * kk * T::kChunkA / 16, ob = 2 * kk * T::kChunkB / 16;
            mma_tf32_lo(d, ah + oa, bh + ob, idesc, !first || kk > 0);
            mma_tf32_lo(d, ah + oa, bl_ + ob, idesc, 1u);
            mma_tf32_lo(d, al + oa, bh + ob, idesc, 1u);
          }
          mma_commit(&free_[j]);
          if (last) mma_commit(&accf[set]);
        }
        __syncwarp();
        ++it;
        if (last) ++bl;
      }
    if (!ok) {   // every MMA issued has to be done before tensor memory is given back
      if (lead) atomicOr(&g_tc05_error, 1u);
      for (int t = max(0, it - 2); t < it; ++t) bar_wait<kWaitLimit>(&free_[t & 1], (t >> 1) & 1);
    }
  } else if (warp == kBWarps + 1) {
    if (lane == 0) {   // X
      int it = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const int bt = u % nbt, k = u / nbt / ntile;
        const unsigned char *src = X + ((size_t)k * nbt + bt) * nst * (2 * T::kB);
        for (int s = 0; s < nst && ok; ++s, ++it) {
          const int j = it & 1;
          if (it >= 2) ok = bar_wait<kWaitLimit>(&free_[j], ((it >> 1) - 1) & 1);
          if (!ok) break;
          bar_expect(&full[j], 2 * T::kB);
          bulk_copy(sbase + j * T::kStage + 2 * T::kA, src + (size_t)s * (2 * T::kB), 2 * T::kB, &full[j]);
        }
      }
      // nothing may still be landing in shared memory when the CTA ends
      for (int t = max(0, it - 2); t < it; ++t) ok = bar_wait<kWaitLimit>(&full[t & 1], (t >> 1) & 1) && ok;
      if (!ok) atomicOr(&g_tc05_error, 1u);
    }
  } else {
    // two projectors of this lane's G, two stages ahead; tasks: pair t / 4, G group t % 4 of t = warp, warp + 16
    float2 v0[2][2], v1[2][2];
    int lu = blockIdx.x, ls = 0;   // unit and stage of the next load
    const float2 *lp = nullptr;
    auto load = [&](float2 (&x)[2][2]) __attribute__((always_inline)) {
      if (lu >= units) return;
      if (ls == 0) {
        const int t = lu / nbt, k = t / ntile;
        lp = A + (size_t)k * as_k + min((t - k * ntile) * 128 + 32 * (warp & 3) + lane, nG - 1);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int jj = ls * kDJ + 2 * ((warp + 16 * i) >> 2);
#pragma unroll
        for (int h = 0; h < 2; ++h) x[i][h] = jj + h < nj ? lp[(size_t)(jj + h) * nG] : make_float2(0.f, 0.f);
      }
      if (++ls == nst) {
        ls = 0;
        lu += gridDim.x;
      }
    };
    auto put = [&](int j, const float2 (&y)[2][2]) __attribute__((always_inline)) {
      const uint32_t o = sbase + j * T::kStage;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float x[4] = {y[i][0].x, y[i][0].y, y[i][1].x, y[i][1].y};
        uint4 hi, lo;
        split4(x, hi, lo);
        const uint32_t d = o + ((warp + 16 * i) >> 2) * T::kChunkA + (32 * (warp & 3) + lane) * 16;
        sts128(d, hi);
        sts128(d + T::kA, lo);
      }
    };
    // sums: G rows 32 (warp % 4) + lane, bands 8 (warp / 4) + 32 c + q
    float re[T::kG][8], im[T::kG][8];
    auto clear = [&]() __attribute__((always_inline)) {
#pragma unroll
      for (int c = 0; c < T::kG; ++c)
#pragma unroll
        for (int q = 0; q < 8; ++q) re[c][q] = im[c][q] = 0.f;
    };
    const uint32_t tq = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * (warp >> 2);
    auto drain = [&](int b) __attribute__((always_inline)) {   // block b
      const int set = b & 1;
      ok = bar_wait<kWaitLimit>(&accf[set], (b >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < T::kG; ++c) {
        uint32_t x[8], y[8];
        TMEM_LD8(tq + set * T::N + 32 * c, x);
        TMEM_LD8(tq + set * T::N + NB + 32 * c, y);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          re[c][q] += __uint_as_float(x[q]);
          im[c][q] += __uint_as_float(y[q]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&acce[set]);
    };
    auto finish = [&](int u) __attribute__((always_inline)) {
      const int bt = u % nbt, t = u / nbt, k = t / ntile;
      const int g = (t - k * ntile) * 128 + 32 * (warp & 3) + lane, b0 = bt * NB + 8 * (warp >> 2);
      float2 *o = out + (size_t)k * os_k + g;
#pragma unroll
      for (int c = 0; c < T::kG; ++c)
#pragma unroll
        for (int r = 0; r < 8; r += 4) {
          float2 w[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int b = b0 + 32 * c + r + q;
            w[q] = ACCUM && g < nG && b < ni ? o[(size_t)b * nG] : make_float2(0.f, 0.f);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int b = b0 + 32 * c + r + q;
            if (g < nG && b < ni) o[(size_t)b * nG] = make_float2(re[c][r + q] + w[q].x, im[c][r + q] + w[q].y);
          }
        }
      clear();
    };
    clear();
    int it = 0, bl = 0, s = 0, u = blockIdx.x;
    load(v0);
    load(v1);
    auto stage = [&](float2 (&x)[2][2]) __attribute__((always_inline)) {
      const int j = it & 1;
      if (it >= 2) ok = bar_wait<kWaitLimit>(&free_[j], ((it >> 1) - 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return;
      put(j, x);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&full[j]);
      load(x);
      ++it;
      if ((s & 1) || s == nst - 1) {   // end of block bl: take the one before, a unit's last one with its store
        if (bl > 0) drain(bl - 1);
        if (ok && bl > 0 && s < 2) finish(u - gridDim.x);
        ++bl;
      }
      if (++s == nst) {
        s = 0;
        u += gridDim.x;
      }
    };
    while (ok && u < units) {
      stage(v0);
      if (ok && u < units) stage(v1);
    }
    if (ok && bl > 0) {
      drain(bl - 1);
      if (ok) finish(u - gridDim.x);
    }
    if (!ok && lane == 0) atomicOr(&g_tc05_error, 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kBWarps) tmem_free(tmem, T::kCols);
}

static int deep_nb(int ni) {   // equal tiles of up to 96 bands, in whole warps
  const int nbt = (ni + 95) / 96;
  return ((ni + nbt - 1) / nbt + 31) / 32 * 32;
}

// Scratch of the packed X; 0 where k_apply_tc05 runs.  That one keeps up to 32 projectors of X in shared
// memory for all its G, and without packing it is quicker below about 3 stages per SM (ncu, one-chunk kernel
// against packing + this one: 40 bands x 64 projectors x 6000 G, 188 stages: 11.2 / 12.8 us;
// 64 x 36 x 20000, 471: 18.7 / 17.4; 80 x 128 x 12000, 752: 30.7 / 19.5; 64 x 64 x 142800: 68.5 / 60.3; 96 x 40 x
// 190000: 152 / 95; Si64, 168 x 256 x 23847: 152 / 71; rms error there 3.7e-6 / 6.0e-7).
size_t apply_tc05_bytes(int nk, int nj, int ni, int nG) {
  if (nj <= kAJ) return 0;
  const int nb = deep_nb(ni);
  const long units = (long)((nG + 127) / 128) * ((ni + nb - 1) / nb) * nk;
  if (units * ((nj + kDJ - 1) / kDJ) < 3 * 152) return 0;
  return (size_t)nk * ((ni + nb - 1) / nb) * ((nj + kDJ - 1) / kDJ) * (32 * kDJ * nb);
}

template <int NB, bool ACCUM>
static addft_status apply_deep_go(int nsm, const float2 *X, int xs_j, int xs_i, size_t xs_k, const float2 *A, size_t as_k,
                                  int nk, int nj, int ni, int nG, float2 *out, size_t os_k, void *work, cudaStream_t st) {
  const int nst = (nj + kDJ - 1) / kDJ, nbt = (ni + NB - 1) / NB;
  k_deep_pack<NB><<<dim3(nst * kDJ / 2, nbt, nk), NB, 0, st>>>(X, xs_j, xs_i, xs_k, nj, ni, nst, nbt, (unsigned char *)work);
  ADDFT_TRY(check_launch("k_deep_pack"));
  const long units = (long)((nG + 127) / 128) * ((ni + NB - 1) / NB) * nk;
  ADDFT_TRY(smem_optin(k_apply_deep<NB, ACCUM>, DT<NB>::kSmem));
  k_apply_deep<NB, ACCUM><<<(int)std::min<long>(units, nsm), kBThreads + 32, DT<NB>::kSmem, st>>>(
      (const unsigned char *)work, A, as_k, nk, nj, ni, nG, out, os_k);
  return check_launch("k_apply_deep");
}

addft_status launch_apply_tc05(bool accum, const float2 *X, int xs_j, int xs_i, size_t xs_k, const float2 *A,
                               size_t as_k, int nk, int nj, int ni, int nG, float2 *out, size_t os_k,
                               void *work, size_t bytes, cudaStream_t st) {
  int dev = 0, nsm = 0;
  ADDFT_CUDA(cudaGetDevice(&dev));
  ADDFT_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const size_t need = apply_tc05_bytes(nk, nj, ni, nG);
  if (need > 0 && work && ((uintptr_t)work & 15) == 0 && bytes >= need) {
    const int nb = deep_nb(ni) / 32;
#define DEEP(c, a) \
  if (nb == c && accum == a) \
    return apply_deep_go<32 * c, a>(nsm, X, xs_j, xs_i, xs_k, A, as_k, nk, nj, ni, nG, out, os_k, work, st);
    DEEP(1, true) DEEP(2, true) DEEP(3, true) DEEP(1, false) DEEP(2, false) DEEP(3, false)
#undef DEEP
  }
  ADDFT_TRY(smem_optin(accum ? k_apply_tc05<true> : k_apply_tc05<false>, kApplySmem));
  const int nbt = (ni + kAB - 1) / kAB, ntile = (nG + kAG - 1) / kAG;
  int gx = (nsm + nbt * nk - 1) / (nbt * nk);   // about one CTA per SM over the whole grid
  if (gx > ntile) gx = ntile;
  if (gx < 1) gx = 1;
  dim3 grid(gx, nbt, nk);
  if (accum)
    k_apply_tc05<true><<<grid, 256, kApplySmem, st>>>(X, xs_j, xs_i, xs_k, A, as_k, nj, ni, nG, out, os_k);
  else
    k_apply_tc05<false><<<grid, 256, kApplySmem, st>>>(X, xs_j, xs_i, xs_k, A, as_k, nj, ni, nG, out, os_k);
  return check_launch("k_apply_tc05");
}

// ---------------------------------------------------------------------------
// Peak rate of kind::tf32 MMAs: one CTA per SM, one thread issues `iters` MMAs of
// 128 x 256 x 8 on fixed shared-memory operands into one tensor-memory accumulator,
// then waits (bounded) for their completion.  Diagnostic for the compute roof.
// ---------------------------------------------------------------------------
namespace {
constexpr int kPeakN = 256;
}  // namespace

__global__ void __launch_bounds__(128, 1) k_peak_tc05(int iters) {
  __shared__ __align__(128) unsigned char a_s[128 * 32];
  __shared__ __align__(128) unsigned char b_s[kPeakN * 32];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int i = tid; i < (int)sizeof(a_s) / 4; i += blockDim.x) reinterpret_cast<float *>(a_s)[i] = 1e-3f;
  for (int i = tid; i < (int)sizeof(b_s) / 4; i += blockDim.x) reinterpret_cast<float *>(b_s)[i] = 1e-3f;
  if (tid == 0) bar_init(&bar);
  if (warp == 0) tmem_alloc(&tslot, kPeakN);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  if (tid == 0) {
    const uint64_t ad = sdesc(smem_addr(a_s), 128, 256), bd = sdesc(smem_addr(b_s), 128, 256);
    const uint32_t idesc = idesc_tf32(128, kPeakN);
    for (int it = 0; it < iters; ++it) mma_tf32(tmem, ad, bd, idesc, it > 0 ? 1u : 0u);
    mma_commit(&bar);
  }
  __syncthreads();   // the issuing loop is finite; only the MMAs still queued remain
  const bool ok = __syncthreads_and(bar_wait<kWaitLimit>(&bar, 0)) != 0;
  if (!ok && tid == 0) atomicOr(&g_tc05_error, 1u);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_free(tmem, kPeakN);
}

// Launches k_peak_tc05 on every SM (warm-up, then a timed launch); *tflops and *ms of the
// timed launch.  Synchronises with the stream.
addft_status peak_tc05(int iters, double *tflops, float *ms, cudaStream_t st) {
  int dev = 0, nsm = 0;
  ADDFT_CUDA(cudaGetDevice(&dev));
  ADDFT_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  k_peak_tc05<<<nsm, 128, 0, st>>>(iters / 16 + 1);
  ADDFT_TRY(check_launch("k_peak_tc05 (warm-up)"));
  cudaEvent_t e0, e1;
  ADDFT_CUDA(cudaEventCreate(&e0));
  ADDFT_CUDA(cudaEventCreate(&e1));
  ADDFT_CUDA(cudaEventRecord(e0, st));
  k_peak_tc05<<<nsm, 128, 0, st>>>(iters);
  const addft_status s = check_launch("k_peak_tc05");
  ADDFT_CUDA(cudaEventRecord(e1, st));
  ADDFT_CUDA(cudaEventSynchronize(e1));
  float t = 0.f;
  ADDFT_CUDA(cudaEventElapsedTime(&t, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  ADDFT_TRY(s);
  *ms = t;
  *tflops = (double)nsm * iters * 2.0 * 128 * kPeakN * 8 / (t * 1e-3) / 1e12;
  return ADDFT_OK;
}

}  // namespace addft

extern "C" {

// Bit set of device-side errors of the tcgen05 kernels since the last call (bit 0: an
// mbarrier wait ran out); reading clears it.  Synchronises with the device.
unsigned addft_tc05_status(void) {
  unsigned v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, addft::g_tc05_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(addft::g_tc05_error, &z, sizeof(z));
  return v | addft::oz_status() | addft::d64_status();
}

}  // extern "C"
