// FP64 transforms between the G-sphere and the box as matrix products on the 5th-generation tensor
// cores (tcgen05.mma kind::f16), FP64 accurate through exact digit slices (see ozgemm.cu).
//
// GB300 issues under two FP64 instructions per SM and cycle, so a 75-point FFT line costs about
// 1,000 SM cycles however it is factored (1,700 instructions).  As a product with the DFT matrix
// it needs 75 x 35 complex multiplications (35 = active indices of the sphere on that axis: only
// those are read by an inverse and produced by a forward transform) and these run on the tensor
// cores at 39 cycles per line, 16 inputs and 64 outputs: 234 and 195 cycles.
//
// A stage transforms one axis:   out[o][line] = sum_k F[o][k] in[k][line]
//   z inverse: sphere columns -> Z[column][z];      y inverse: Z -> Y[plane][z][y];
//   x inverse: Y -> times V into U[z][y][x], or |.|^2 summed over bands, or psi(r);
//   x forward: U (or a real-space field) -> X[z][y][plane];  y forward: X -> W[z][plane][y index];
//   z forward: W -> the sphere (scaled, plus kin psi for H psi).
// Every stage writes its output index fastest and the next one takes neighbouring lines along that
// index, so loads (lanes = lines) and stores (lanes = outputs) are both coalesced.
//
// k_d64: persistent, one CTA per SM, on blocks of 32 lines.  F stays in shared memory as digits: per 16 k
// and slice the rows [-Im F | Re F | Im F] of R outputs, so that [Re; Im] and [-Im; Re] (2 R <= 128
// rows) are the same bytes from two offsets and one accumulator row holds Re or Im of an output:
//   D = [Re F; Im F] Re x + [-Im F; Re F] Im x.
// Producer warps load 8 inputs of a line per lane, agree on the line's largest exponent and write
// its 8 digits per component (62 bits below that exponent) into a ring of operand buffers;
// one thread issues the MMAs (slice s of F against slices 0 .. 7 - s of the lines, side by side along
// N = 32 (8 - s), landing on levels s .. 7; F has 7 slices); twelve epilogue warps empty one of the two accumulators
// (8 levels x 32 lines) while the other is filled, add the levels in 64-bit integers and round once
// to FP64.  All waits are bounded (status as in ozgemm.cu).  The error of an output is that of the slicing, 2^-62
// of the line's largest component and 2^-55 of F per term, of the level sums (2^-55 of that component), and of one
// rounding: like an FFT's it is relative to the line, and against 80-bit transforms it is at or below the FFT kernels'
// (densities, rms: 32 x 32 x 60 1.3e-16 both, 27 x 27 x 54 3.8e-16 -> 1.4e-16, 36^3 2.1e-16 -> 1.3e-16).  A line with an
// infinity or a NaN is NaN as a whole, where an FFT leaves infinities in some components.
//   Si64, 75^3, 160 bands: local H psi 11.5 -> 3.9 ms, density 9.2 -> 2.3 ms; 15^3, 64 bands, H psi with its
// projectors 328 -> 160 us (six launches of 13 to 21 us: filling F and the first lines, not rates).
#include <algorithm>
#include <cmath>

#include "dft64.cuh"
#include "mma16.cuh"
#include "ozgemm.cuh"
#include "roots.hpp"

namespace addft {

namespace {

__device__ unsigned g_d64_error = 0;

constexpr int kS = 8;            // digits of a line's inputs
constexpr int kBits = 62;
constexpr int kSF = 7;           // digits of F: entries up to 1 to 2^-54, below their own rounding
constexpr int kFBits = 54;
constexpr int kLines = 32;       // lines per block
constexpr int kStep = 16;        // k per MMA
constexpr int kMaxK = 128;       // a level's 256 (l + 1) products of 2^14: exact below 2^24, 2^25 with aligned digits at most
constexpr int kMaxRing = 8;      // operand buffers (one kstep of 32 lines each)
constexpr int kItem = 2 * kS * kLines * kStep * 2;   // 16 KB
// Warps 0 .. 15 with warp % 4 < 3 empty the accumulator rows 32 (warp % 4) .. of 8 lines each (2 R <= 96
// rows); warps 3, 7, 11 and those of 16 .. 26 with warp % 4 < 3 produce; warp 15 issues MMAs, on the
// scheduler that has no epilogue warps.
constexpr int kEpi = 12, kProd = 12, kEpiLines = 8;
constexpr int kThreads = 32 * 27;
constexpr int kMaxGroups = 4;    // groups of producers, each on blocks of its own
constexpr int kLex = 32;         // blocks whose exponents are kept
constexpr int kWait = 1 << 20;
constexpr int kMaxR = 48;
constexpr size_t kRoom = 221000;      // shared memory for F and the ring
constexpr size_t kMaxF = kRoom - 4 * kItem;
constexpr int kSms = 152;

enum Stage { ZI, YI, XI_V, XI_R, XI_C, XI_D, XF, XR_R, XR_C, YF, ZF, ZF_H };

struct Args {
  PlanDev pd;
  D64Mat m;
  const unsigned char *F;
  int nq, nz;              // as in D64Plan
  const int *col_zg, *col_of, *col_pq;
  long lines;              // over all bands of the chunk (XI_D: per band)
  int nb;                  // bands of the chunk
  const double2 *in;
  double2 *out;
  const double *rin;       // XR_R
  const double *V;         // XI_V: [z][y][x], scaled
  double scale;
  long sz, sy;             // YF: strides of z and y in X
  const double2 *psi;      // ZF_H
  const double *kin;
  int nb_per_k, batch0;
  const double *wocc;      // XI_D
  double *part;            //   [group][z][y][x]
  int groups, per;         //   band groups, bands per group
  int ring, pw, ngrp, spg; // operand buffers; warps of a producer group, groups, buffers of each
};

// where a line reads its inputs (line numbers of a chunk stay below 2^30)
struct Line { long base; int aux; };

template <int ST>
__device__ __forceinline__ Line line_at(const Args &a, unsigned l) {
  const PlanDev &pd = a.pd;
  Line r;
  r.aux = 0;
  if (ST == ZI) {
    const unsigned b = l / (unsigned)pd.nrows;
    r.base = (long)b * pd.nG;
    r.aux = (int)(l - b * pd.nrows) * a.nz;
  } else if (ST == YI) {
    const unsigned t = l / (unsigned)pd.n3, b = t / (unsigned)pd.np;
    r.base = (long)b * pd.nrows * pd.n3 + (l - t * pd.n3);
    r.aux = (int)(t - b * pd.np) * a.nq;
  } else if (ST == XI_V || ST == XI_R || ST == XI_C || ST == XI_D) {
    const unsigned n = pd.n2 * pd.n3, b = l / n;
    r.base = (long)b * pd.np * n + (l - b * n);
  } else if (ST == XF) {
    r.base = (long)l * pd.n1;
  } else if (ST == XR_R || ST == XR_C) {   // lines (band, y, z)
    const unsigned n = pd.n2 * pd.n3, b = l / n;
    r.base = (long)b * n * pd.n1 + (l - b * n);
  } else if (ST == YF) {
    const unsigned t = l / (unsigned)pd.np, b = t / (unsigned)pd.n3;
    r.base = (long)b * pd.n2 * pd.n3 * pd.np + (t - b * pd.n3) * a.sz + (l - t * pd.np);
  } else {
    const unsigned b = l / (unsigned)pd.nrows;
    r.base = (long)b * pd.n3 * pd.np * a.nq + a.col_pq[l - b * pd.nrows];
  }
  return r;
}

// lines of one band in the stages whose stores need the band
template <int ST>
__device__ __forceinline__ unsigned period(const PlanDev &pd) {
  return ST == XI_V ? pd.n2 * pd.n3 : (ST == ZF || ST == ZF_H ? pd.nrows : 0x7fffffff);
}

template <int ST>
__device__ __forceinline__ double2 load_at(const Args &a, const Line &l, int k) {
  const PlanDev &pd = a.pd;
  const double2 z = make_double2(0.0, 0.0);
  if (ST == ZI) {
    const int g = a.col_zg[l.aux + k];
    return g >= 0 ? a.in[l.base + g] : z;
  } else if (ST == YI) {
    const int c = a.col_of[l.aux + k];
    return c >= 0 ? a.in[l.base + (long)c * pd.n3] : z;
  } else if (ST == XI_V || ST == XI_R || ST == XI_C || ST == XI_D || ST == XR_C) {
    return a.in[l.base + (long)k * pd.n2 * pd.n3];
  } else if (ST == XR_R) {
    return make_double2(a.rin[l.base + (long)k * pd.n2 * pd.n3], 0.0);
  } else if (ST == XF) {
    return a.in[l.base + k];
  } else if (ST == YF) {
    return a.in[l.base + k * a.sy];
  } else {
    return a.in[l.base + (long)k * pd.np * a.nq];
  }
}

// What a store needs beside the value, read before the accumulator is waited for: V(r), or the sphere
// point and kin psi there (reading it between the stores of a block cost a memory latency each).
template <int ST>
__device__ __forceinline__ void pre_at(const Args &a, unsigned band, unsigned rem, int o, int comp, double &x, int &g) {
  const PlanDev &pd = a.pd;
  if (ST == XI_V) x = __ldg(a.V + (long)rem * pd.n1 + o);
  if (ST == ZF || ST == ZF_H) g = __ldg(a.col_zg + rem * a.nz + o);
  if (ST == ZF_H) {
    x = 0.0;
    if (g >= 0)
      x = __ldg(a.kin + (long)((a.batch0 + (int)band) / a.nb_per_k) * pd.nG + g) *
          __ldg(reinterpret_cast<const double *>(a.psi) + 2 * ((long)band * pd.nG + g) + comp);
  }
}

// one component of output o of line l (of band `band`)
template <int ST>
__device__ __forceinline__ void store_at(const Args &a, unsigned l, unsigned band, int o, int comp, double v, double x,
                                         int g) {
  const PlanDev &pd = a.pd;
  double *out = reinterpret_cast<double *>(a.out);
  if (ST == ZI) out[2 * ((long)l * pd.n3 + o) + comp] = v;
  else if (ST == YI) out[2 * ((long)l * pd.n2 + o) + comp] = v;
  else if (ST == XI_V) out[2 * ((long)l * pd.n1 + o) + comp] = v * x;
  else if (ST == XI_C) out[2 * ((long)l * pd.n1 + o) + comp] = v * a.scale;
  else if (ST == XI_R) { if (!comp) out[(long)l * pd.n1 + o] = v * a.scale; }
  else if (ST == XF || ST == XR_R || ST == XR_C) out[2 * ((long)l * pd.np + o) + comp] = v;
  else if (ST == YF) out[2 * ((long)l * a.nq + o) + comp] = v;
  else if (g >= 0) out[2 * ((long)band * pd.nG + g) + comp] = ST == ZF_H ? v + x : v * a.scale;
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// T 2^n rounded to FP64, n in -1000 .. 900.  `scaled` takes one conversion on the FP64 pipe and an
// exponent addition; to_double stays on the integer pipes (three times the instructions), for the
// x inverse, whose products with V or squares keep the FP64 pipe busy already.
__device__ __forceinline__ double scaled(long long T, int n) {
  const double d = __ll2double_rn(T);
  return T == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (n << 20), __double2loint(d));
}
__device__ __forceinline__ double to_double(long long T, int n) {
  const unsigned long long u = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
  if (u == 0) return 0.0;
  const int z = __clzll((long long)u);
  const unsigned long long top = u << z, sign = (unsigned long long)T & 0x8000000000000000ull;
  // the leading one of top >> 11 adds one to the exponent
  const unsigned long long r = ((unsigned long long)(62 - z + n + 1023) << 52) + (top >> 11) + ((top >> 10) & 1);
  return __longlong_as_double((long long)(r | sign));
}

// x as q = trunc(x 2^(62 - E)) of a line with exponent field em, 128 added to every byte but the top
__device__ __forceinline__ uint64_t d64_bytes(double x, int em) {
  const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
  const int e = (int)(xh >> 20) & 0x7ff;
  // 53 significand bits with the leading one at bit 61, then down by the exponents' difference
  uint32_t h = (__funnelshift_l(xl, xh, 9) & 0x1fffffffu) | (e ? 0x20000000u : 0u), l = xl << 9;
  int d = em - max(e, 1);
  if (d >= 32) {
    l = h;
    h = 0;
    d -= 32;
  }
  l = __funnelshift_rc(l, h, d);
  h = d < 32 ? h >> d : 0;
  const uint32_t s = (uint32_t)((int)xh >> 31);
  const uint64_t q = ((uint64_t)(h ^ s) << 32) | (l ^ s);
  return q + (0x0080808080808080ull - (uint64_t)(int64_t)(int)s);
}

template <int ST>
__global__ void __launch_bounds__(kThreads, 1) k_d64(Args a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((1024 - (smem_addr(smem_raw) & 1023)) & 1023);
  __shared__ __align__(8) uint64_t fullB[kMaxRing], emptyB[kMaxRing], accf[2], acce[2], fbar;
  __shared__ uint16_t pm[2][kProd][kLines];   // exponents found by each producer warp
  __shared__ uint16_t lex[kLex][kLines];      // exponents of the lines of the last blocks
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nks = a.m.nks, R = a.m.R, tile = blockIdx.y;
  const int ngrp = a.ngrp, spg = a.spg;
  const unsigned nblk = (unsigned)((a.lines + kLines - 1) / kLines);
  const unsigned units = ST == XI_D ? nblk * a.groups : nblk;
  if (tid == 0) {
    for (int i = 0; i < a.ring; ++i) {
      bar_init(&fullB[i], 2);
      bar_init(&emptyB[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      bar_init(&accf[i], 1);
      bar_init(&acce[i], kEpi);
    }
    bar_init(&fbar, 1);
  }
  if (warp == 0) tmem_alloc(&tslot, 512);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tslot;
  const uint32_t sring = smem_addr(smem), sF = sring + a.ring * kItem;   // F last: its 128-row reads may run past it
  bool ok = true;

  // a block: 32 lines starting at l0 (XI_D: of one band); `inner` blocks share a unit
  auto unit_info = [&](unsigned u, unsigned &l0, int &b0, int &inner) {
    if (ST == XI_D) {
      const unsigned lb = u / (unsigned)a.groups;
      const int g = (int)(u - lb * a.groups);
      l0 = lb * kLines;
      b0 = g * a.per;
      inner = max(0, min(a.per, a.nb - b0));
    } else {
      l0 = u * kLines;
      b0 = 0;
      inner = 1;
    }
  };

  const bool epi = warp < 16 && (warp & 3) < 3;
  if (!epi && warp != 15) {
    // ---- producers: lane = line, warp = 8 inputs (and 8 more where a group has fewer warps).  Groups
    // take blocks in turn, so one loads while another converts; each has buffers of its own (at
    // least a block's), or, alone, may share one between inputs of the same warps: the previous
    // user of a buffer has then always been filled when its release is waited for.
    const int pi = warp < 16 ? warp >> 2 : 3 * (warp >> 2) + (warp & 3) - 9, grp = pi / a.pw, me = pi - grp * a.pw;
    const int noct = 2 * nks;
    unsigned blk = 0;
    if (grp < ngrp && (warp < 16 || (warp & 3) < 3))
    for (unsigned u = blockIdx.x; u < units; u += gridDim.x) {
      unsigned l0;
      int b0, inner;
      unit_info(u, l0, b0, inner);
      for (int it = 0; it < inner; ++it, ++blk) {
        const unsigned turn = blk / (unsigned)ngrp;
        if ((int)(blk - turn * ngrp) != grp) continue;
        unsigned l = l0 + lane;
        const bool live = l < a.lines;
        if (ST == XI_D) l += (unsigned)(b0 + it) * (unsigned)a.lines;
        const Line ln = line_at<ST>(a, live ? l : 0);
        double2 x[8];
        auto load = [&](int o) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int k = 8 * o + j;
            x[j] = live && k < a.m.K ? load_at<ST>(a, ln, k) : make_double2(0.0, 0.0);
          }
        };
        int em = 0;
        // with more than 64 inputs a warp has two groups of 8; the first stays in registers
#pragma unroll 1
        for (int o = noct > a.pw ? me + a.pw : me; o >= 0; o -= a.pw) {
          load(o);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            em = max(em, max((__double2hiint(x[j].x) >> 20) & 0x7ff, (__double2hiint(x[j].y) >> 20) & 0x7ff));
        }
        uint16_t(*p)[kLines] = pm[turn & 1] + grp * a.pw;
        p[me][lane] = (uint16_t)em;
        // every warp of the group gets here, failed or not
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * a.pw) : "memory");
        for (int w = 0; w < a.pw; ++w) em = max(em, (int)p[w][lane]);
        if (me == 0) lex[blk % kLex][lane] = (uint16_t)em;
#pragma unroll 1
        for (int o = me; o < noct; o += a.pw) {
          if (o > me) load(o);
          const unsigned t = turn * nks + (o >> 1), round = t / (unsigned)spg;
          const int slot = grp * spg + (int)(t - round * spg);
          if (ok && round > 0) ok = __all_sync(0xffffffffu, bar_wait<kWait>(&emptyB[slot], (round - 1) & 1));
          if (!ok) continue;
          const uint32_t dst = sring + slot * kItem + (lane >> 3) * 256 + (o & 1) * 128 + (lane & 7) * 16;
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            uint64_t q[8];
#pragma unroll
            // a line that is not finite is all NaN in the epilogue, whatever its digits
            for (int j = 0; j < 8; ++j) q[j] = d64_bytes(em == 0x7ff ? 0.0 : (part ? x[j].y : x[j].x), max(em, 1));
#pragma unroll
            for (int s = 0; s < kS; ++s) {
              uint32_t hh[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) hh[j] = digit_pair<kS>(q[2 * j], q[2 * j + 1], s);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + (part * kS + s) * (kLines * kStep * 2)),
                           "r"(hh[0]), "r"(hh[1]), "r"(hh[2]), "r"(hh[3])
                           : "memory");
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) bar_arrive(&fullB[slot]);
        }
      }
    }
    if (!ok && lane == 0) atomicOr(&g_d64_error, 1u);
  } else if (!epi) {
    // ---- F, then MMAs
    const bool lead = elect_one();
    if (lead) {
      const uint32_t bytes = (uint32_t)a.m.tile_bytes;
      const unsigned char *src = a.F + a.m.off + (size_t)tile * bytes;
      bar_expect(&fbar, bytes);
      for (uint32_t o = 0; o < bytes; o += 32768) bulk_copy(sF + o, src + o, min(32768u, bytes - o), &fbar);
    }
    ok = bar_wait<kWait>(&fbar, 0);
    const uint32_t sl = (3 * R * 32) >> 4;   // one slice of F, in descriptor units
    const uint32_t fre = desc_lo(sF + R * 32), fim = desc_lo(sF), ring0 = desc_lo(sring);
    unsigned blk = 0, slot = 0, grp = 0;     // blk % ngrp; each group's buffers in turn
    unsigned round = 0, pos = 0;             // of the current group's next buffer
    bool issued = false;
    for (unsigned u = blockIdx.x; u < units && ok; u += gridDim.x) {
      unsigned l0;
      int b0, inner;
      unit_info(u, l0, b0, inner);
      for (int it = 0; it < inner && ok; ++it, ++blk) {
        const unsigned buf = blk & 1;
        if (blk >= 2) ok = bar_wait<kWait>(&acce[buf], (blk / 2 - 1) & 1);
        const unsigned turn = blk / (unsigned)ngrp;
        grp = blk - turn * ngrp;
        round = turn * nks / (unsigned)spg;
        pos = turn * nks - round * spg;
        for (int j = 0; j < nks && ok; ++j) {
          slot = grp * spg + pos;
          ok = bar_wait<kWait>(&fullB[slot], round & 1);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          issued = true;
          if (lead) {
            const uint32_t d = tmem + 256 * buf, b = ring0 + slot * (kItem >> 4), f = j * kSF * sl;
#pragma unroll
            for (int i = 0; i < kSF; ++i)   // [Re; Im] Re x
              mma_f16(d + 32 * i, fre + f + i * sl, b, idesc_f16(32 * (kS - i), false), !(j == 0 && i == 0));
#pragma unroll
            for (int i = 0; i < kSF; ++i)   // [-Im; Re] Im x
              mma_f16(d + 32 * i, fim + f + i * sl, b + ((kS * kLines * kStep * 2) >> 4), idesc_f16(32 * (kS - i), false), 1);
            mma_commit(&emptyB[slot]);
            if (j == nks - 1) mma_commit(&accf[buf]);
          }
          __syncwarp();
          if (++pos == (unsigned)spg) {
            pos = 0;
            ++round;
          }
        }
      }
    }
    if (!ok) {
      if (lead) atomicOr(&g_d64_error, 1u);
      bar_wait<kWait>(&fbar, 0);
      if (issued) {   // no MMA may be in flight when tensor memory is given back
        if (lead) mma_commit(&accf[0]);
        __syncwarp();
        bar_wait<kWait>(&accf[0], 0);
        bar_wait<kWait>(&accf[0], 1);
      }
    }
  } else {
    // ---- epilogue: warp reads accumulator rows 32 (w % 4) .. of kEpiLines lines
    const int q = warp & 3, c0 = kEpiLines * (warp >> 2);
    const int row = 32 * q + lane, comp = row >= R ? 1 : 0, r = comp ? row - R : row;
    const int o = tile * a.m.per + r;
    const bool on = row < 2 * R && r < a.m.per && o < a.m.outs;
    const bool any = 32 * q < 2 * R;
    // the level sums as hi 2^32 + lo, hi <= 2^36 2 K: keep as many of lo's bits as 62 bits hold (17 to 20)
    const int keep = 62 - 36 - (32 - __clz(2 * a.m.K));
    const int w4 = 1 << (keep - 8), w5 = 1 << (keep - 16);
    const float w67 = __int_as_float((127 - 32 + keep) << 23);
    // q_F q_x = 256^6 (hi 2^32 + lo); F = q 2^-54, x = q 2^(E - 62), E = field - 1022
    const int nbase = 48 + 32 - keep - kFBits - 1022 - kBits;
    double acc[kEpiLines];
#pragma unroll
    for (int c = 0; c < kEpiLines; ++c) acc[c] = 0.0;
    unsigned blk = 0;
    for (unsigned u = blockIdx.x; u < units && ok; u += gridDim.x) {
      unsigned l0;
      int b0, inner;
      unit_info(u, l0, b0, inner);
      for (int it = 0; it < inner && ok; ++it, ++blk) {
        const int buf = (int)(blk & 1);
        const unsigned per = period<ST>(a.pd);
        double px[kEpiLines];
        int pg[kEpiLines];
        if ((ST == XI_V || ST == ZF || ST == ZF_H) && on) {
          unsigned band = (l0 + c0) / per, rem = (l0 + c0) - band * per;
#pragma unroll
          for (int c = 0; c < kEpiLines; ++c) {
            px[c] = 0.0;
            pg[c] = -1;
            if (l0 + c0 + c < a.lines) pre_at<ST>(a, band, rem, o, comp, px[c], pg[c]);
            if (++rem == per) {
              rem = 0;
              ++band;
            }
          }
        }
        ok = __all_sync(0xffffffffu, bar_wait<kWait>(&accf[buf], (uint32_t)(blk / 2) & 1));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t base = tmem + 256 * buf + ((uint32_t)(32 * q) << 16) + c0;
        long long T[kEpiLines];
        if (any) {
          uint32_t v[2][kEpiLines];
#pragma unroll
          for (int l = 0; l < kS; l += 2) {
            TMEM_LD8(base + 32 * l, v[0]);
            TMEM_LD8(base + 32 * l + 32, v[1]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < kEpiLines; ++c) {
              const float f0 = __uint_as_float(v[0][c]), f1 = __uint_as_float(v[1][c]);
              if (l == 0) T[c] = mad_wide(__float2int_rn(f0), 1 << 24, mad_wide(__float2int_rn(f1), 1 << 16, 0));
              else if (l == 2) T[c] = mad_wide(__float2int_rn(f0), 1 << 8, mad_wide(__float2int_rn(f1), 1, T[c])) << keep;
              else if (l == 4) T[c] = mad_wide(__float2int_rn(f0), w4, mad_wide(__float2int_rn(f1), w5, T[c]));
              else T[c] = mad_wide(__float2int_rn(fmaf(f0, 256.0f, f1) * w67), 1, T[c]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(&acce[buf]);   // the accumulator has been read
        if (!on) continue;
        const double wb = ST == XI_D ? a.wocc[b0 + it] : 0.0;
        unsigned band = (l0 + c0) / per, rem = (l0 + c0) - band * per;
#pragma unroll
        for (int c = 0; c < kEpiLines; ++c) {
          const unsigned l = l0 + c0 + c;
          if (l >= a.lines) break;
          if (c > 0 && ++rem == per) {
            rem = 0;
            ++band;
          }
          const int em = lex[blk % kLex][c0 + c], n = nbase + max(em, 1);
          double v;
          if (n >= -1000 && n <= 900) v = ST == XI_D || ST == XI_V ? to_double(T[c], n) : scaled(T[c], n);
          else v = scale2(scale2((double)T[c], n / 2), n - n / 2);
          if (em == 0x7ff) v = __longlong_as_double(0x7ff8000000000000ll);
          if (ST == XI_D) acc[c] = fma(wb * v, v, acc[c]);
          else store_at<ST>(a, l, band, o, comp, v, px[c], pg[c]);
        }
      }
      if (ST == XI_D && ok) {   // Re^2 and Im^2 sit in different rows: [group][2][z][y][x]
        const int g = b0 / a.per;
        double *dst = a.part + ((size_t)g * 2 + comp) * a.lines * a.pd.n1;
#pragma unroll
        for (int c = 0; c < kEpiLines; ++c) {
          const unsigned l = l0 + c0 + c;
          if (on && l < a.lines) dst[(long)l * a.pd.n1 + o] = acc[c];
          acc[c] = 0.0;
        }
      }
    }
    if (!ok && lane == 0) atomicOr(&g_d64_error, 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 512);
}

// Vt[z][y][x] = V[x][y][z] * s, through shared-memory tiles of 32 x 32 (x, z) per y
__global__ void __launch_bounds__(256) k_d64_v(PlanDev pd, const double *__restrict__ V, double s, double *__restrict__ Vt) {
  __shared__ double T[32][33];
  const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 32, y = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int x = w; x < 32; x += 8)
    if (x0 + x < pd.n1 && z0 + lane < pd.n3) T[x][lane] = V[((long)(x0 + x) * pd.n2 + y) * pd.n3 + z0 + lane] * s;
  __syncthreads();
  for (int z = w; z < 32; z += 8)
    if (z0 + z < pd.n3 && x0 + lane < pd.n1) Vt[((long)(z0 + z) * pd.n2 + y) * pd.n1 + x0 + lane] = T[lane][z];
}

// out[x][y][z] (+)= sum_j in[j][z][y][x], j < nsum slabs
template <typename T>
__global__ void __launch_bounds__(256)
k_d64_out(PlanDev pd, const T *__restrict__ in, int nsum, double scale, int acc, T *__restrict__ out);

template <>
__global__ void __launch_bounds__(256)
k_d64_out<double>(PlanDev pd, const double *__restrict__ in, int nsum, double scale, int acc, double *__restrict__ out) {
  __shared__ double T[32][33];
  const long N = (long)pd.n1 * pd.n2 * pd.n3;
  const int nzt = (pd.n3 + 31) / 32;
  const int x0 = blockIdx.x * 32, z0 = (blockIdx.y % nzt) * 32, b = blockIdx.y / nzt, y = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int z = w; z < 32; z += 8)
    if (z0 + z < pd.n3 && x0 + lane < pd.n1) {
      const double *p = in + (size_t)b * N + ((long)(z0 + z) * pd.n2 + y) * pd.n1 + x0 + lane;
      double s = 0.0;
      for (int j = 0; j < nsum; ++j) s += p[(size_t)j * N];
      T[z][lane] = s * scale;
    }
  __syncthreads();
  for (int x = w; x < 32; x += 8)
    if (x0 + x < pd.n1 && z0 + lane < pd.n3) {
      double *o = out + (size_t)b * N + ((long)(x0 + x) * pd.n2 + y) * pd.n3 + z0 + lane;
      *o = acc ? *o + T[lane][x] : T[lane][x];
    }
}

template <>
__global__ void __launch_bounds__(256)
k_d64_out<double2>(PlanDev pd, const double2 *__restrict__ in, int, double, int, double2 *__restrict__ out) {
  __shared__ double2 T[32][33];
  const long N = (long)pd.n1 * pd.n2 * pd.n3;
  const int nzt = (pd.n3 + 31) / 32;
  const int x0 = blockIdx.x * 32, z0 = (blockIdx.y % nzt) * 32, b = blockIdx.y / nzt, y = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int z = w; z < 32; z += 8)
    if (z0 + z < pd.n3 && x0 + lane < pd.n1) T[z][lane] = in[(size_t)b * N + ((long)(z0 + z) * pd.n2 + y) * pd.n1 + x0 + lane];
  __syncthreads();
  for (int x = w; x < 32; x += 8)
    if (x0 + x < pd.n1 && z0 + lane < pd.n3) out[(size_t)b * N + ((long)(x0 + x) * pd.n2 + y) * pd.n3 + z0 + lane] = T[lane][x];
}

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// The two scratch regions of a band: Z, U, W in the first, Y, X in the second.
inline size_t region1(const PlanDev &pd) {
  const size_t z = (size_t)pd.nrows * pd.n3, u = (size_t)pd.n1 * pd.n2 * pd.n3, w = (size_t)pd.n3 * pd.np * pd.d64->nq;
  return al256(std::max(std::max(z, u), w) * sizeof(double2));
}
inline size_t region2(const PlanDev &pd) { return al256((size_t)pd.np * pd.n2 * pd.n3 * sizeof(double2)); }

template <int ST>
addft_status stage(const PlanDev &pd, int axis, Args &a, long lines, cudaStream_t st) {
  const D64Plan &t = *pd.d64;
  a.m = t.mat[axis];
  a.F = t.F;
  a.nq = t.nq;
  a.nz = t.nz;
  a.col_zg = t.col_zg;
  a.col_of = t.col_of;
  a.col_pq = t.col_pq;
  a.lines = lines;
  a.ring = std::min<int>(kMaxRing, (int)((kRoom - a.m.tile_bytes) / kItem));
  const int noct = 2 * a.m.nks;
  a.pw = std::min(std::min(noct, kProd), 2 * a.ring);
  a.ngrp = std::max(1, std::min(std::min(kMaxGroups, kProd / a.pw), a.ring / a.m.nks));
  a.spg = a.ring / a.ngrp;
  const size_t sm = (size_t)a.ring * kItem + a.m.tile_bytes + 4096 + 1024;   // a 128-row read may pass F's end
  ADDFT_TRY(smem_optin(k_d64<ST>, sm));
  const long blocks = (lines + kLines - 1) / kLines * (ST == XI_D ? a.groups : 1);
  const int gx = (int)std::max<long>(1, std::min<long>(blocks, kSms / a.m.tiles));
  k_d64<ST><<<dim3(gx, a.m.tiles), kThreads, sm, st>>>(a);
  return check_launch("k_d64");
}

inline Args base_args(const PlanDev &pd, int nb) {
  Args a;
  memset(&a, 0, sizeof(a));
  a.pd = pd;
  a.nb = nb;
  a.scale = 1.0;
  a.nb_per_k = 1;
  return a;
}

// z and y inverse of nb bands: psi -> r1 (Z) -> r2 (Y)
addft_status to_planes(const PlanDev &pd, int nb, const double2 *psi, double2 *r1, double2 *r2, cudaStream_t st) {
  Args a = base_args(pd, nb);
  a.in = psi;
  a.out = r1;
  ADDFT_TRY((stage<ZI>(pd, 2, a, (long)nb * pd.nrows, st)));
  a.in = r1;
  a.out = r2;
  return stage<YI>(pd, 1, a, (long)nb * pd.np * pd.n3, st);
}

// Every entry needs `fixed` bytes and a band's: callers ask for that (d64_runs), and with less nothing runs.
addft_status room(const PlanDev &pd, size_t bytes, size_t fixed) {
  ADDFT_REQUIRE(bytes >= fixed + d64_band_bytes(pd), ADDFT_INVALID_ARG, "dft64: work needs %zu B, got %zu",
                fixed + d64_band_bytes(pd), bytes);
  return ADDFT_OK;
}

}  // namespace

int d64_chunk(const PlanDev &pd, int nbatch, size_t bytes) {
  // as many bands at once as the scratch holds, in equal chunks: every launch has the ramp of 152 CTAs
  // that load F first (160 bands of Si64 in chunks of 10 / 20 / 40 / 80: 6.6 / 6.0 / 5.6 / 5.5 ms)
  const size_t lines = (size_t(1) << 30) / ((size_t)pd.n2 * pd.n3), grid = 65535 / ((pd.n3 + 31) / 32);   // k_d64_out's y
  const int fit = (int)std::min(std::min(bytes / d64_band_bytes(pd), std::min(lines, grid)), (size_t)nbatch);
  if (fit < 1) return 0;
  const int chunks = (nbatch + fit - 1) / fit;
  return (nbatch + chunks - 1) / chunks;
}

bool d64_handles(const PlanDev &pd, D64Op op, int bands) {
  // tuning that asks for the split stages or for other kernels than the defaults keeps to the FFT kernels
  if (!pd.d64->F || !pd.tun.colfft || pd.tun.plane_split) return false;
  for (int a = 0; a < 6; ++a)
    if (pd.d64->mat[a].tiles == 0) return false;
  // Where the products start, in box points x bands at once, by (n1 n2 n3)^(1/3).  They take 65 to 80 (H psi) or
  // 36 to 48 us (density, one way) before the work shows, launches that load F first; the FFT kernels 40 to 60 and
  // 20 to 35, growing with the box.  Measured on 39 boxes from 9^3 to 80^3, cubes and 1 : 1 : 1.25 to 2, 1 to
  // 64 bands, spheres of 0.45 and 0.25 n; FFT / products in us, spheres of 0.45:
  //   H psi    18^3 x 64 bands 97 / 132, 20^3 x 64 130 / 152, 24^3 x 32 109 / 125, x 64 181 / 185, 25^3 x 16 89 / 101,
  //            x 32 144 / 132, 30^3 x 8 80 / 88, x 16 134 / 107, 32^3 x 16 125 / 125, x 32 196 / 180, 36^3 x 8 109 / 109,
  //            32 x 32 x 64 x 4 82 / 103, x 8 142 / 136, 40^3 x 4 116 / 92, 45^3 x 1 98 / 79, 75^3 x 1 239 / 146
  //   density  18^3 x 64 87 / 107, 20^3 x 64 120 / 109, 24^3 x 16 58 / 60, x 32 89 / 79, 30^3 x 8 48 / 53, x 16 74 / 63,
  //            32^3 x 16 72 / 66, 36^3 x 4 54 / 51, x 8 93 / 66, 40^3 x 8 95 / 70, 45^3 x 1 54 / 48
  //   one way  18^3 x 32 46 / 53, x 64 81 / 67, 24^3 x 16 53 / 49, 30^3 x 8 46 / 48, x 16 72 / 55, 32^3 x 16 68 / 62,
  //            36^3 x 1 49 / 43, 45^3 x 1 60 / 44
  struct Row { double size, from[3]; };
  static const Row rows[] = {{22.0, {1300e3, 600e3, 260e3}}, {26.5, {800e3, 400e3, 380e3}}, {31.9, {430e3, 320e3, 320e3}},
                             {33.0, {500e3, 600e3, 520e3}},  {36.5, {400e3, 370e3, 290e3}}, {42.0, {300e3, 430e3, 0}},
                             {1e9, {0, 0, 0}}};
  const double points = (double)pd.n1 * pd.n2 * pd.n3, work = points * bands;
  // Axes of one pass (up to 16 points) give the FFT kernels a CTA per plane and band with one line per thread: their time
  // follows planes x bands and starts early (H psi 12^3 x 32 78 / 68, 15^3 x 32 132 / 80, 16^3 x 32 129 / 89, x 16
  // 72 / 68, 12 x 12 x 24 x 32 78 / 83; density 16^3 x 32 74 / 66, 12^3 x 64 93 / 91; one way 16^3 x 32 50 / 45).
  if (pd.ax[0].nst == 1 && pd.ax[1].nst == 1) {
    const double planes = (double)pd.np * bands;
    return op == D64Op::kHpsi ? planes >= 300 && work >= 55e3 : planes >= 450 && work >= (op == D64Op::kDensity ? 100e3 : 55e3);
  }
  const double size = std::cbrt(points);
  for (const Row &r : rows)
    if (size < r.size) return work >= r.from[(int)op];
  return true;
}

size_t d64_band_bytes(const PlanDev &pd) { return region1(pd) + region2(pd); }
size_t d64_v_bytes(const PlanDev &pd) { return al256((size_t)pd.n1 * pd.n2 * pd.n3 * sizeof(double)); }

addft_status d64_hpsi(const PlanDev &pd, int nbatch, const double2 *psi, const double *v_r, double2 *hpsi,
                      const double *kin, int nb_per_k, void *work, size_t bytes, cudaStream_t st) {
  const long N = (long)pd.n1 * pd.n2 * pd.n3;
  ADDFT_TRY(room(pd, bytes, d64_v_bytes(pd)));
  double *Vt = (double *)work;
  char *w = (char *)work + d64_v_bytes(pd);
  const int nc = d64_chunk(pd, nbatch, bytes - d64_v_bytes(pd));
  k_d64_v<<<dim3((pd.n1 + 31) / 32, (pd.n3 + 31) / 32, pd.n2), 256, 0, st>>>(pd, v_r, 1.0 / (double)N, Vt);
  ADDFT_TRY(check_launch("k_d64_v"));
  double2 *r1 = (double2 *)w, *r2 = (double2 *)(w + (size_t)nc * region1(pd));
  for (int b0 = 0; b0 < nbatch; b0 += nc) {
    const int nb = std::min(nc, nbatch - b0);
    const double2 *pin = psi + (size_t)b0 * pd.nG;
    ADDFT_TRY(to_planes(pd, nb, pin, r1, r2, st));
    Args a = base_args(pd, nb);
    a.V = Vt;
    a.in = r2;
    a.out = r1;
    ADDFT_TRY((stage<XI_V>(pd, 0, a, (long)nb * pd.n2 * pd.n3, st)));
    a.in = r1;
    a.out = r2;
    ADDFT_TRY((stage<XF>(pd, 3, a, (long)nb * pd.n2 * pd.n3, st)));
    a.in = r2;
    a.out = r1;
    a.sz = (long)pd.n2 * pd.np;
    a.sy = pd.np;
    ADDFT_TRY((stage<YF>(pd, 4, a, (long)nb * pd.n3 * pd.np, st)));
    a.in = r1;
    a.out = hpsi + (size_t)b0 * pd.nG;
    a.psi = pin;
    a.kin = kin;
    a.nb_per_k = nb_per_k;
    a.batch0 = b0;
    ADDFT_TRY((stage<ZF_H>(pd, 5, a, (long)nb * pd.nrows, st)));
  }
  return ADDFT_OK;
}

addft_status d64_density(const PlanDev &pd, int nbatch, const double2 *psi, const double *wocc, double dscale, double *rho,
                         void *work, size_t bytes, cudaStream_t st) {
  const long N = (long)pd.n1 * pd.n2 * pd.n3, lines = (long)pd.n2 * pd.n3;
  // band groups so that the CTAs of a tile share the (block, group) units evenly
  const long blocks = (lines + kLines - 1) / kLines;
  int groups = (int)std::max<long>(1, std::min<long>(4, (8 * kSms / pd.d64->mat[0].tiles + blocks - 1) / blocks));
  groups = std::min(groups, nbatch);
  auto part_bytes = [N](int g) { return al256((size_t)g * 2 * N * sizeof(double)); };
  while (groups > 1 && bytes < part_bytes(groups) + d64_band_bytes(pd)) --groups;
  const size_t pb = part_bytes(groups);
  ADDFT_TRY(room(pd, bytes, pb));
  double *part = (double *)work;
  char *w = (char *)work + pb;
  const int nc = d64_chunk(pd, nbatch, bytes - pb);
  double2 *r1 = (double2 *)w, *r2 = (double2 *)(w + (size_t)nc * region1(pd));
  for (int b0 = 0; b0 < nbatch; b0 += nc) {
    const int nb = std::min(nc, nbatch - b0);
    ADDFT_TRY(to_planes(pd, nb, psi + (size_t)b0 * pd.nG, r1, r2, st));
    Args a = base_args(pd, nb);
    a.in = r2;
    a.wocc = wocc + b0;
    a.part = part;
    a.per = (nb + groups - 1) / groups;
    a.groups = (nb + a.per - 1) / a.per;
    ADDFT_TRY((stage<XI_D>(pd, 0, a, lines, st)));
    k_d64_out<double><<<dim3((pd.n1 + 31) / 32, (pd.n3 + 31) / 32, pd.n2), 256, 0, st>>>(pd, part, 2 * a.groups, dscale,
                                                                                        b0 > 0 ? 1 : 0, rho);
    ADDFT_TRY(check_launch("k_d64_out"));
  }
  return ADDFT_OK;
}

addft_status d64_to_real(const PlanDev &pd, int nbatch, const double2 *psi, double scale, void *out, bool real_part,
                         void *work, size_t bytes, cudaStream_t st) {
  const long N = (long)pd.n1 * pd.n2 * pd.n3;
  ADDFT_TRY(room(pd, bytes, 0));
  const int nc = d64_chunk(pd, nbatch, bytes);
  double2 *r1 = (double2 *)work, *r2 = (double2 *)((char *)work + (size_t)nc * region1(pd));
  for (int b0 = 0; b0 < nbatch; b0 += nc) {
    const int nb = std::min(nc, nbatch - b0);
    ADDFT_TRY(to_planes(pd, nb, psi + (size_t)b0 * pd.nG, r1, r2, st));
    Args a = base_args(pd, nb);
    a.in = r2;
    a.out = r1;
    a.scale = scale;
    const dim3 grid((pd.n1 + 31) / 32, (pd.n3 + 31) / 32 * nb, pd.n2);
    if (real_part) {
      ADDFT_TRY((stage<XI_R>(pd, 0, a, (long)nb * pd.n2 * pd.n3, st)));
      k_d64_out<double><<<grid, 256, 0, st>>>(pd, (const double *)r1, 1, 1.0, 0, (double *)out + (size_t)b0 * N);
    } else {
      ADDFT_TRY((stage<XI_C>(pd, 0, a, (long)nb * pd.n2 * pd.n3, st)));
      k_d64_out<double2><<<grid, 256, 0, st>>>(pd, r1, 1, 1.0, 0, (double2 *)out + (size_t)b0 * N);
    }
    ADDFT_TRY(check_launch("k_d64_out"));
  }
  return ADDFT_OK;
}

addft_status d64_from_real(const PlanDev &pd, int nbatch, const void *in, bool in_real, double scale, double2 *psi,
                           void *work, size_t bytes, cudaStream_t st) {
  const long N = (long)pd.n1 * pd.n2 * pd.n3;
  ADDFT_TRY(room(pd, bytes, 0));
  const int nc = d64_chunk(pd, nbatch, bytes);
  double2 *r1 = (double2 *)work, *r2 = (double2 *)((char *)work + (size_t)nc * region1(pd));
  for (int b0 = 0; b0 < nbatch; b0 += nc) {
    const int nb = std::min(nc, nbatch - b0);
    Args a = base_args(pd, nb);
    a.out = r2;
    if (in_real) {
      a.rin = (const double *)in + (size_t)b0 * N;
      ADDFT_TRY((stage<XR_R>(pd, 3, a, (long)nb * pd.n2 * pd.n3, st)));
    } else {
      a.in = (const double2 *)in + (size_t)b0 * N;
      ADDFT_TRY((stage<XR_C>(pd, 3, a, (long)nb * pd.n2 * pd.n3, st)));
    }
    a.in = r2;
    a.out = r1;
    a.sz = pd.np;                       // X[y][z][plane] here
    a.sy = (long)pd.n3 * pd.np;
    ADDFT_TRY((stage<YF>(pd, 4, a, (long)nb * pd.n3 * pd.np, st)));
    a.in = r1;
    a.out = psi + (size_t)b0 * pd.nG;
    a.scale = scale;
    ADDFT_TRY((stage<ZF>(pd, 5, a, (long)nb * pd.nrows, st)));
  }
  return ADDFT_OK;
}

unsigned d64_status() {
  unsigned v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, g_d64_error, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v) cudaMemcpyToSymbol(g_d64_error, &z, sizeof(z));
  return v;
}

// ---------------------------------------------------------------------------
// transform matrices
// ---------------------------------------------------------------------------
static uint16_t half_int(int d) {   // FP16 bits of an integer, |d| <= 128
  if (d == 0) return 0;
  const unsigned a = d < 0 ? -d : d;
  int e = 0;
  while ((a >> (e + 1)) != 0) ++e;
  return (uint16_t)((d < 0 ? 0x8000u : 0u) | ((unsigned)(e + 15) << 10) | ((a << (10 - e)) & 0x3ffu));
}

static void digits_of(int64_t q, uint16_t *h) {   // |q| <= 2^kFBits
  const uint64_t u = (uint64_t)q + 0x0000808080808080ull;
  h[0] = half_int((int)((int64_t)u >> 48));
  for (int s = 1; s < kSF; ++s) h[s] = half_int((int)((u >> (48 - 8 * s)) & 0xff) - 128);
}

void d64_build(int n1, int n2, int n3, const std::vector<int> &xact, const std::vector<int> &yact,
               const std::vector<int> &zact, D64Mat (&dm)[6], std::vector<unsigned char> &blob) {
  const int n[3] = {n1, n2, n3};
  const std::vector<int> *act[3] = {&xact, &yact, &zact};
  for (int m = 0; m < 6; ++m) {
    const int ax = m % 3;
    const bool inv = m < 3;
    D64Mat &d = dm[m];
    memset(&d, 0, sizeof(d));
    d.K = inv ? (int)act[ax]->size() : n[ax];
    d.outs = inv ? n[ax] : (int)act[ax]->size();
    d.nks = (d.K + kStep - 1) / kStep;
    if (d.K > kMaxK) continue;
    for (int t = 1; t <= 8; ++t) {
      const int per = (d.outs + t - 1) / t, R = (per + 7) / 8 * 8;
      const size_t bytes = (size_t)d.nks * kSF * 3 * R * 32;
      if (R > kMaxR || bytes > kMaxF) continue;
      d.tiles = t;
      d.per = per;
      d.R = R;
      d.tile_bytes = (int)bytes;
      break;
    }
    if (d.tiles == 0) continue;
    // digits of the n-th roots of unity: -Im, Re, Im of e^{+-2 pi i t / n}
    std::vector<uint16_t> dig((size_t)n[ax] * 3 * kSF);
    Rounded re, im;
    rounded_roots(n[ax], !inv, kFBits, re, im);
    for (int t = 0; t < n[ax]; ++t) {
      digits_of(-im.q[t], &dig[(size_t)(3 * t) * kSF]);
      digits_of(re.q[t], &dig[(size_t)(3 * t + 1) * kSF]);
      digits_of(im.q[t], &dig[(size_t)(3 * t + 2) * kSF]);
    }
    while (blob.size() % 256) blob.push_back(0);
    d.off = (long)blob.size();
    blob.resize(blob.size() + (size_t)d.tiles * d.tile_bytes, 0);
    for (int t = 0; t < d.tiles; ++t)
      for (int r = 0; r < d.per; ++r) {
        const int o = t * d.per + r;
        if (o >= d.outs) break;
        for (int k = 0; k < d.K; ++k) {
          const long j = inv ? (long)o * (*act[ax])[k] : (long)(*act[ax])[o] * k;
          const int i = (int)(j % n[ax]);
          for (int b = 0; b < 3; ++b) {
            const uint16_t *h = &dig[(size_t)(3 * i + b) * kSF];
            const int row = b * d.R + r;
            for (int s = 0; s < kSF; ++s) {
              unsigned char *p = blob.data() + d.off + (size_t)t * d.tile_bytes +
                                 (size_t)(k / kStep * kSF + s) * (3 * d.R * 32) + (row >> 3) * 256 +
                                 ((k % kStep) / 8) * 128 + (row & 7) * 16 + (k % 8) * 2;
              p[0] = (unsigned char)(h[s] & 0xff);
              p[1] = (unsigned char)(h[s] >> 8);
            }
          }
        }
      }
  }
}

}  // namespace addft
