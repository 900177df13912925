// Nonlocal pseudopotential on GB300: projector tables, the two projector
// contractions of V_NL psi, the nonlocal energy and its envelope gradients,
// and the full matrix-free H psi entry point.
//
// Reference: src/addft/physics/nonlocal_op.py:25-82 (dion_full, projectors,
// becp, vnl_apply, nonlocal_energy), ylm.py:8-26, psp.py:122-128, and
// src/addft/ops/hpsi.py:35-50.
#include "ozgemm.cuh"
#include "radial.cuh"
#include "transforms.cuh"

namespace addft {

constexpr int kMaxAtoms = 256;
constexpr int kMaxK = 64;
constexpr int kMaxNh = 16;

// Kernel-parameter view of the geometry + pseudopotential (no device allocation).
struct GeoParams {
  double B[9];                 // reciprocal rows
  double inv_sqrt_omega;
  int nat, nh, nk;
  double pos[kMaxAtoms * 3];
  double kpt[kMaxK * 3];
  // per projector channel c in [0, nh): radial index, l, m
  int ch_rad[kMaxNh], ch_l[kMaxNh], ch_m[kMaxNh];
  double w[4], b[4];
  int kind;            // 0 analytic, 1 tabulated (rt)
  RadialTab rt;
};

inline addft_status make_geo(GeoParams &g, const double *bvec, double omega, int nk,
                             const double *kpts, int nat, const double *pos, const addft_psp *psp) {
  ADDFT_REQUIRE(nat >= 0 && nat <= kMaxAtoms, ADDFT_UNSUPPORTED, "nat = %d exceeds %d", nat, kMaxAtoms);
  ADDFT_REQUIRE(nk >= 1 && nk <= kMaxK, ADDFT_UNSUPPORTED, "nk = %d exceeds %d", nk, kMaxK);
  ADDFT_REQUIRE(omega > 0, ADDFT_INVALID_ARG, "omega must be > 0");
  memset(&g, 0, sizeof(g));
  for (int i = 0; i < 9; ++i) g.B[i] = bvec[i];
  g.inv_sqrt_omega = 1.0 / sqrt(omega);
  g.nat = nat;
  g.nk = nk;
  for (int i = 0; i < 3 * nat; ++i) g.pos[i] = pos[i];
  for (int i = 0; i < 3 * nk; ++i) g.kpt[i] = kpts ? kpts[i] : 0.0;
  g.nh = 0;
  if (psp) {
    ADDFT_REQUIRE(psp->nrad >= 0 && psp->nrad <= 4, ADDFT_UNSUPPORTED, "psp nrad > 4");
    ADDFT_REQUIRE(psp->kind == 0 || psp->kind == 1, ADDFT_INVALID_ARG, "psp kind must be 0 or 1");
    if (psp->kind == 1)
      ADDFT_REQUIRE(psp->tab != nullptr && psp->nq >= 2 && psp->dq > 0, ADDFT_INVALID_ARG,
                    "tabulated psp needs tab, nq >= 2, dq > 0");
    g.kind = psp->kind;
    g.rt.tab = psp->tab;
    g.rt.nq = psp->nq;
    g.rt.dq = psp->dq;
    for (int ib = 0; ib < psp->nrad; ++ib) {
      ADDFT_REQUIRE(psp->l[ib] >= 0 && psp->l[ib] <= 2, ADDFT_UNSUPPORTED,
                    "projector l = %d not supported (l <= 2)", psp->l[ib]);
      g.w[ib] = psp->w[ib];
      g.b[ib] = psp->b[ib];
      for (int m = 0; m < 2 * psp->l[ib] + 1; ++m) {
        ADDFT_REQUIRE(g.nh < kMaxNh, ADDFT_UNSUPPORTED, "too many projector channels");
        g.ch_rad[g.nh] = ib;
        g.ch_l[g.nh] = psp->l[ib];
        g.ch_m[g.nh] = m;
        ++g.nh;
      }
    }
  }
  return ADDFT_OK;
}

// beta~(q), d beta~/dq, Y_lm, grad Y_lm, for one channel at v = k+G.
struct ProjEval {
  double beta;       // beta~(q) Y_lm  (phase-free)
  double grad[3];    // d(beta~ Y)/dv
};

__device__ __forceinline__ ProjEval proj_eval(const GeoParams &gp, int c, double vx, double vy,
                                              double vz) {
  const double r2 = vx * vx + vy * vy + vz * vz;
  const bool pos = r2 > 1e-30;
  const double q = pos ? sqrt(r2) : 0.0;        // safe_norm (basis.py:170-179)
  const double rs = pos ? q : 1.0;
  const int ib = gp.ch_rad[c], l = gp.ch_l[c], m = gp.ch_m[c];
  double bq, dbq;
  if (gp.kind == 1) {
    radial_eval(gp.rt, ib, q, bq, dbq);                           // psp.py:130-138
  } else {
    // beta(q) = w q^l exp(-(q b)^2/2), q clamped at 1e-12 (psp.py:122-128);
    // d beta/dq = w exp(..) (l q^(l-1) - q^(l+1) b^2), zero below the clamp
    const double w = gp.w[ib], bb = gp.b[ib];
    const double qq = fmax(q, 1e-12);
    const double e = exp(-0.5 * (qq * bb) * (qq * bb));
    const double qlm1 = l == 0 ? 0.0 : (l == 1 ? 1.0 : qq);       // q^(l-1) for l >= 1
    const double ql = l == 0 ? 1.0 : qlm1 * qq;
    bq = w * ql * e;
    dbq = (q > 1e-12) ? w * e * ((double)l * qlm1 - ql * qq * bb * bb) : 0.0;
  }
  ProjEval out;
  const double c0 = 0.28209479177387814347;   // 1/sqrt(4 pi)
  const double c1 = 0.48860251190291992159;   // sqrt(3/(4 pi))
  const double u[3] = {pos ? vx / rs : 0.0, pos ? vy / rs : 0.0, pos ? vz / rs : 0.0};
  double Y, dY[3] = {0.0, 0.0, 0.0};
  if (l == 0) {
    Y = c0;
  } else if (l == 1) {
    // m = 0: +z, 1: -x, 2: -y  (ABACUS order, ylm.py:15-25)
    const int comp = m == 0 ? 2 : (m == 1 ? 0 : 1);
    const double sgn = m == 0 ? 1.0 : -1.0;
    Y = sgn * c1 * (comp == 0 ? vx : (comp == 1 ? vy : vz)) / rs;
    if (pos) {
      for (int a = 0; a < 3; ++a) dY[a] = sgn * c1 * ((a == comp ? 1.0 : 0.0) - u[comp] * u[a]) / rs;
    }
  } else {
    // l = 2, m = 0, +1, -1, +2, -2 (ylm.py:18-25): Y = P(v) / r^2 with P a quadratic
    // form, dY/dv = grad P / r^2 - 2 P v / r^4
    const double c20 = 0.31539156525252000603;   // sqrt(5/(4 pi)) / 2
    const double c21 = 1.09254843059207907054;   // sqrt(15/(4 pi))
    const double c22 = 0.54627421529603953527;   // sqrt(15/(16 pi))
    const double r2 = rs * rs;
    double P, dP[3];
    switch (m) {
      case 0: P = c20 * (2.0 * vz * vz - vx * vx - vy * vy);
              dP[0] = -2.0 * c20 * vx; dP[1] = -2.0 * c20 * vy; dP[2] = 4.0 * c20 * vz; break;
      case 1: P = -c21 * vx * vz; dP[0] = -c21 * vz; dP[1] = 0.0; dP[2] = -c21 * vx; break;
      case 2: P = -c21 * vy * vz; dP[0] = 0.0; dP[1] = -c21 * vz; dP[2] = -c21 * vy; break;
      case 3: P = c22 * (vx * vx - vy * vy); dP[0] = 2.0 * c22 * vx; dP[1] = -2.0 * c22 * vy; dP[2] = 0.0; break;
      default: P = c21 * vx * vy; dP[0] = c21 * vy; dP[1] = c21 * vx; dP[2] = 0.0; break;
    }
    Y = P / r2;
    if (pos) {
      const double v3[3] = {vx, vy, vz};
      for (int a = 0; a < 3; ++a) dY[a] = dP[a] / r2 - 2.0 * P * v3[a] / (r2 * r2);
    }
  }
  out.beta = bq * Y;
  for (int a = 0; a < 3; ++a) out.grad[a] = dbq * u[a] * Y + bq * dY[a];
  return out;
}

__device__ __forceinline__ void kg_vec(const PlanDev &pd, const GeoParams &gp, int g, int k, double *G, double *v) {
  const double m1 = pd.miller[3 * g], m2 = pd.miller[3 * g + 1], m3 = pd.miller[3 * g + 2];
  for (int a = 0; a < 3; ++a) {
    G[a] = m1 * gp.B[a] + m2 * gp.B[3 + a] + m3 * gp.B[6 + a];
    v[a] = G[a] + gp.kpt[3 * k + a];
  }
}

// b_a . R / 2 pi of the atoms, for phases e^{-2 pi i m frac}: a parameter of its own (12 KB) that only the kernels
// with tables take
struct Fracs { Turns f[kMaxAtoms * 3]; };
struct NoFracs {};
template <int FORM>
using FracsOf = std::conditional_t<FORM == 0, NoFracs, Fracs>;

template <int FORM>
FracsOf<FORM> make_fracs(const GeoParams &gp) {
  FracsOf<FORM> fr;
  if constexpr (FORM != 0) {
    memset(&fr, 0, sizeof(fr));
    for (int i = 0; i < gp.nat; ++i)
      for (int a = 0; a < 3; ++a) fr.f[3 * i + a] = phase_turns(gp.B + 3 * a, gp.pos + 3 * i);
  }
  return fr;
}

// The phases e^{-i(k+G).R} of one atom, from tables in shared memory: with G = sum_a m_a b_a they
// are e12[m1, m2] e3[m3], e12 holding e^{-ik.R} too, so a phase costs one complex product where
// its sincos costs some 60 FP64 instructions (GB300 issues under two per SM and cycle).
// Entries e^{-2 pi i m f} come from sincospi, which reduces its argument exactly (phase_exp).
struct PhaseTab {
  double2 *e1, *e2, *e3, *e12;   // e12 == nullptr: no room for the products, e1 e2 instead
  int M1, M2, M3;
};

__host__ __device__ inline size_t phase_small(const PlanDev &pd) {   // entries of e1, e2, e3
  return 2 * ((size_t)pd.mmax[0] + pd.mmax[1] + pd.mmax[2]) + 3;
}
__host__ __device__ inline size_t phase_pairs(const PlanDev &pd) {
  return (2 * (size_t)pd.mmax[0] + 1) * (2 * (size_t)pd.mmax[1] + 1);
}
// Shared-memory forms: 2 = with e12 (up to 64 KB, three CTAs per SM), 1 = e1, e2, e3 only,
// 0 = a sincos per phase: shells with few G per table entry (building the tables then takes longer
// than the phases; nG below about 800), and Miller indices far outside a box, which the plan wraps.
constexpr size_t kPhaseBytes = 64 << 10;
inline int phase_form(const PlanDev &pd, size_t &bytes) {
  const size_t small = phase_small(pd) * sizeof(double2), all = small + phase_pairs(pd) * sizeof(double2);
  if ((size_t)pd.nG < 16 * phase_small(pd)) { bytes = 0; return 0; }
  if (all <= kPhaseBytes) { bytes = all; return 2; }
  if (small <= kPhaseBytes) { bytes = small; return 1; }
  bytes = 0;
  return 0;
}

template <int FORM>
__device__ __forceinline__ PhaseTab phase_build(const PlanDev &pd, const GeoParams &gp, const FracsOf<FORM> &fr, int i,
                                                int k, double2 *sm) {
  PhaseTab t;
  if constexpr (FORM != 0) {
    t.M1 = pd.mmax[0];
    t.M2 = pd.mmax[1];
    t.M3 = pd.mmax[2];
    t.e1 = sm;
    t.e2 = t.e1 + 2 * t.M1 + 1;
    t.e3 = t.e2 + 2 * t.M2 + 1;
    t.e12 = FORM == 2 ? t.e3 + 2 * t.M3 + 1 : nullptr;
    const int n1 = 2 * t.M1 + 1, n2 = 2 * t.M2 + 1, n3 = 2 * t.M3 + 1;
    const double kr = gp.kpt[3 * k] * gp.pos[3 * i] + gp.kpt[3 * k + 1] * gp.pos[3 * i + 1] +
                      gp.kpt[3 * k + 2] * gp.pos[3 * i + 2];
    for (int t0 = threadIdx.x; t0 < n1 + n2 + n3; t0 += blockDim.x) {
      const int ax = t0 < n1 ? 0 : (t0 < n1 + n2 ? 1 : 2);
      const int m = ax == 0 ? t0 - t.M1 : (ax == 1 ? t0 - n1 - t.M2 : t0 - n1 - n2 - t.M3);
      double2 e = phase_exp(m, fr.f[3 * i + ax]);
      if (ax == 0 && kr != 0.0) {
        double sn, cs;
        sincos(kr, &sn, &cs);
        e = cmul(e, make_double2(cs, -sn));
      }
      sm[t0] = e;
    }
    __syncthreads();
    if (FORM == 2) {
      for (int p = threadIdx.x; p < n1 * n2; p += blockDim.x) t.e12[p] = cmul(t.e1[p / n2], t.e2[p % n2]);
      __syncthreads();
    }
  }
  return t;
}

// e^{-i v.R_i} at G index g (v = k + G)
template <int FORM>
__device__ __forceinline__ double2 phase_at(const PlanDev &pd, const GeoParams &gp, const PhaseTab &t, int i, int k,
                                            int g) {
  if (FORM == 0) {
    double G[3], v[3], sn, cs;
    kg_vec(pd, gp, g, k, G, v);
    sincos(v[0] * gp.pos[3 * i] + v[1] * gp.pos[3 * i + 1] + v[2] * gp.pos[3 * i + 2], &sn, &cs);
    return make_double2(cs, -sn);
  }
  const int m1 = pd.miller[3 * g] + t.M1, m2 = pd.miller[3 * g + 1] + t.M2, m3 = pd.miller[3 * g + 2] + t.M3;
  const double2 a = FORM == 2 ? t.e12[m1 * (2 * t.M2 + 1) + m2] : cmul(t.e1[m1], t.e2[m2]);
  return cmul(a, t.e3[m3]);
}

// Projectors of few atoms, in one launch: a thread evaluates form factor and phase of its (p, g).  Up to
// kDirectProj of them (k points x projectors x G), 35 to 50 us a call from Python against 45 to 58 for the three
// launches with tables: 8 k points of 2 atoms, 925 G, 39 / 55; one of 16 atoms, 3,071 G, 43 / 59; 236,800
// 49 / 57; beyond, 263,000 52 / 50 to 55, 393,000 72 / 56 to 66, 786,000 136 / 58.
template <typename R>
__global__ void __launch_bounds__(128) k_proj_direct(PlanDev pd, GeoParams gp, typename Cx<R>::T *__restrict__ proj) {
  using C = typename Cx<R>::T;
  const int g = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y, k = blockIdx.z;
  if (g >= pd.nG) return;
  const int i = p / gp.nh, c = p - i * gp.nh;
  double G[3], v[3], sn, cs;
  kg_vec(pd, gp, g, k, G, v);
  const double a = proj_eval(gp, c, v[0], v[1], v[2]).beta * gp.inv_sqrt_omega;
  sincos(v[0] * gp.pos[3 * i] + v[1] * gp.pos[3 * i + 1] + v[2] * gp.pos[3 * i + 2], &sn, &cs);
  C o;
  o.x = (R)(a * cs);
  o.y = (R)(-a * sn);   // e^{-i v.R}
  proj[((size_t)k * gridDim.y + p) * pd.nG + g] = o;
}
constexpr double kDirectProj = 3e5;

// beta~_c(|k+G|) Y_lm(k+G) / sqrt(omega) of every channel, once per G instead of once per atom and
// G: as doubles in the rows of the last atom of proj (8 or 16 bytes per element), which
// k_projectors turns into that atom's projectors in its last launch.
template <typename R>
__global__ void __launch_bounds__(128)
k_proj_forms(PlanDev pd, GeoParams gp, typename Cx<R>::T *__restrict__ proj) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (g >= pd.nG) return;
  double G[3], v[3];
  kg_vec(pd, gp, g, k, G, v);
  auto *last = proj + ((size_t)k * gp.nat + gp.nat - 1) * gp.nh * pd.nG;
  for (int c = 0; c < gp.nh; ++c)
    *reinterpret_cast<double *>(last + (size_t)c * pd.nG + g) = proj_eval(gp, c, v[0], v[1], v[2]).beta * gp.inv_sqrt_omega;
}

// proj[k][p][g], p = atom * nh + channel: the channels' form factors (k_proj_forms) times the
// atom's phase.  A CTA takes one atom (i0 + blockIdx.y) and `per` G.  Bound by the FP64 pipe, 12
// instructions per atom and G and the store of 16 nh bytes; evaluating form factor and sincos for
// every (p, G) took 1,038 us for 256 projectors x 23,847 G, 70 us so.
template <typename R, int FORM>
__global__ void __launch_bounds__(256)
k_projectors(PlanDev pd, GeoParams gp, FracsOf<FORM> fr, int i0, int per, typename Cx<R>::T *__restrict__ proj) {
  using C = typename Cx<R>::T;
  extern __shared__ __align__(16) double2 ph_smem[];
  const int i = i0 + blockIdx.y, k = blockIdx.z;
  const PhaseTab t = phase_build<FORM>(pd, gp, fr, i, k, ph_smem);
  const C *form = proj + ((size_t)k * gp.nat + gp.nat - 1) * gp.nh * pd.nG;
  C *out = proj + ((size_t)k * gp.nat + i) * gp.nh * pd.nG;
  const int g1 = min(pd.nG, (int)(blockIdx.x + 1) * per);
  for (int g = blockIdx.x * per + threadIdx.x; g < g1; g += 256) {
    const double2 p = phase_at<FORM>(pd, gp, t, i, k, g);
    for (int c = 0; c < gp.nh; ++c) {
      const double f = *reinterpret_cast<const double *>(form + (size_t)c * pd.nG + g);
      C o;
      o.x = (R)(f * p.x);
      o.y = (R)(f * p.y);
      out[(size_t)c * pd.nG + g] = o;
    }
  }
}

// kinetic diagonal 1/2 |k+G|^2
template <typename R>
__global__ void k_kinetic(PlanDev pd, GeoParams gp, R *__restrict__ kin) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (g >= pd.nG) return;
  const double m1 = pd.miller[3 * g], m2 = pd.miller[3 * g + 1], m3 = pd.miller[3 * g + 2];
  const double vx = m1 * gp.B[0] + m2 * gp.B[3] + m3 * gp.B[6] + gp.kpt[3 * k];
  const double vy = m1 * gp.B[1] + m2 * gp.B[4] + m3 * gp.B[7] + gp.kpt[3 * k + 1];
  const double vz = m1 * gp.B[2] + m2 * gp.B[5] + m3 * gp.B[8] + gp.kpt[3 * k + 2];
  kin[(size_t)k * pd.nG + g] = (R)(0.5 * (vx * vx + vy * vy + vz * vz));
}

// ---------------------------------------------------------------------------
// becp[k][p][b] = sum_g conj(proj[k][p][g]) psi[k][b][g]
//   CTA tile 32 (p) x 64 (b) over one G chunk (split-K); 256 threads, each
//   2 p x 4 b outputs (p = tp + 16 i, b = tb + 16 j: conflict-free smem reads)
// ---------------------------------------------------------------------------
constexpr int kBP = 32, kBB = 64, kBK = 16;

template <typename R>
__global__ void __launch_bounds__(256)
k_becp(const typename Cx<R>::T *__restrict__ proj, const typename Cx<R>::T *__restrict__ psi,
       int nb, int nG, int nproj, int nsplit, int gchunk, typename Cx<R>::T *__restrict__ out) {
  using C = typename Cx<R>::T;
  __shared__ __align__(16) C sP[2][kBP][kBK + 1];
  __shared__ __align__(16) C sX[2][kBB][kBK + 1];
  const int p0 = blockIdx.y * kBP, b0 = blockIdx.x * kBB;
  const int nkz = gridDim.z / nsplit;
  const int k = blockIdx.z / nsplit, sp = blockIdx.z - k * nsplit;
  const int ga = sp * gchunk, gb = min(nG, ga + gchunk);
  const C *Pk = proj + (size_t)k * nproj * nG;
  const C *Xk = psi + (size_t)k * nb * nG;
  const int tb = threadIdx.x & 15, tp = threadIdx.x >> 4;
  C acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = czero<C>();
  // 2-stage cp.async pipeline over G steps of kBK
  auto issue = [&](int g0, int buf) {
    for (int i = threadIdx.x; i < (kBP + kBB) * kBK; i += 256) {
      const int r = i / kBK, c = i - r * kBK;
      const int g = g0 + c;
      if (r < kBP) {
        const bool ok = p0 + r < nproj && g < gb;
        cp_async_el(&sP[buf][r][c], ok ? Pk + (size_t)(p0 + r) * nG + g : Pk, ok);
      } else {
        const int rr = r - kBP;
        const bool ok = b0 + rr < nb && g < gb;
        cp_async_el(&sX[buf][rr][c], ok ? Xk + (size_t)(b0 + rr) * nG + g : Xk, ok);
      }
    }
    cp_async_commit();
  };
  int buf = 0;
  if (ga < gb) issue(ga, 0);
  for (int g0 = ga; g0 < gb; g0 += kBK) {
    if (g0 + kBK < gb) {
      issue(g0 + kBK, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll 4
    for (int c = 0; c < kBK; ++c) {
      C av[2], xv[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) av[i] = sP[buf][tp + 16 * i][c];
#pragma unroll
      for (int j = 0; j < 4; ++j) xv[j] = sX[buf][tb + 16 * j][c];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // conj(a) * x
          acc[i][j].x += av[i].x * xv[j].x + av[i].y * xv[j].y;
          acc[i][j].y += av[i].x * xv[j].y - av[i].y * xv[j].x;
        }
    }
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int p = p0 + tp + 16 * i;
    if (p >= nproj) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int bb = b0 + tb + 16 * j;
      if (bb < nb) out[(((size_t)sp * nkz + k) * nproj + p) * nb + bb] = acc[i][j];
    }
  }
}

// Deterministic two-pass sum over splits, out[i] = sum_s part[s][i]:
//   pass 1 (grid: outputs / 256 x split groups) sums groups of kSplitGroup splits,
//   pass 2 (8 lanes per output) sums the groups: lane l takes groups l, l + 8, ...,
//   then a fixed xor-shuffle tree; every load is coalesced along i.
constexpr int kSplitGroup = 16;
constexpr int kSumLanes = 8;

template <typename C>
__global__ void __launch_bounds__(256) k_sum_splits1(const C *__restrict__ part, int nsplit, size_t n,
                                                     C *__restrict__ tmp) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j0 = blockIdx.y * kSplitGroup, j1 = min(nsplit, j0 + kSplitGroup);
  C s = czero<C>();
  for (int j = j0; j < j1; ++j) s = cadd(s, part[(size_t)j * n + i]);
  tmp[(size_t)blockIdx.y * n + i] = s;
}

template <typename C>
__global__ void __launch_bounds__(256) k_sum_splits2(const C *__restrict__ tmp, int ngroup, size_t n,
                                                     C *__restrict__ out) {
  const size_t i = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) / kSumLanes;
  const int l = threadIdx.x % kSumLanes;
  C s = czero<C>();
  if (i < n)
    for (int g = l; g < ngroup; g += kSumLanes) s = cadd(s, tmp[(size_t)g * n + i]);
#pragma unroll
  for (int o = kSumLanes / 2; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  if (i < n && l == 0) out[i] = s;
}

inline int split_groups(int ns) { return (ns + kSplitGroup - 1) / kSplitGroup; }

// DB[k][p][b] = sum_q D[p][q] becp[k][q][b]   (optionally scaled by wocc[k][b])
// A CTA takes one row p of D (nonzero in one atom's block of nh^2 at most): it lists the row's
// nonzeros in order, then its threads walk the bands over that list only.  Reading every D[p][q]
// per output cost 113 us at P = 256, 160 bands (FP64).
constexpr int kDList = 1024;

template <typename R>
__global__ void __launch_bounds__(128)
k_dbecp(const R *__restrict__ D, const typename Cx<R>::T *__restrict__ becp, int nproj, int nb,
        const double *__restrict__ wocc, typename Cx<R>::T *__restrict__ out) {
  using C = typename Cx<R>::T;
  __shared__ int qs[kDList];
  __shared__ R ds[kDList];
  __shared__ int wcnt[4];
  const int p = blockIdx.x, k = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const C *Bk = becp + (size_t)k * nproj * nb;
  C *o = out + ((size_t)k * nproj + p) * nb;
  for (int q0 = 0; q0 < nproj; q0 += kDList) {
    const int q1 = min(nproj, q0 + kDList);
    int cnt = 0;
    for (int c0 = q0; c0 < q1; c0 += 128) {
      const int q = c0 + threadIdx.x;
      const R d = q < q1 ? D[(size_t)p * nproj + q] : (R)0;
      const bool nz = d != (R)0;
      const unsigned m = __ballot_sync(0xffffffffu, nz);
      if (lane == 0) wcnt[warp] = __popc(m);
      __syncthreads();
      int at = cnt;
      for (int w = 0; w < warp; ++w) at += wcnt[w];
      if (nz) {
        const int i = at + __popc(m & ((1u << lane) - 1));
        qs[i] = q;
        ds[i] = d;
      }
      cnt += wcnt[0] + wcnt[1] + wcnt[2] + wcnt[3];
      __syncthreads();
    }
    for (int b = threadIdx.x; b < nb; b += 128) {
      C s = q0 ? o[b] : czero<C>();
      for (int i = 0; i < cnt; ++i) s = cadd(s, cscale(Bk[(size_t)qs[i] * nb + b], ds[i]));
      if (wocc && q1 == nproj) s = cscale(s, (R)wocc[(size_t)k * nb + b]);
      o[b] = s;
    }
    __syncthreads();
  }
}

// out[k][i][g] (+)= sum_j X[k][j, i] op(A[k][j][g]);  X element (j, i) at j*xs_j + i*xs_i
// CTA tile: TG g x 32 i, j in steps of 16 (cp.async double buffer); 256 threads;
// TG = 128: each thread 4 g (lane + 32 u) x 4 i (warp * 4 + v); TG = 32: 1 g x 4 i.
constexpr int kAI = 32, kAJ = 16;

template <typename R, bool CONJ_A, bool ACCUM, int TG>
__global__ void __launch_bounds__(256)
k_apply(const typename Cx<R>::T *__restrict__ Xm, int xs_j, int xs_i, size_t xs_k,
        const typename Cx<R>::T *__restrict__ A, size_t as_k, int nj, int ni, int nG,
        typename Cx<R>::T *__restrict__ out, size_t os_k) {
  using C = typename Cx<R>::T;
  constexpr int U = TG / 32;
  __shared__ __align__(16) C sA[2][kAJ][TG];
  __shared__ __align__(16) C sX[2][kAJ][kAI];
  const int g0 = blockIdx.x * TG, i0 = blockIdx.y * kAI, k = blockIdx.z;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const C *Ak = A + (size_t)k * as_k;
  const C *Xk = Xm + (size_t)k * xs_k;
  C acc[U][4];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = czero<C>();
  auto issue = [&](int j0, int buf) {
    for (int t = threadIdx.x; t < kAJ * TG; t += 256) {
      const int r = t / TG, c = t - r * TG;
      const bool ok = j0 + r < nj && g0 + c < nG;
      cp_async_el(&sA[buf][r][c], ok ? Ak + (size_t)(j0 + r) * nG + g0 + c : Ak, ok);
    }
    for (int t = threadIdx.x; t < kAJ * kAI; t += 256) {
      const int r = t / kAI, c = t - r * kAI;
      const bool ok = j0 + r < nj && i0 + c < ni;
      cp_async_el(&sX[buf][r][c], ok ? Xk + (size_t)(j0 + r) * xs_j + (size_t)(i0 + c) * xs_i : Xk, ok);
    }
    cp_async_commit();
  };
  int buf = 0;
  issue(0, 0);
  for (int j0 = 0; j0 < nj; j0 += kAJ) {
    if (j0 + kAJ < nj) {
      issue(j0 + kAJ, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < kAJ; ++r) {
      C av[U], xv[4];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        av[u] = sA[buf][r][lane + 32 * u];
        if (CONJ_A) av[u].y = -av[u].y;
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) xv[v] = sX[buf][r][w * 4 + v];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          acc[u][v].x += av[u].x * xv[v].x - av[u].y * xv[v].y;
          acc[u][v].y += av[u].x * xv[v].y + av[u].y * xv[v].x;
        }
    }
    __syncthreads();
    buf ^= 1;
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const int i = i0 + w * 4 + v;
    if (i >= ni) continue;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int g = g0 + lane + 32 * u;
      if (g < nG) {
        C *o = out + (size_t)k * os_k + (size_t)i * nG + g;
        *o = ACCUM ? cadd(*o, acc[u][v]) : acc[u][v];
      }
    }
  }
}

// E_NL partial per (k, b): wocc * Re(B^H D B); writes partial[k*nb + b].  32 bands per CTA, its
// eight rows of threads share the projectors (one thread per band took 128 us at 160 x 256).
template <typename R>
__global__ void __launch_bounds__(256)
k_nl_energy(const typename Cx<R>::T *__restrict__ becp, const typename Cx<R>::T *__restrict__ dbecp, int nproj, int nb,
            const double *__restrict__ wocc, double *__restrict__ out) {
  __shared__ double red[8][33];
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5, b = blockIdx.x * 32 + lane, k = blockIdx.y;
  double s = 0.0;
  if (b < nb)
    for (int p = row; p < nproj; p += 8) {
      const auto x = becp[((size_t)k * nproj + p) * nb + b];
      const auto y = dbecp[((size_t)k * nproj + p) * nb + b];
      s += (double)x.x * (double)y.x + (double)x.y * (double)y.y;
    }
  red[row][lane] = s;
  __syncthreads();
  if (row == 0 && b < nb) {
    for (int r = 1; r < 8; ++r) s += red[r][lane];
    out[(size_t)k * nb + b] = wocc[(size_t)k * nb + b] * s;
  }
}

template <typename R>
addft_status nl_energy_t(const void *becp, const void *dbecp, int nk, int nproj, int nb, const double *wocc, double *out,
                         cudaStream_t st) {
  using C = typename Cx<R>::T;
  k_nl_energy<R><<<dim3((nb + 31) / 32, nk), 256, 0, st>>>((const C *)becp, (const C *)dbecp, nproj, nb, wocc, out);
  return check_launch("k_nl_energy");
}

// Envelope gradients of E_NL from Y[k][p][g] = sum_b wocc (D B)[p][b] conj(psi_b(g)):
//   dE/dR_{i,a} = sum_{p in i} sum_g 2 v_a Im(beta_p y)
//   dE/deps_ab  = -2 sum_p sum_g Re(Q_pa y) G_b            (the -E_NL delta_ab term is added later)
// A CTA takes one atom, one k and one of nsplit ranges of g; partial[((k nat + i) nsplit + s) * 12 + j].
// Channels are summed before the v and G factors are applied, and phases come from the tables above
// (form[k][c][4][g]: beta and its gradient per channel, shared by the atoms, or nullptr: evaluated
// here).  One CTA per (k, p) with a sincos and a form factor per (p, g) took 2,796 us on Si64, 190 us so.
template <typename R>
__global__ void __launch_bounds__(128)
k_nl_forms(PlanDev pd, GeoParams gp, double *__restrict__ form) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
  if (g >= pd.nG) return;
  double G[3], v[3];
  kg_vec(pd, gp, g, k, G, v);
  double *f = form + (size_t)k * gp.nh * 4 * pd.nG + g;
  for (int c = 0; c < gp.nh; ++c) {
    const ProjEval e = proj_eval(gp, c, v[0], v[1], v[2]);
    f[(size_t)(4 * c) * pd.nG] = e.beta;
    for (int a = 0; a < 3; ++a) f[(size_t)(4 * c + 1 + a) * pd.nG] = e.grad[a];
  }
}

template <typename R, int FORM>
__global__ void __launch_bounds__(256, 2)
k_nl_grad(PlanDev pd, GeoParams gp, FracsOf<FORM> fr, const typename Cx<R>::T *__restrict__ Y, const double *__restrict__ form,
          int nsplit, double *__restrict__ partial) {
  extern __shared__ __align__(16) double2 ph_smem[];
  const int i = blockIdx.x, sp = blockIdx.y, k = blockIdx.z;
  const PhaseTab t = phase_build<FORM>(pd, gp, fr, i, k, ph_smem);
  const auto *Yi = Y + ((size_t)k * gp.nat + i) * gp.nh * pd.nG;
  const double *fk = form ? form + (size_t)k * gp.nh * 4 * pd.nG : nullptr;
  const int per = (pd.nG + nsplit - 1) / nsplit;
  const int ga = sp * per, gb = min(pd.nG, ga + per);
  double acc[12];
#pragma unroll
  for (int j = 0; j < 12; ++j) acc[j] = 0.0;
  for (int g = ga + threadIdx.x; g < gb; g += blockDim.x) {
    double G[3], v[3];
    kg_vec(pd, gp, g, k, G, v);
    const double2 p = phase_at<FORM>(pd, gp, t, i, k, g);
    double s = 0.0, r[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < gp.nh; ++c) {
      const auto yv = Yi[(size_t)c * pd.nG + g];
      const double yr = yv.x, yi = yv.y;
      const double pr = p.x * yr - p.y * yi, pim = p.x * yi + p.y * yr;   // phase * y
      double b, gr[3];
      if (fk) {
        b = fk[(size_t)(4 * c) * pd.nG + g];
        for (int a = 0; a < 3; ++a) gr[a] = fk[(size_t)(4 * c + 1 + a) * pd.nG + g];
      } else {
        const ProjEval e = proj_eval(gp, c, v[0], v[1], v[2]);
        b = e.beta;
        for (int a = 0; a < 3; ++a) gr[a] = e.grad[a];
      }
      s += b * pim;
#pragma unroll
      for (int a = 0; a < 3; ++a) r[a] += gr[a] * pr;
    }
    s *= 2.0 * gp.inv_sqrt_omega;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      acc[a] += v[a] * s;
      const double ra = -2.0 * gp.inv_sqrt_omega * r[a];
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[3 + 3 * a + b] += ra * G[b];
    }
  }
  // block reduce 12 values
  __shared__ double red[8][12];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 12; ++j) {
    double x = acc[j];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][j] = x;
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) s += red[w][threadIdx.x];
    partial[(((size_t)k * gp.nat + i) * nsplit + sp) * 12 + threadIdx.x] = s;
  }
}

// out: [0] E_NL, [1..3nat] dE/dR, [1+3nat..] dE/deps (9); a warp per output
__global__ void __launch_bounds__(128)
k_nl_grad_final(const double *__restrict__ epart, int nkb, const double *__restrict__ gpart, int nk, int nat,
                int nsplit, double *__restrict__ out) {
  const int lane = threadIdx.x & 31, t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= 1 + 3 * nat + 9) return;
  auto warp_sum = [&](double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  double s = 0.0;
  if (t >= 1 && t < 1 + 3 * nat) {
    const int i = (t - 1) / 3, a = (t - 1) % 3;
    for (int q = lane; q < nk * nsplit; q += 32)
      s += gpart[(((size_t)(q / nsplit) * nat + i) * nsplit + q % nsplit) * 12 + a];
    s = warp_sum(s);
  } else {
    const int ab = t - 1 - 3 * nat;
    double e = 0.0;
    if (t == 0 || ab % 4 == 0)
      for (int q = lane; q < nkb; q += 32) e += epart[q];
    e = warp_sum(e);
    if (t > 0) {
      for (int q = lane; q < nk * nat * nsplit; q += 32) s += gpart[(size_t)q * 12 + 3 + ab];
      s = warp_sum(s);
      if (ab % 4 == 0) s -= e;
    } else {
      s = e;
    }
  }
  if (lane == 0) out[t] = s;
}

// kinetic stress partials: -sum wocc |psi|^2 (k+G)_a G_b
template <typename R>
__global__ void __launch_bounds__(256)
k_kin_stress(PlanDev pd, GeoParams gp, const typename Cx<R>::T *__restrict__ psi, int nb,
             const double *__restrict__ wocc, double *__restrict__ partial) {
  double acc[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) acc[j] = 0.0;
  const size_t total = (size_t)gp.nk * pd.nG;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total;
       t += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(t / pd.nG), g = (int)(t - (size_t)k * pd.nG);
    double p2 = 0.0;
    for (int b = 0; b < nb; ++b) {
      const auto x = psi[((size_t)k * nb + b) * pd.nG + g];
      p2 += wocc[(size_t)k * nb + b] * ((double)x.x * x.x + (double)x.y * x.y);
    }
    const double m1 = pd.miller[3 * g], m2 = pd.miller[3 * g + 1], m3 = pd.miller[3 * g + 2];
    const double G[3] = {m1 * gp.B[0] + m2 * gp.B[3] + m3 * gp.B[6],
                         m1 * gp.B[1] + m2 * gp.B[4] + m3 * gp.B[7],
                         m1 * gp.B[2] + m2 * gp.B[5] + m3 * gp.B[8]};
    const double v[3] = {G[0] + gp.kpt[3 * k], G[1] + gp.kpt[3 * k + 1], G[2] + gp.kpt[3 * k + 2]};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc[3 * a + b] -= p2 * v[a] * G[b];
  }
  block_reduce_store<9>(acc, partial);
}

// ---------------------------------------------------------------------------
// host drivers
// ---------------------------------------------------------------------------
inline int pick_nsplit(int tiles, int nG, int ctas_per_sm = 8) {
  if (tiles < 1) return 1;   // an empty problem, in a size query
  int ns = (ctas_per_sm * 152 + tiles - 1) / tiles;
  const int maxs = (nG + 63) / 64;
  if (ns > maxs) ns = maxs;
  if (ns < 1) ns = 1;
  return ns;
}

// becp_tc.cu: split-precision TF32 tensor-core becp (FP32), same grid and partial layout as k_becp;
// proj_simt.cu: register-tiled FP32 FMA becp, same layout
addft_status launch_becp_tc(int nk, int nb, int nG, int nproj, int nsplit, int gchunk, const float2 *proj,
                            const float2 *psi, float2 *out, cudaStream_t st);
addft_status launch_becp_f32(int nk, int nb, int nG, int nproj, int nsplit, int gchunk, const float2 *proj,
                             const float2 *psi, float2 *out, cudaStream_t st);
// tc05.cu: split-TF32 becp on tcgen05 with a tensor-memory accumulator, same partial layout, its tile
void becp_tc05_tile(int nb, int *pt, int *bt);
addft_status launch_becp_tc05(int nk, int nb, int nG, int nproj, int nsplit, const float2 *proj, const float2 *psi,
                              float2 *out, cudaStream_t st);

// Kernel of the FP32 projector contractions, read once per process from ADDFT_BECP_TC /
// ADDFT_APPLY_TC: 0 = register-tiled FP32 FMA, 1 = split-TF32 mma.sync tensor cores,
// 2 = the generic SIMT kernels of this file, 3 = split-TF32 tcgen05 with a tensor-memory
// accumulator (the default of both: the fastest and, its sums being taken out of the truncating
// accumulators every 32 G, the most accurate.  becp, 1 against 3: 72^3 box, 64 bands x 32
// projectors 60 -> 38 us, Si64 168 x 256 234 -> 84, 8 k points of Si2 8.2 -> 5.5; rms error 9.7e-7 -> 2.4e-7,
// 3.3e-6 -> 2.6e-7, 3.0e-7 -> 1.9e-7).
static int proj_mode(const char *var, int dflt) {
  const char *v = getenv(var);
  const int m = v ? atoi(v) : dflt;
  return m >= 0 && m <= 3 ? m : dflt;
}
static int becp_mode() {
  static const int m = proj_mode("ADDFT_BECP_TC", 3);
  return m;
}

// K splits of the tcgen05 becp: the fewest waves of 32-G stages, each CTA about 6 stages' time on top.  For each
// number of waves up to two the splits that fill them, as few as give the same stages per CTA.
static int becp_tc05_nsplit(int tiles, int nG) {
  const int steps = (nG + 31) / 32;
  int best = 1;
  long least = ((long)tiles + 151) / 152 * (steps + 6);
  for (int w = 1; w <= 2; ++w) {
    const int most = std::min(steps, 152 * w / tiles);
    if (most < 1) continue;
    const int per = (steps + most - 1) / most, ns = (steps + per - 1) / per;
    const long t = ((long)tiles * ns + 151) / 152 * (per + 6);
    if (t < least) {
      least = t;
      best = ns;
    }
  }
  return best;
}

// CTAs per SM of split-K work for the tensor-core and register-tiled becp kernels
// (ADDFT_BECP_CTAS, 1..8, read once per process; default 4).
static int becp_ctas_per_sm() {
  static const int m = [] {
    const char *v = getenv("ADDFT_BECP_CTAS");
    const int x = v ? atoi(v) : 4;
    return x >= 1 && x <= 8 ? x : 4;
  }();
  return m;
}

// partial sums of the split-K kernels at their default number of splits
template <typename R>
size_t becp_partial_bytes(int nk, int nb, int nG, int nproj) {
  using C = typename Cx<R>::T;
  const int tiles = ((nproj + kBP - 1) / kBP) * ((nb + kBB - 1) / kBB) * nk;
  const int ns = pick_nsplit(tiles, nG);
  return ns > 1 ? (size_t)(ns + split_groups(ns)) * nk * nproj * nb * sizeof(C) : 0;
}

template <typename R>
size_t becp_work_bytes(int nk, int nb, int nG, int nproj) {
  const size_t least = becp_partial_bytes<R>(nk, nb, nG, nproj);
  return sizeof(R) == 8 ? std::max(least, oz_work_bytes(8, nproj, nb, nG, nk)) : least;
}

template <typename R>
addft_status becp_t(int nk, int nb, int nG, int nproj, const void *proj, const void *psi, void *becp,
                    void *work, size_t bytes, cudaStream_t st) {
  using C = typename Cx<R>::T;
  if constexpr (sizeof(R) == 8) {
    if (oz_fits(8, nproj, nb, nG, nk, work, bytes)) {
      const OzMat b = {proj, nG, 1, (size_t)nproj * nG, 1}, x = {psi, nG, 1, (size_t)nb * nG, 0};
      return oz_gemm(8, nproj, nb, nG, nk, b, x, becp, nb, 1, (size_t)nproj * nb, false, work, bytes, st);
    }
  }
  const int tiles = ((nproj + kBP - 1) / kBP) * ((nb + kBB - 1) / kBB) * nk;
  const int mode = sizeof(R) == 4 ? becp_mode() : 2;
  const bool tc = mode == 1;
  // the tensor-core and register-tiled forms hold 2 / 4 CTAs per SM: 4 per SM of work keeps
  // 1-2 waves of long K chunks
  int ns = pick_nsplit(tiles, nG, mode != 2 ? becp_ctas_per_sm() : 8);
  if (mode == 3) {   // one CTA per SM
    int pt, bt;
    becp_tc05_tile(nb, &pt, &bt);
    ns = std::min(ns, becp_tc05_nsplit(((nproj + pt - 1) / pt) * ((nb + bt - 1) / bt) * nk, nG));
  }
  const size_t per = (size_t)nk * nproj * nb * sizeof(C);
  // partials (ns) + pass-1 group sums (ceil(ns / kSplitGroup)) must fit the work buffer
  while (ns > 1 && (work == nullptr || bytes < per * (size_t)(ns + split_groups(ns)))) --ns;
  if (ns < 1) ns = 1;
  int gchunk = (nG + ns - 1) / ns;
  if (tc) {   // whole 32-G stages per chunk; never more partials than the work buffer holds
    gchunk = (gchunk + 31) / 32 * 32;
    ns = (nG + gchunk - 1) / gchunk;
  }
  dim3 grid((nb + kBB - 1) / kBB, (nproj + kBP - 1) / kBP, nk * ns);
  C *dst = ns > 1 ? (C *)work : (C *)becp;
  bool done = false;
  if constexpr (sizeof(R) == 4) {
    if (mode == 1) {
      ADDFT_TRY(launch_becp_tc(nk, nb, nG, nproj, ns, gchunk, (const float2 *)proj, (const float2 *)psi,
                               (float2 *)dst, st));
      done = true;
    } else if (mode == 0) {
      ADDFT_TRY(launch_becp_f32(nk, nb, nG, nproj, ns, gchunk, (const float2 *)proj, (const float2 *)psi,
                                (float2 *)dst, st));
      done = true;
    } else if (mode == 3) {
      ADDFT_TRY(launch_becp_tc05(nk, nb, nG, nproj, ns, (const float2 *)proj, (const float2 *)psi, (float2 *)dst, st));
      done = true;
    }
  }
  if (!done) {
    k_becp<R><<<grid, 256, 0, st>>>((const C *)proj, (const C *)psi, nb, nG, nproj, ns, gchunk, dst);
    ADDFT_TRY(check_launch("k_becp"));
  }
  if (ns > 1) {
    const size_t n = (size_t)nk * nproj * nb;
    const int ng = split_groups(ns);
    C *tmp = dst + (size_t)ns * n;
    k_sum_splits1<C><<<dim3((unsigned)((n + 255) / 256), ng), 256, 0, st>>>(dst, ns, n, tmp);
    ADDFT_TRY(check_launch("k_sum_splits1"));
    k_sum_splits2<C><<<(unsigned)((n * kSumLanes + 255) / 256), 256, 0, st>>>(tmp, ng, n, (C *)becp);
    ADDFT_TRY(check_launch("k_sum_splits2"));
  }
  return ADDFT_OK;
}

template <typename R>
addft_status dbecp_t(const void *D, const void *becp, int nk, int nproj, int nb, const double *wocc,
                     void *out, cudaStream_t st) {
  using C = typename Cx<R>::T;
  k_dbecp<R><<<dim3(nproj, nk), 128, 0, st>>>((const R *)D, (const C *)becp, nproj, nb, wocc, (C *)out);
  return check_launch("k_dbecp");
}

// apply_tc.cu: split-precision TF32 tensor-core apply (FP32, no conjugation);
// proj_simt.cu: register-tiled FP32 FMA apply
addft_status launch_apply_tc(bool accum, const float2 *X, int xs_j, int xs_i, size_t xs_k, const float2 *A,
                             size_t as_k, int nk, int nj, int ni, int nG, float2 *out, size_t os_k,
                             cudaStream_t st);
addft_status launch_apply_f32(bool accum, const float2 *X, int xs_j, int xs_i, size_t xs_k, const float2 *A,
                              size_t as_k, int nk, int nj, int ni, int nG, float2 *out, size_t os_k,
                              cudaStream_t st);
// tc05.cu: split-TF32 apply on tcgen05 with a tensor-memory accumulator, the scratch it wants
addft_status launch_apply_tc05(bool accum, const float2 *X, int xs_j, int xs_i, size_t xs_k, const float2 *A,
                               size_t as_k, int nk, int nj, int ni, int nG, float2 *out, size_t os_k,
                               void *work, size_t bytes, cudaStream_t st);
size_t apply_tc05_bytes(int nk, int nj, int ni, int nG);

static int apply_mode() {
  static const int m = proj_mode("ADDFT_APPLY_TC", 3);
  return m;
}

// scratch (work, bytes) serves the FP64 tensor-core form, without enough of it the SIMT kernel runs, and the
// packed X of the FP32 one
template <typename R>
size_t apply_work_bytes(int nk, int nj, int ni, int nG) {
  return sizeof(R) == 8 ? oz_work_bytes(8, ni, nG, nj, nk) : apply_tc05_bytes(nk, nj, ni, nG);
}

template <typename R, bool CONJ_A, bool ACCUM>
addft_status apply_t(const void *X, int xs_j, int xs_i, size_t xs_k, const void *A, size_t as_k,
                     int nk, int nj, int ni, int nG, void *out, size_t os_k, void *work, size_t bytes,
                     cudaStream_t st) {
  using C = typename Cx<R>::T;
  if constexpr (sizeof(R) == 8) {
    if (oz_fits(8, ni, nG, nj, nk, work, bytes)) {
      const OzMat x = {X, xs_i, xs_j, xs_k, 0}, a = {A, 1, nG, as_k, CONJ_A ? 1 : 0};
      return oz_gemm(8, ni, nG, nj, nk, x, a, out, nG, 1, os_k, ACCUM, work, bytes, st);
    }
  }
  if constexpr (sizeof(R) == 4 && !CONJ_A) {
    if (apply_mode() == 1)
      return launch_apply_tc(ACCUM, (const float2 *)X, xs_j, xs_i, xs_k, (const float2 *)A, as_k, nk, nj, ni, nG,
                             (float2 *)out, os_k, st);
    if (apply_mode() == 0)
      return launch_apply_f32(ACCUM, (const float2 *)X, xs_j, xs_i, xs_k, (const float2 *)A, as_k, nk, nj, ni, nG,
                              (float2 *)out, os_k, st);
    if (apply_mode() == 3)
      return launch_apply_tc05(ACCUM, (const float2 *)X, xs_j, xs_i, xs_k, (const float2 *)A, as_k, nk, nj, ni, nG,
                               (float2 *)out, os_k, work, bytes, st);
  }
  const long ctas128 = (long)((nG + 127) / 128) * ((ni + kAI - 1) / kAI) * nk;
  if (ctas128 >= 4 * 152) {
    dim3 grid((nG + 127) / 128, (ni + kAI - 1) / kAI, nk);
    k_apply<R, CONJ_A, ACCUM, 128><<<grid, 256, 0, st>>>((const C *)X, xs_j, xs_i, xs_k, (const C *)A, as_k, nj,
                                                         ni, nG, (C *)out, os_k);
  } else {
    dim3 grid((nG + 31) / 32, (ni + kAI - 1) / kAI, nk);
    k_apply<R, CONJ_A, ACCUM, 32><<<grid, 256, 0, st>>>((const C *)X, xs_j, xs_i, xs_k, (const C *)A, as_k, nj,
                                                        ni, nG, (C *)out, os_k);
  }
  return check_launch("k_apply");
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// one region serves becp's partials and, after it, the apply's operands
template <typename R>
size_t nl_split_bytes(int nk, int nb, int nG, int nproj) {
  return std::max(becp_work_bytes<R>(nk, nb, nG, nproj), apply_work_bytes<R>(nk, nproj, nb, nG));
}

template <typename R>
size_t nl_scratch(int nk, int nb, int nG, int nproj) {
  using C = typename Cx<R>::T;
  if (nproj == 0) return 0;
  return align256(2 * (size_t)nk * nproj * nb * sizeof(C)) + align256(nl_split_bytes<R>(nk, nb, nG, nproj));
}

// the region shared by becp and the back-contraction Y of the gradients
inline size_t nl_grad_scratch(addft_dtype dt, int nk, int nb, int nG, int nproj) {
  return dt == ADDFT_F64
             ? std::max(becp_work_bytes<double>(nk, nb, nG, nproj), apply_work_bytes<double>(nk, nb, nproj, nG))
             : becp_work_bytes<float>(nk, nb, nG, nproj);
}

// H psi with the work buffer split as [becp | D becp | becp split-K partials | local FFT scratch].
// The local part needs at least one band of FFT scratch (addft_work_bytes(plan, 1)); becp gets what
// remains beyond that, up to what it asks for, and lowers the number of splits to fit (down to one, which
// needs no partials).
// The projector chain (becp, split sums, D becp) only reads psi and the beta tables and
// writes its own part of the work buffer, so it can run beside the local FFT pipeline.
// ADDFT_HPSI_OVERLAP (read once per process): 0 = one stream; 1 (default) = the chain on a
// second stream of the calling thread, forked from and joined back into the caller's stream
// with events (also inside a stream capture); 2 = the same with that stream at the highest
// priority.  72^3 microbench, 64 bands, with becp on mma.sync: 0.428 ms (0), 0.399 ms (1), 0.400 ms
// (2); with it on tcgen05 0.388 ms (1).
static int overlap_mode() {
  static const int m = [] {
    const char *v = getenv("ADDFT_HPSI_OVERLAP");
    const int x = v ? atoi(v) : 1;
    return x >= 0 && x <= 2 ? x : 1;
  }();
  return m;
}

// The calling thread's side stream on the current device (created on first use, kept).
static addft_status side_stream(int prio_mode, cudaStream_t *out) {
  constexpr int kDev = 64;
  static thread_local cudaStream_t side[kDev] = {};
  int dev = 0;
  ADDFT_CUDA(cudaGetDevice(&dev));
  ADDFT_REQUIRE(dev >= 0 && dev < kDev, ADDFT_UNSUPPORTED, "hpsi: device index %d >= %d", dev, kDev);
  if (side[dev] == nullptr) {
    int lo = 0, hi = 0;
    ADDFT_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    ADDFT_CUDA(cudaStreamCreateWithPriority(&side[dev], cudaStreamNonBlocking, prio_mode == 2 ? hi : lo));
  }
  *out = side[dev];
  return ADDFT_OK;
}

template <typename R>
addft_status hpsi_t(addft_plan plan, int nk, int nb, const void *psi, const void *kin, const void *v_r, int nproj,
                    const void *proj, const void *dion, void *hpsi, void *work, size_t work_bytes, cudaStream_t st,
                    bool allow_overlap) {
  using C = typename Cx<R>::T;
  const PlanDev &pd = plan->dev;
  const addft_dtype dt = sizeof(R) == 8 ? ADDFT_F64 : ADDFT_F32;
  const size_t arrays = nproj > 0 ? align256(2 * (size_t)nk * nproj * nb * sizeof(C)) : 0;
  const size_t local_min = work_bytes_min(pd, 1, sizeof(C));
  ADDFT_REQUIRE(work && work_bytes >= arrays + local_min, ADDFT_INVALID_ARG,
                "hpsi: work buffer of %zu B too small (need >= %zu B)", work_bytes, arrays + local_min);
  size_t split = 0;
  if (nproj > 0) {
    const size_t spare = (work_bytes - arrays - local_min) & ~size_t(255);
    split = align256(nl_split_bytes<R>(nk, nb, pd.nG, nproj));
    if (split > spare) {
      // Short of that: up to half of what is spare where the products of FP64 go in pieces of it, else the split
      // partials.  What a form would leave unused belongs to the transforms: their bands at once decide their time.
      const size_t half = std::min(align256(oz_work_bytes(8, nproj, nb, pd.nG, nk)), (spare / 2) & ~size_t(255));
      split = std::min(align256(becp_partial_bytes<R>(nk, nb, pd.nG, nproj)), spare);
      if (sizeof(R) == 8 && oz_fits(8, nproj, nb, pd.nG, nk, (char *)work + arrays, half)) split = std::max(split, half);
    }
  }
  C *becp = (C *)work;
  C *db = becp + (size_t)nk * nproj * nb;
  char *bw = (char *)work + arrays;
  const size_t used = arrays + split;
  if (nproj > 0 && allow_overlap && overlap_mode() != 0) {
    cudaStream_t side = nullptr;
    ADDFT_TRY(side_stream(overlap_mode(), &side));
    cudaEvent_t fork = nullptr, join = nullptr;
    ADDFT_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    cudaError_t e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      cudaEventDestroy(fork);
      ADDFT_CUDA(e);
    }
    // events are released once their work completes; destroying them here is safe
    struct Release {
      cudaEvent_t a, b;
      ~Release() { cudaEventDestroy(a); cudaEventDestroy(b); }
    } release{fork, join};
    ADDFT_CUDA(cudaEventRecord(fork, st));
    ADDFT_CUDA(cudaStreamWaitEvent(side, fork, 0));
    addft_status s = becp_t<R>(nk, nb, pd.nG, nproj, proj, psi, becp, split ? bw : nullptr, split, side);
    if (s == ADDFT_OK) s = dbecp_t<R>(dion, becp, nk, nproj, nb, nullptr, db, side);
    // join even after an error, so a stream capture is never left forked
    ADDFT_CUDA(cudaEventRecord(join, side));
    const addft_status sl = s == ADDFT_OK
                                ? hpsi_local_t<R>(plan, nk, nb, psi, kin, v_r, hpsi, (char *)work + used,
                                                  work_bytes - used, st)
                                : s;
    ADDFT_CUDA(cudaStreamWaitEvent(st, join, 0));
    ADDFT_TRY(sl);
    // the becp partials and the FFT scratch are free by now
    return apply_t<R, false, true>(db, nb, 1, (size_t)nproj * nb, proj, (size_t)nproj * pd.nG, nk, nproj, nb,
                                   pd.nG, hpsi, (size_t)nb * pd.nG, bw, work_bytes - arrays, st);
  }
  if (nproj > 0) {
    ADDFT_TRY(becp_t<R>(nk, nb, pd.nG, nproj, proj, psi, becp, split ? bw : nullptr, split, st));
    ADDFT_TRY(dbecp_t<R>(dion, becp, nk, nproj, nb, nullptr, db, st));
  }
  ADDFT_TRY(hpsi_local_t<R>(plan, nk, nb, psi, kin, v_r, hpsi, (char *)work + used, work_bytes - used, st));
  if (nproj > 0)
    ADDFT_TRY((apply_t<R, false, true>(db, nb, 1, (size_t)nproj * nb, proj, (size_t)nproj * pd.nG, nk, nproj, nb,
                                       pd.nG, hpsi, (size_t)nb * pd.nG, bw, work_bytes - arrays, st)));
  return ADDFT_OK;
}

template <typename R, int FORM>
addft_status projectors_form(const PlanDev &pd, const GeoParams &gp, size_t smem, typename Cx<R>::T *proj,
                             cudaStream_t st) {
  ADDFT_TRY(smem_optin(k_projectors<R, FORM>, smem));
  const auto fr = make_fracs<FORM>(gp);
  // about 4 CTAs per SM, each with enough G to pay for its phase tables
  auto go = [&](int i0, int n) {
    int chunks = (4 * 152 + n * gp.nk - 1) / (n * gp.nk);
    chunks = std::max(1, std::min(chunks, (pd.nG + 1023) / 1024));
    const int per = ((pd.nG + chunks - 1) / chunks + 255) / 256 * 256;
    k_projectors<R, FORM><<<dim3((pd.nG + per - 1) / per, n, gp.nk), 256, smem, st>>>(pd, gp, fr, i0, per, proj);
    return check_launch("k_projectors");
  };
  if (gp.nat > 1) ADDFT_TRY(go(0, gp.nat - 1));
  return go(gp.nat - 1, 1);   // in place, over the form factors
}

template <typename R>
addft_status projectors_t(const PlanDev &pd, const GeoParams &gp, void *proj, cudaStream_t st) {
  using C = typename Cx<R>::T;
  size_t smem = 0;
  const int form = phase_form(pd, smem);
  if (form == 0 || (double)gp.nk * gp.nat * gp.nh * pd.nG < kDirectProj) {
    k_proj_direct<R><<<dim3((pd.nG + 127) / 128, gp.nat * gp.nh, gp.nk), 128, 0, st>>>(pd, gp, (C *)proj);
    return check_launch("k_proj_direct");
  }
  k_proj_forms<R><<<dim3((pd.nG + 127) / 128, gp.nk), 128, 0, st>>>(pd, gp, (C *)proj);
  ADDFT_TRY(check_launch("k_proj_forms"));
  return form == 2 ? projectors_form<R, 2>(pd, gp, smem, (C *)proj, st) : projectors_form<R, 1>(pd, gp, smem, (C *)proj, st);
}

// splits of the gradients' G range per atom: about four CTAs per SM, at least 256 G each
inline int nl_grad_splits(int nk, int nat, int nG) {
  if (nk < 1 || nat < 1) return 1;
  return std::max(1, std::min((4 * 152 + nk * nat - 1) / (nk * nat), (nG + 255) / 256));
}

template <typename R>
addft_status nl_grad_t(const PlanDev &pd, const GeoParams &gp, const void *Y, void *scratch, size_t scratch_bytes,
                       int nsplit, double *part, cudaStream_t st) {
  using C = typename Cx<R>::T;
  // channel tables shared by the atoms, where there are several and the scratch holds them
  double *form = nullptr;
  if (gp.nat >= 4 && scratch_bytes >= (size_t)gp.nk * gp.nh * 4 * pd.nG * sizeof(double)) {
    form = (double *)scratch;
    k_nl_forms<R><<<dim3((pd.nG + 127) / 128, gp.nk), 128, 0, st>>>(pd, gp, form);
    ADDFT_TRY(check_launch("k_nl_forms"));
  }
  size_t smem = 0;
  const int f = phase_form(pd, smem);
  const dim3 grid(gp.nat, nsplit, gp.nk);
  auto go = [&](auto kern, const auto &fr) {
    ADDFT_TRY(smem_optin(kern, smem));
    kern<<<grid, 256, smem, st>>>(pd, gp, fr, (const C *)Y, form, nsplit, part);
    return check_launch("k_nl_grad");
  };
  return f == 2   ? go(k_nl_grad<R, 2>, make_fracs<2>(gp))
         : f == 1 ? go(k_nl_grad<R, 1>, make_fracs<1>(gp))
                  : go(k_nl_grad<R, 0>, make_fracs<0>(gp));
}

// addft_hpsi on the caller's stream only (no second stream, no events): the form the
// no-allocation entry point runs, which creates no CUDA objects per call.
addft_status hpsi_one_stream(addft_plan plan, addft_dtype dt, int nk, int nb, const void *psi, const void *kin,
                             const void *v_r, int nproj, const void *proj, const void *dion, void *hpsi, void *work,
                             size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(plan && nk >= 1 && nb >= 0 && nproj >= 0, ADDFT_INVALID_ARG, "hpsi: bad arguments");
  if (nb == 0) return ADDFT_OK;   // no bands: the data pointers may be NULL
  ADDFT_REQUIRE(psi && kin && v_r && hpsi, ADDFT_INVALID_ARG, "hpsi: null pointer");
  ADDFT_REQUIRE(nproj == 0 || (proj && dion), ADDFT_INVALID_ARG, "hpsi: null projector tables");
  ADDFT_REQUIRE(psi != hpsi, ADDFT_INVALID_ARG, "hpsi: output aliases input");
  return dt == ADDFT_F64 ? hpsi_t<double>(plan, nk, nb, psi, kin, v_r, nproj, proj, dion, hpsi, work, work_bytes,
                                          as_stream(stream), false)
                         : hpsi_t<float>(plan, nk, nb, psi, kin, v_r, nproj, proj, dion, hpsi, work, work_bytes,
                                         as_stream(stream), false);
}

}  // namespace addft

using namespace addft;

extern "C" {

addft_status addft_kinetic(addft_plan plan, addft_dtype dt, const double *bvec, int nk,
                           const double *kpts, void *kin, void *stream) {
  ADDFT_REQUIRE(plan && bvec && kin && nk >= 1, ADDFT_INVALID_ARG, "kinetic: bad arguments");
  GeoParams gp;
  ADDFT_TRY(make_geo(gp, bvec, 1.0, nk, kpts, 0, nullptr, nullptr));
  dim3 grid((plan->dev.nG + 255) / 256, nk);
  if (dt == ADDFT_F64)
    k_kinetic<double><<<grid, 256, 0, as_stream(stream)>>>(plan->dev, gp, (double *)kin);
  else
    k_kinetic<float><<<grid, 256, 0, as_stream(stream)>>>(plan->dev, gp, (float *)kin);
  return check_launch("k_kinetic");
}

addft_status addft_projectors(addft_plan plan, addft_dtype dt, const double *bvec, double omega, int nk,
                              const double *kpts, int nat, const double *pos, const addft_psp *psp,
                              void *proj, void *stream) {
  ADDFT_REQUIRE(plan && bvec && psp && proj && (nat == 0 || pos), ADDFT_INVALID_ARG,
                "projectors: bad arguments");
  GeoParams gp;
  ADDFT_TRY(make_geo(gp, bvec, omega, nk, kpts, nat, pos, psp));
  if (nat * gp.nh == 0) return ADDFT_OK;
  return dt == ADDFT_F64 ? projectors_t<double>(plan->dev, gp, proj, as_stream(stream))
                         : projectors_t<float>(plan->dev, gp, proj, as_stream(stream));
}

addft_status addft_becp(addft_dtype dt, int nk, int nb, int nG, int nproj, const void *proj,
                        const void *psi, void *becp, void *work, size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(nk >= 0 && nb >= 0 && nG > 0 && nproj >= 0, ADDFT_INVALID_ARG, "becp: bad sizes");
  if (nk * nb * nproj == 0) return ADDFT_OK;
  ADDFT_REQUIRE(proj && psi && becp, ADDFT_INVALID_ARG, "becp: null pointer");
  return dt == ADDFT_F64
             ? becp_t<double>(nk, nb, nG, nproj, proj, psi, becp, work, work_bytes, as_stream(stream))
             : becp_t<float>(nk, nb, nG, nproj, proj, psi, becp, work, work_bytes, as_stream(stream));
}

addft_status addft_vnl_apply(addft_dtype dt, int nk, int nb, int nG, int nproj, const void *proj,
                             const void *dion, const void *becp, void *hpsi, void *work,
                             size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(nk >= 0 && nb >= 0 && nG > 0 && nproj >= 0, ADDFT_INVALID_ARG, "vnl_apply: bad sizes");
  if (nk * nb * nproj == 0) return ADDFT_OK;
  const size_t csz = dt == ADDFT_F64 ? 16 : 8;
  ADDFT_REQUIRE(proj && dion && becp && hpsi && work && work_bytes >= (size_t)nk * nproj * nb * csz,
                ADDFT_INVALID_ARG, "vnl_apply: null pointer or work < nk*nproj*nb complex");
  cudaStream_t st = as_stream(stream);
  const size_t Pk = (size_t)nproj * nG, Xk = (size_t)nproj * nb, Ok = (size_t)nb * nG;
  // what the buffer holds beyond D becp (from a 256-byte boundary on) is the apply's scratch
  const size_t db = (size_t)nk * nproj * nb * csz;
  char *rest = (char *)(((uintptr_t)work + db + 255) & ~(uintptr_t)255);
  const size_t off = (size_t)(rest - (char *)work), left = work_bytes > off ? work_bytes - off : 0;
  if (dt == ADDFT_F64) {
    ADDFT_TRY(dbecp_t<double>(dion, becp, nk, nproj, nb, nullptr, work, st));
    return apply_t<double, false, true>(work, nb, 1, Xk, proj, Pk, nk, nproj, nb, nG, hpsi, Ok, rest, left, st);
  }
  ADDFT_TRY(dbecp_t<float>(dion, becp, nk, nproj, nb, nullptr, work, st));
  return apply_t<float, false, true>(work, nb, 1, Xk, proj, Pk, nk, nproj, nb, nG, hpsi, Ok, rest, left, st);
}

addft_status addft_nonlocal_energy(addft_dtype dt, int nk, int nb, int nproj, const void *becp,
                                   const void *dion, const double *wocc, double *e_out, void *work,
                                   size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(nk >= 0 && nb >= 0 && nproj >= 0 && e_out, ADDFT_INVALID_ARG, "nonlocal_energy: bad sizes");
  cudaStream_t st = as_stream(stream);
  if (nk * nb * nproj == 0) {
    ADDFT_CUDA(cudaMemsetAsync(e_out, 0, sizeof(double), st));
    return ADDFT_OK;
  }
  const size_t csz = dt == ADDFT_F64 ? 16 : 8;
  const size_t need = align256((size_t)nk * nproj * nb * csz) + (size_t)nk * nb * sizeof(double);
  ADDFT_REQUIRE(becp && dion && wocc && work && work_bytes >= need, ADDFT_INVALID_ARG,
                "nonlocal_energy: null pointer or work < %zu B", need);
  char *w = (char *)work;
  double *ep = (double *)(w + align256((size_t)nk * nproj * nb * csz));
  if (dt == ADDFT_F64) {
    ADDFT_TRY(dbecp_t<double>(dion, becp, nk, nproj, nb, nullptr, w, st));
    ADDFT_TRY(nl_energy_t<double>(becp, w, nk, nproj, nb, wocc, ep, st));
  } else {
    ADDFT_TRY(dbecp_t<float>(dion, becp, nk, nproj, nb, nullptr, w, st));
    ADDFT_TRY(nl_energy_t<float>(becp, w, nk, nproj, nb, wocc, ep, st));
  }
  return finalize_sums(ep, 1, nk * nb, e_out, false, st);
}

addft_status addft_hpsi(addft_plan plan, addft_dtype dt, int nk, int nb, const void *psi, const void *kin,
                        const void *v_r, int nproj, const void *proj, const void *dion, void *hpsi,
                        void *work, size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(plan && nk >= 1 && nb >= 0 && nproj >= 0, ADDFT_INVALID_ARG, "hpsi: bad arguments");
  if (nb == 0) return ADDFT_OK;   // no bands: the data pointers may be NULL
  ADDFT_REQUIRE(psi && kin && v_r && hpsi, ADDFT_INVALID_ARG, "hpsi: null pointer");
  ADDFT_REQUIRE(nproj == 0 || (proj && dion), ADDFT_INVALID_ARG, "hpsi: null projector tables");
  ADDFT_REQUIRE(psi != hpsi, ADDFT_INVALID_ARG, "hpsi: output aliases input");
  return dt == ADDFT_F64 ? hpsi_t<double>(plan, nk, nb, psi, kin, v_r, nproj, proj, dion, hpsi, work, work_bytes,
                                          as_stream(stream), true)
                         : hpsi_t<float>(plan, nk, nb, psi, kin, v_r, nproj, proj, dion, hpsi, work, work_bytes,
                                         as_stream(stream), true);
}

size_t addft_hpsi_work_bytes(addft_plan plan, addft_dtype dt, int nk, int nb, int nproj, int nbatch_chunk) {
  if (!plan) return 0;
  const size_t nls = dt == ADDFT_F64 ? nl_scratch<double>(nk, nb, plan->dev.nG, nproj)
                                     : nl_scratch<float>(nk, nb, plan->dev.nG, nproj);
  return nls + addft_work_bytes(plan, nbatch_chunk < 1 ? 1 : nbatch_chunk, dt);
}

addft_status addft_kinetic_stress(addft_plan plan, addft_dtype dt, const double *bvec, int nk,
                                  const double *kpts, int nb, const void *psi, const double *wocc,
                                  double *out9, void *work, size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(plan && bvec && psi && wocc && out9 && work && work_bytes >= 9 * kRedBlocks * sizeof(double),
                ADDFT_INVALID_ARG, "kinetic_stress: bad arguments");
  GeoParams gp;
  ADDFT_TRY(make_geo(gp, bvec, 1.0, nk, kpts, 0, nullptr, nullptr));
  cudaStream_t st = as_stream(stream);
  double *part = (double *)work;
  if (dt == ADDFT_F64)
    k_kin_stress<double><<<kRedBlocks, 256, 0, st>>>(plan->dev, gp, (const double2 *)psi, nb, wocc, part);
  else
    k_kin_stress<float><<<kRedBlocks, 256, 0, st>>>(plan->dev, gp, (const float2 *)psi, nb, wocc, part);
  ADDFT_TRY(check_launch("k_kin_stress"));
  return finalize_sums(part, 9, kRedBlocks, out9, true, st);
}

addft_status addft_nonlocal_gradients(addft_plan plan, addft_dtype dt, const double *bvec, double omega,
                                      int nk, const double *kpts, int nb, int nat, const double *pos,
                                      const addft_psp *psp, const void *psi, const double *wocc,
                                      const void *dion, double *out, void *work, size_t work_bytes,
                                      void *stream) {
  ADDFT_REQUIRE(plan && bvec && psp && psi && wocc && dion && out && work, ADDFT_INVALID_ARG,
                "nonlocal_gradients: bad arguments");
  GeoParams gp;
  ADDFT_TRY(make_geo(gp, bvec, omega, nk, kpts, nat, pos, psp));
  cudaStream_t st = as_stream(stream);
  const int nproj = nat * gp.nh;
  const int nG = plan->dev.nG;
  if (nproj == 0) {
    ADDFT_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (1 + 3 * nat + 9), st));
    return ADDFT_OK;
  }
  const size_t csz = dt == ADDFT_F64 ? 16 : 8;
  // layout: proj | becp | DB | Mw | Y | epart | gpart | becp split scratch
  size_t off = 0;
  auto take = [&](size_t b) { size_t o = off; off += align256(b); return o; };
  const size_t o_proj = take((size_t)nk * nproj * nG * csz);
  const size_t o_becp = take((size_t)nk * nproj * nb * csz);
  const size_t o_db = take((size_t)nk * nproj * nb * csz);
  const size_t o_mw = take((size_t)nk * nproj * nb * csz);
  const size_t o_y = take((size_t)nk * nproj * nG * csz);
  const size_t o_ep = take((size_t)nk * nb * sizeof(double));
  // fewer splits of the G range and less scratch for the contractions, where the buffer is short of what is asked for
  const size_t partials = align256(dt == ADDFT_F64 ? becp_partial_bytes<double>(nk, nb, nG, nproj)
                                                   : becp_partial_bytes<float>(nk, nb, nG, nproj));
  auto sums = [&](int n) { return (size_t)nk * nat * n * 12 * sizeof(double); };
  int nsplit = nl_grad_splits(nk, nat, nG);
  while (nsplit > 1 && off + align256(sums(nsplit)) + partials > work_bytes) --nsplit;
  const size_t o_gp = take(sums(nsplit)), o_bw = off;
  off += partials;
  ADDFT_REQUIRE(work_bytes >= off, ADDFT_INVALID_ARG, "nonlocal_gradients: work needs %zu B, got %zu B",
                off, work_bytes);
  const size_t bwb = work_bytes - o_bw;   // becp's partials or operands, then the operands of Y
  char *w = (char *)work;
  ADDFT_TRY(addft_projectors(plan, dt, bvec, omega, nk, kpts, nat, pos, psp, w + o_proj, stream));
  if (dt == ADDFT_F64) {
    ADDFT_TRY(becp_t<double>(nk, nb, nG, nproj, w + o_proj, psi, w + o_becp, w + o_bw, bwb, st));
    ADDFT_TRY(dbecp_t<double>(dion, w + o_becp, nk, nproj, nb, nullptr, w + o_db, st));
    ADDFT_TRY(dbecp_t<double>(dion, w + o_becp, nk, nproj, nb, wocc, w + o_mw, st));
    ADDFT_TRY((apply_t<double, true, false>(w + o_mw, 1, nb, (size_t)nproj * nb, psi, (size_t)nb * nG, nk, nb,
                                            nproj, nG, w + o_y, (size_t)nproj * nG, w + o_bw, bwb, st)));
    ADDFT_TRY(nl_energy_t<double>(w + o_becp, w + o_db, nk, nproj, nb, wocc, (double *)(w + o_ep), st));
    // the projector table has been used; its place takes the channel tables
    ADDFT_TRY(nl_grad_t<double>(plan->dev, gp, w + o_y, w + o_proj, (size_t)nk * nproj * nG * csz, nsplit,
                                (double *)(w + o_gp), st));
  } else {
    ADDFT_TRY(becp_t<float>(nk, nb, nG, nproj, w + o_proj, psi, w + o_becp, w + o_bw, bwb, st));
    ADDFT_TRY(dbecp_t<float>(dion, w + o_becp, nk, nproj, nb, nullptr, w + o_db, st));
    ADDFT_TRY(dbecp_t<float>(dion, w + o_becp, nk, nproj, nb, wocc, w + o_mw, st));
    ADDFT_TRY((apply_t<float, true, false>(w + o_mw, 1, nb, (size_t)nproj * nb, psi, (size_t)nb * nG, nk, nb,
                                           nproj, nG, w + o_y, (size_t)nproj * nG, w + o_bw, bwb, st)));
    ADDFT_TRY(nl_energy_t<float>(w + o_becp, w + o_db, nk, nproj, nb, wocc, (double *)(w + o_ep), st));
    ADDFT_TRY(nl_grad_t<float>(plan->dev, gp, w + o_y, w + o_proj, (size_t)nk * nproj * nG * csz, nsplit,
                               (double *)(w + o_gp), st));
  }
  k_nl_grad_final<<<(1 + 3 * nat + 9 + 3) / 4, 128, 0, st>>>((const double *)(w + o_ep), nk * nb,
                                                            (const double *)(w + o_gp), nk, nat, nsplit, out);
  return check_launch("k_nl_grad_final");
}

size_t addft_nonlocal_gradients_work_bytes(addft_dtype dt, int nk, int nb, int nG, int nat, int nh) {
  const size_t csz = dt == ADDFT_F64 ? 16 : 8;
  const int nproj = nat * nh;
  size_t s = 0;
  s += align256((size_t)nk * nproj * nG * csz) * 2;
  s += align256((size_t)nk * nproj * nb * csz) * 3;
  s += align256((size_t)nk * nb * sizeof(double));
  s += nat > 0 ? align256((size_t)nk * nat * nl_grad_splits(nk, nat, nG) * 12 * sizeof(double)) : 0;
  s += align256(nl_grad_scratch(dt, nk, nb, nG, nproj));
  return s;
}

}  // extern "C"
