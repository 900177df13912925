// Ewald ion-ion energy with its position and strain derivatives, f64 on the
// device.  Reference: src/addft/physics/ewald.py:34-77 (nmax translations
// per axis in real space, (2 nmax + 5)^3 reciprocal vectors, eta = 0.9
// default), E = E_real + E_recip + E_self + E_bg.
#include <algorithm>

#include "common.cuh"

namespace addft {

constexpr int kMaxAtomsE = 256;
constexpr int kRecipCtas = 456;    // three reciprocal CTAs per SM, columns (a, b) dealt out
constexpr int kRecipChunk = 16;    // third-axis indices held in shared memory at a time

struct EwaldParams {
  double L[9];     // lattice rows
  double B[9];     // reciprocal rows
  double omega, eta;
  int nat, nmax;
  int nr[3];       // translations per axis that reach within the real-space cut
  double z[kMaxAtomsE];
};
// positions (real-space sum) and fractional coordinates (phases of the reciprocal sum): each a parameter of the one
// kernel that reads it
struct EwaldPos { double r[kMaxAtomsE * 3]; };
struct EwaldFracs { Turns f[kMaxAtomsE * 3]; };

// Pairs further apart than this times 1/eta add erfc(10) < 3e-45 per unit charge: nothing that an
// FP64 sum beside the self term could show, so they are not evaluated (Si64, nmax = 8: 27 of the
// 4,913 translations remain).
constexpr double kRealCut = 10.0;

// Real-space sum of atom i over all atoms and translations, split over gridDim.y:
// partial[i * ns + split][13] = {E, dE/dR_i (3), dE/deps (9)}.  Translations come in +- pairs, so
// the force on i from its pairs (i, j) and (j, i) is twice the sum over (i, j).
// Bound by the FP64 pipe (erfc, exp, sqrt and two divisions per term): 7.85 ms with every
// translation of every pair and one CTA per pair, 0.06 ms so (Si64).
__global__ void __launch_bounds__(256) k_ewald_real(EwaldParams ep, EwaldPos at, double *__restrict__ partial) {
  const int i = blockIdx.x, ns = gridDim.y;
  const int s1 = 2 * ep.nr[0] + 1, s2 = 2 * ep.nr[1] + 1, s3 = 2 * ep.nr[2] + 1, nt = s1 * s2 * s3;
  // translations of one pair fit 32 bits, pairs times translations need not (a small eta reaches far)
  const long total = (long)ep.nat * nt, stride = (long)ns * blockDim.x;
  const double rp = 1.1283791670955125739 * ep.eta;   // 2 eta / sqrt(pi)
  const double cut2 = (kRealCut / ep.eta) * (kRealCut / ep.eta);
  double acc[13];
#pragma unroll
  for (int t = 0; t < 13; ++t) acc[t] = 0.0;
  for (long q = blockIdx.y * blockDim.x + threadIdx.x; q < total; q += stride) {
    const int j = total <= 0x7fffffff ? (int)q / nt : (int)(q / nt), t = (int)(q - (long)j * nt);
    const int a = t / (s2 * s3) - ep.nr[0], b = (t / s3) % s2 - ep.nr[1], c = t % s3 - ep.nr[2];
    if (i == j && a == 0 && b == 0 && c == 0) continue;
    double d[3];
    for (int x = 0; x < 3; ++x)
      d[x] = at.r[3 * i + x] - at.r[3 * j + x] + a * ep.L[x] + b * ep.L[3 + x] + c * ep.L[6 + x];
    const double d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    if (d2 > cut2) continue;
    const double zz = ep.z[i] * ep.z[j];
    const double dist = sqrt(d2 + 1e-30);
    const double phi = erfc(ep.eta * dist) / dist;
    const double dphi = -phi / dist - rp * exp(-(ep.eta * dist) * (ep.eta * dist)) / dist;
    acc[0] += 0.5 * zz * phi;
    const double f = 0.5 * zz * dphi / dist;
    if (i != j)
      for (int x = 0; x < 3; ++x) acc[1 + x] += 2.0 * f * d[x];
    for (int x = 0; x < 3; ++x)
      for (int y = 0; y < 3; ++y) acc[4 + 3 * x + y] += f * d[x] * d[y];
  }
  __shared__ double red[8][13];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q = 0; q < 13; ++q) {
    double x = acc[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][q] = x;
  }
  __syncthreads();
  if (threadIdx.x < 13) {
    double s = 0.0;
    for (int w = 0; w < (blockDim.x >> 5); ++w) s += red[w][threadIdx.x];
    partial[((size_t)i * ns + blockIdx.y) * 13 + threadIdx.x] = s;
  }
}

// Reciprocal sum, energy, strain and forces in one pass.  A thread owns an atom; a CTA takes the
// columns (a, b) of the reciprocal grid in turn: phases e^{-iG.R} = e12 e3 of one chunk of the
// third axis go to shared memory, warps reduce the structure factors S(G), then every thread
// adds its atom's force.  A phase costs one complex product (the tables hold e^{-2 pi i m f}) where
// a sincos per atom and G, once for S and again in every atom's force sum, took 5.0 ms (Si64):
// 0.10 ms so.  partial[cta][10 + 3 nat] = {sum w |S|^2, sum coef |S|^2 G_a G_b, forces}.
__global__ void __launch_bounds__(256) k_ewald_recip(EwaldParams ep, EwaldFracs fr, double *__restrict__ partial) {
  extern __shared__ double2 ew_smem[];
  const int nat = ep.nat, M = ep.nmax + 2, side = 2 * M + 1;
  double2 *e3 = ew_smem, *ph = e3 + kRecipChunk * nat;   // [chunk][atom]
  __shared__ double2 S[kRecipChunk];
  __shared__ double wgt[kRecipChunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // rows of natp threads (atoms), each taking every nrow-th third-axis index
  const int natp = (nat + 31) & ~31, nrow = blockDim.x / natp, row = threadIdx.x / natp, i = threadIdx.x - row * natp;
  const bool on = i < nat && row < nrow;
  const double e4 = 4.0 * ep.eta * ep.eta;
  double F[3] = {0.0, 0.0, 0.0}, sums[10];
  for (int q = 0; q < 10; ++q) sums[q] = 0.0;   // used by lane 0 of each warp
  for (int c0 = 0; c0 < side; c0 += kRecipChunk) {
    const int nc = min(kRecipChunk, side - c0);
    if (on)
      for (int c = row; c < nc; c += nrow) e3[c * nat + i] = phase_exp(c0 + c - M, fr.f[3 * i + 2]);
    for (int col = blockIdx.x; col < side * side; col += gridDim.x) {
      const int a = col / side - M, b = col % side - M;
      if (on) {
        const double2 p1 = phase_exp(a, fr.f[3 * i]), p2 = phase_exp(b, fr.f[3 * i + 1]), e12 = cmul(p1, p2);
        for (int c = row; c < nc; c += nrow) ph[c * nat + i] = cmul(e12, e3[c * nat + i]);
      }
      __syncthreads();
      for (int c = warp; c < nc; c += nw) {
        double sr = 0.0, si = 0.0;
        for (int j = lane; j < nat; j += 32) {
          const double2 p = ph[c * nat + j];
          sr += ep.z[j] * p.x;
          si += ep.z[j] * p.y;
        }
        for (int o = 16; o > 0; o >>= 1) {
          sr += __shfl_down_sync(0xffffffffu, sr, o);
          si += __shfl_down_sync(0xffffffffu, si, o);
        }
        if (lane == 0) {
          const int m3 = c0 + c - M;
          double g[3];
          for (int x = 0; x < 3; ++x) g[x] = a * ep.B[x] + b * ep.B[3 + x] + m3 * ep.B[6 + x];
          const double g2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
          const bool keep = g2 > 1e-12;
          const double ex = keep ? exp(-g2 / e4) : 0.0, w = keep ? ex / g2 : 0.0;
          S[c] = make_double2(sr, si);
          wgt[c] = w;
          if (keep) {
            const double q2 = sr * sr + si * si;
            sums[0] += w * q2;
            const double coef = ex * (1.0 / (e4 * g2) + 1.0 / (g2 * g2)) * 2.0 * q2;
            for (int x = 0; x < 3; ++x)
              for (int y = 0; y < 3; ++y) sums[1 + 3 * x + y] += coef * g[x] * g[y];
          }
        }
      }
      __syncthreads();
      if (on) {
        // 2 w Re(conj(S) z_i (-i) p) = 2 w z_i (Sr p.y - Si p.x), times G
        double t0 = 0.0, t1 = 0.0;
        for (int c = row; c < nc; c += nrow) {
          const double2 p = ph[c * nat + i];
          const double re = 2.0 * wgt[c] * ep.z[i] * (S[c].x * p.y - S[c].y * p.x);
          t0 += re;
          t1 += re * (c0 + c - M);
        }
        for (int x = 0; x < 3; ++x) F[x] += t0 * (a * ep.B[x] + b * ep.B[3 + x]) + t1 * ep.B[6 + x];
      }
      __syncthreads();
    }
  }
  double *out = partial + (size_t)blockIdx.x * (10 + 3 * nat);
  double *sums_of = reinterpret_cast<double *>(ph);   // the rows' forces, added in row order
  if (on)
    for (int x = 0; x < 3; ++x) sums_of[(row * nat + i) * 3 + x] = F[x];
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * nat; t += blockDim.x) {
    double s = 0.0;
    for (int r = 0; r < nrow; ++r) s += sums_of[r * nat * 3 + t];
    out[10 + t] = s;
  }
  __shared__ double red[8][10];
  if (lane == 0)
    for (int q = 0; q < 10; ++q) red[warp][q] = sums[q];
  __syncthreads();
  if (threadIdx.x < 10) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += red[w][threadIdx.x];
    out[threadIdx.x] = s;
  }
}

// out: [0] E, [1 ..] dE/dR, then dE/deps (9); a warp per output sums the partials
__global__ void __launch_bounds__(128)
k_ewald_final(EwaldParams ep, const double *__restrict__ real_part, int ns, const double *__restrict__ recip, int nctas,
              double *__restrict__ out) {
  const int nat = ep.nat, lane = threadIdx.x & 31, rs = 10 + 3 * nat;
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= 1 + 3 * nat + 9) return;
  const double pref = 2.0 * 3.14159265358979323846 / ep.omega;
  const double sqpi = 1.7724538509055160273;
  auto warp_sum = [&](double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
  };
  auto recip_sum = [&](int q) {
    double s = 0.0;
    for (int c = lane; c < nctas; c += 32) s += recip[(size_t)c * rs + q];
    return pref * warp_sum(s);
  };
  double ztot = 0.0, z2 = 0.0;
  for (int i = 0; i < nat; ++i) { ztot += ep.z[i]; z2 += ep.z[i] * ep.z[i]; }
  const double e_self = -(ep.eta / sqpi) * z2;
  const double e_bg = -(3.14159265358979323846 / (2.0 * ep.omega * ep.eta * ep.eta)) * ztot * ztot;
  double v = 0.0;
  if (t >= 1 && t < 1 + 3 * nat) {
    const int i = (t - 1) / 3, x = (t - 1) % 3;
    for (int s = lane; s < ns; s += 32) v += real_part[((size_t)i * ns + s) * 13 + 1 + x];
    v = warp_sum(v) + recip_sum(10 + 3 * i + x);
  } else {
    const int ab = t - 1 - 3 * nat, q = t == 0 ? 0 : 4 + ab;
    for (int p = lane; p < nat * ns; p += 32) v += real_part[(size_t)p * 13 + q];
    v = warp_sum(v);
    if (t == 0) v += recip_sum(0) + e_self + e_bg;
    else {
      v += recip_sum(1 + ab);
      if (ab % 4 == 0) v += -recip_sum(0) - e_bg;
    }
  }
  if (lane == 0) out[t] = v;
}

}  // namespace addft

using namespace addft;

extern "C" {

size_t addft_ewald_work_bytes(int nat) {
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  return al((size_t)nat * nat * 13 * sizeof(double)) + al((size_t)kRecipCtas * (10 + 3 * nat) * sizeof(double));
}

addft_status addft_ewald(const double *lattice, int nat, const double *pos, const double *charges, double eta,
                         int nmax, double *out, void *work, size_t work_bytes, void *stream) {
  ADDFT_REQUIRE(lattice && out && nat >= 1 && pos && charges && eta > 0 && nmax >= 0, ADDFT_INVALID_ARG,
                "ewald: bad arguments");
  ADDFT_REQUIRE(nat <= kMaxAtomsE, ADDFT_UNSUPPORTED, "ewald: nat = %d exceeds %d", nat, kMaxAtomsE);
  // partial sums of the pairs, then of the reciprocal CTAs: as many of those as the buffer holds, four at least
  const size_t pairs = (((size_t)nat * nat * 13 * sizeof(double)) + 255) & ~size_t(255), per = (10 + 3 * nat) * sizeof(double);
  ADDFT_REQUIRE(work && work_bytes >= pairs + 4 * per, ADDFT_INVALID_ARG, "ewald: work needs %zu B", pairs + 4 * per);
  EwaldParams ep;
  memset(&ep, 0, sizeof(ep));
  for (int i = 0; i < 9; ++i) ep.L[i] = lattice[i];
  // B = 2 pi inv(L)^T, Omega = |det L|
  const double *L = lattice;
  const double det = L[0] * (L[4] * L[8] - L[5] * L[7]) - L[1] * (L[3] * L[8] - L[5] * L[6]) +
                     L[2] * (L[3] * L[7] - L[4] * L[6]);
  ADDFT_REQUIRE(fabs(det) > 0, ADDFT_INVALID_ARG, "ewald: singular lattice");
  double inv[9];
  inv[0] = (L[4] * L[8] - L[5] * L[7]) / det;
  inv[1] = (L[2] * L[7] - L[1] * L[8]) / det;
  inv[2] = (L[1] * L[5] - L[2] * L[4]) / det;
  inv[3] = (L[5] * L[6] - L[3] * L[8]) / det;
  inv[4] = (L[0] * L[8] - L[2] * L[6]) / det;
  inv[5] = (L[2] * L[3] - L[0] * L[5]) / det;
  inv[6] = (L[3] * L[7] - L[4] * L[6]) / det;
  inv[7] = (L[1] * L[6] - L[0] * L[7]) / det;
  inv[8] = (L[0] * L[4] - L[1] * L[3]) / det;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) ep.B[3 * r + c] = 2.0 * M_PI * inv[3 * c + r];
  ep.omega = fabs(det);
  ep.eta = eta;
  ep.nat = nat;
  ep.nmax = nmax;
  EwaldPos at;
  EwaldFracs fr;
  memset(&at, 0, sizeof(at));
  memset(&fr, 0, sizeof(fr));
  for (int i = 0; i < 3 * nat; ++i) at.r[i] = pos[i];
  for (int i = 0; i < nat; ++i) ep.z[i] = charges[i];
  cudaStream_t st = as_stream(stream);
  char *w = (char *)work;
  double *real_part = (double *)w, *recip = (double *)(w + pairs);
  // translations within the cut: |a + f_i - f_j| h <= cut on every axis, h = 2 pi / |b_a|
  for (int a = 0; a < 3; ++a) {
    double lo = 0.0, hi = 0.0;
    for (int i = 0; i < nat; ++i) {
      const double *r = pos + 3 * i, *bv = ep.B + 3 * a;
      const double f = (r[0] * bv[0] + r[1] * bv[1] + r[2] * bv[2]) / (2.0 * M_PI);
      lo = i ? std::min(lo, f) : f;
      hi = i ? std::max(hi, f) : f;
      fr.f[3 * i + a] = phase_turns(bv, r);
    }
    const double b = sqrt(ep.B[3 * a] * ep.B[3 * a] + ep.B[3 * a + 1] * ep.B[3 * a + 1] + ep.B[3 * a + 2] * ep.B[3 * a + 2]);
    const double reach = kRealCut / eta * b / (2.0 * M_PI) + (hi - lo) + 1e-6;
    ep.nr[a] = reach < nmax ? (int)reach : nmax;
  }
  // splits of an atom's sum: about 2 CTAs per SM, at least 256 terms each; the buffer holds nat
  const double cells = (2.0 * ep.nr[0] + 1) * (2.0 * ep.nr[1] + 1) * (2.0 * ep.nr[2] + 1);
  ADDFT_REQUIRE(cells <= 2147483647.0, ADDFT_UNSUPPORTED, "ewald: %.0f translations within reach", cells);
  const long terms = (long)nat * (long)cells;
  const int ns = (int)std::max<long>(1, std::min<long>(std::min<long>(nat, (terms + 255) / 256), (304 + nat - 1) / nat));
  k_ewald_real<<<dim3(nat, ns), 256, 0, st>>>(ep, at, real_part);
  ADDFT_TRY(check_launch("k_ewald_real"));
  const int side = 2 * (nmax + 2) + 1, nctas = (int)std::min<size_t>(std::min(kRecipCtas, side * side), (work_bytes - pairs) / per);
  const size_t sm = 2 * (size_t)kRecipChunk * nat * sizeof(double2);
  ADDFT_TRY(smem_optin(k_ewald_recip, sm));
  const int natp = (nat + 31) / 32 * 32;
  k_ewald_recip<<<nctas, natp * std::max(1, 256 / natp), sm, st>>>(ep, fr, recip);
  ADDFT_TRY(check_launch("k_ewald_recip"));
  k_ewald_final<<<(1 + 3 * nat + 9 + 3) / 4, 128, 0, st>>>(ep, real_part, ns, recip, nctas, out);
  return check_launch("k_ewald_final");
}

}  // extern "C"
