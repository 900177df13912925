// Roots of unity for the digit-slice transforms (dft64.cu), in fixed point.  Host code only, so that its
// properties can be checked without a GPU.
#pragma once
#include <cmath>
#include <cstdint>
#include <vector>

namespace addft {

// Roots of unity to about 2^-100 (double-double Taylor series on |angle| <= pi / 4): cos(2 pi t / n) of a
// double angle is off by up to 4e-16, eight times what the digits resolve, and that error would be the
// transform's largest.
struct DD { double hi, lo; };
inline DD dd_add(DD a, DD b) {
  const double s = a.hi + b.hi, v = s - a.hi, e = (a.hi - (s - v)) + (b.hi - v) + a.lo + b.lo;
  const double r = s + e;
  return {r, e - (r - s)};
}
inline DD dd_mul(DD a, DD b) {
  const double p = a.hi * b.hi, e = std::fma(a.hi, b.hi, -p) + (a.hi * b.lo + a.lo * b.hi);
  const double r = p + e;
  return {r, e - (r - p)};
}
inline DD dd_div(DD a, double n) {
  const double q = a.hi / n, e = (std::fma(-q, n, a.hi) + a.lo) / n;
  const double r = q + e;
  return {r, e - (r - q)};
}
inline void root_of_unity(long t, long n, DD &c, DD &s) {   // e^{2 pi i t / n}, 0 <= t < n
  const long q = (4 * t + n / 2) / n, r = 4 * t - q * n;     // quarter turns and the rest, |r| <= n / 2
  const DD x = dd_div(dd_mul({1.5707963267948966, 6.123233995736766e-17}, {(double)r, 0.0}), (double)n);
  const DD x2 = dd_mul(x, x);
  DD term = {1.0, 0.0}, odd = x;
  c = term;
  s = odd;
  for (int k = 1; k <= 13; ++k) {
    term = dd_div(dd_mul(term, x2), -(double)((2 * k - 1) * (2 * k)));
    odd = dd_div(dd_mul(odd, x2), -(double)((2 * k) * (2 * k + 1)));
    c = dd_add(c, term);
    s = dd_add(s, odd);
  }
  for (long i = 0; i < (q & 3); ++i) {
    const DD o = c;
    c = {-s.hi, -s.lo};
    s = o;
  }
}

// The n roots' parts in units of 2^-bits, rounded so that the sums over the subgroups of order 2, 3
// and 5 stay exactly zero: a constant line then gives exact zeros beside its mean, as an FFT's
// butterflies do (a density's small components are multiplied by 1 / G^2 later).
struct Rounded { std::vector<int64_t> q; std::vector<double> e; };   // value, its excess over the root
inline void add_rounded(Rounded &r, DD x, int bits) {
  const double y = std::ldexp(x.hi, bits), f = std::floor(y), rest = (y - f) + std::ldexp(x.lo, bits);
  const int64_t up = std::llrint(rest);
  r.q.push_back((int64_t)f + up);
  r.e.push_back((double)up - rest);
}
inline void keep_sums(Rounded &r, int n) {
  // order 2 holds already: opposite roots are rounded alike.  Orders 3 and 5: tables of 3 x 5 (3, 5)
  // roots whose columns (rows) have to sum to zero.
  const int rows = n % 3 == 0 ? 3 : 1, cols = n % 5 == 0 ? 5 : 1, half = n % 2 == 0 ? n / 2 : 0;
  if (rows * cols == 1) return;
  std::vector<char> seen((size_t)n, 0);
  for (int t = 0; t < n; ++t) {
    if (seen[t]) continue;
    int at[3][5];
    int64_t R[3] = {0, 0, 0}, C[5] = {0, 0, 0, 0, 0};   // row sums (where cols = 5), column sums (rows = 3)
    for (int i = 0; i < rows; ++i)
      for (int j = 0; j < cols; ++j) {
        const int a = at[i][j] = (t + i * (n / 3) + j * (n / 5)) % n;
        seen[a] = 1;
        if (half) seen[(a + half) % n] = 1;
        if (cols > 1) R[i] += r.q[a];
        if (rows > 1) C[j] += r.q[a];
      }
    auto move = [&](int i, int j, int by) {
      const int a = at[i][j];
      r.q[a] += by;
      r.e[a] += by;
      if (half) {
        r.q[(a + half) % n] -= by;
        r.e[(a + half) % n] -= by;
      }
      if (cols > 1) R[i] += by;
      if (rows > 1) C[j] += by;
    };
    // each step takes one unit off sums that are not zero, at the entries furthest off that way; the
    // sums are a few units, so the steps are few
    for (int step = 0; step < 64; ++step) {
      int bi = -1, bj = -1, bk = -1, dir = 0;
      double best = -1e9;
      for (int d = -1; d <= 1; d += 2)
        for (int i = 0; i < rows; ++i)
          for (int j = 0; j < cols; ++j)
            if ((cols == 1 || R[i] * d < 0) && (rows == 1 || C[j] * d < 0) && -d * r.e[at[i][j]] > best) {
              best = -d * r.e[at[i][j]];
              bi = i, bj = j, dir = d;
            }
      if (dir) {
        move(bi, bj, dir);
        continue;
      }
      for (int i = 0; i < rows; ++i)   // rows of both signs are left: one unit from one to the other
        for (int k = 0; k < rows; ++k)
          for (int j = 0; j < cols; ++j)
            if (R[i] > 0 && R[k] < 0 && r.e[at[i][j]] - r.e[at[k][j]] > best) {
              best = r.e[at[i][j]] - r.e[at[k][j]];
              bi = i, bj = j, bk = k, dir = 1;
            }
      if (dir) {
        move(bi, bj, -1);
        move(bk, bj, 1);
        continue;
      }
      for (int i = 0; i < rows; ++i)   // columns alike
        for (int k = 0; k < cols; ++k)
          for (int j = 0; j < cols; ++j)
            if (C[j] > 0 && C[k] < 0 && r.e[at[i][j]] - r.e[at[i][k]] > best) {
              best = r.e[at[i][j]] - r.e[at[i][k]];
              bi = i, bj = j, bk = k, dir = 1;
            }
      if (!dir) break;
      move(bi, bj, -1);
      move(bi, bk, 1);
    }
  }
}

// Re and Im of e^{2 pi i t / n} (forward: of its conjugate), t = 0 .. n - 1, rounded
inline void rounded_roots(int n, bool forward, int bits, Rounded &re, Rounded &im) {
  for (int t = 0; t < n; ++t) {
    DD c, s;
    root_of_unity(forward ? (n - t) % n : t, n, c, s);
    add_rounded(re, c, bits);
    add_rounded(im, s, bits);
  }
  keep_sums(re, n);
  keep_sums(im, n);
}

}  // namespace addft
