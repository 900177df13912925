// Host harness of tests/test_roots_host.py.
#include "roots.hpp"

using namespace addft;

extern "C" void roots(int n, int forward, int bits, int64_t *re, int64_t *im, double *ere, double *eim) {
  Rounded a, b;
  rounded_roots(n, forward != 0, bits, a, b);
  for (int t = 0; t < n; ++t) {
    re[t] = a.q[t];
    im[t] = b.q[t];
    ere[t] = a.e[t];
    eim[t] = b.e[t];
  }
}
