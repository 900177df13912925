// Host harness of tests/test_ozlayout_host.py: what the pieces of a digit-slice product take.
#include "ozlayout.hpp"

using namespace addft;

// Largest layout over all pieces of an r x c x K product in `bytes` of scratch (0: it does not go at all);
// *covered counts the outputs times K of all pieces, *splits the most K splits of one.
extern "C" size_t oz_most(int digits, int r, int c, int K, int batch, size_t bytes, double *covered, int *splits, int *n) {
  OzPieces p;
  *covered = 0;
  *splits = *n = 0;
  if (!oz_pieces(digits, r, c, K, batch, bytes, p)) return 0;
  size_t most = 0;
  oz_each_piece(r, c, K, batch, p, [&](int, int, int, int, int nb, int nr, int nc, int nk) {
    const OzLayout l = oz_layout(digits, nr, nc, nk, nb, p.nsplit);
    most = std::max(most, l.total);
    *covered += (double)nb * nr * nc * nk;
    *splits = std::max(*splits, l.nsplit);
    ++*n;
    return 0;
  });
  return most;
}

extern "C" size_t oz_whole(int digits, int r, int c, int K, int batch) { return oz_layout(digits, r, c, K, batch).total; }
