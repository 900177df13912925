// Scratch layout of the digit-slice GEMM (ozgemm.cu): tiles, K splits and pieces.  Host code only, so
// that the sizes can be checked without a GPU.
#pragma once
#include <algorithm>
#include <cstddef>

namespace addft {

constexpr int kOzRowsA = 128, kOzRowsB = 32;   // rows of an A / B tile
constexpr int kOzStep = 16;                    // k per stage
constexpr int kOzDrain = 8;                    // stages per accumulation block
constexpr int kOzSms = 152;
constexpr int kOzMinPieceK = 1024;             // K is not cut below this when scratch is short

inline size_t oz_al256(size_t x) { return (x + 255) & ~size_t(255); }

struct OzLayout {
  int ta, tb, nks, nsplit, steps;      // row / column tiles, stages, K splits, stages per split
  size_t pa, pb;                       // packed bytes per batch entry
  size_t o_ex, o_pa, o_pb, o_part, total;
};

// rows / cols as the kernel sees them (rows on the 128-row side); at most max_split K splits
inline OzLayout oz_layout(int digits, int rows, int cols, int K, int batch, int max_split = 2 * kOzSms) {
  OzLayout l;
  l.ta = (rows + kOzRowsA - 1) / kOzRowsA;
  l.tb = (cols + kOzRowsB - 1) / kOzRowsB;
  l.nks = (K + kOzStep - 1) / kOzStep;
  // A CTA fills an SM, so a split count costs waves x (accumulation blocks per CTA + about one
  // block's time to start and to end a CTA); splits keep whole accumulation blocks.
  const long tiles = (long)l.ta * l.tb * batch;
  const int blocks = (l.nks + kOzDrain - 1) / kOzDrain;
  int per = blocks;
  long best = -1;
  for (int ns = 1; ns <= std::min(blocks, max_split); ++ns) {
    const int b = (blocks + ns - 1) / ns, used = (blocks + b - 1) / b;
    const long cost = (tiles * used + kOzSms - 1) / kOzSms * (b + 1) + (used > 1 ? 1 : 0);
    if (best < 0 || cost < best) {
      best = cost;
      per = b;
    }
    if (tiles >= 8 * kOzSms) break;   // many waves: nothing to fill
  }
  l.steps = per * kOzDrain;
  l.nsplit = (l.nks + l.steps - 1) / l.steps;
  l.pa = (size_t)l.ta * l.nks * (2 * digits * kOzRowsA * kOzStep * 2);
  l.pb = (size_t)l.tb * l.nks * (2 * digits * kOzRowsB * kOzStep * 2);
  l.o_ex = 0;
  l.o_pa = oz_al256((size_t)batch * (rows + cols) * sizeof(int));
  l.o_pb = l.o_pa + oz_al256(l.pa * batch);
  l.o_part = l.o_pb + oz_al256(l.pb * batch);
  l.total = l.o_part + (l.nsplit > 1 ? (size_t)l.nsplit * rows * cols * batch * 2 * sizeof(double) : 0);
  return l;
}

// Pieces of a product that fit the scratch: batch entries at a time, then rows, columns or K cut
// down, whichever packs largest.  Pieces at the edges are smaller, and with as many K splits at most as a
// whole one they need no more scratch; left to themselves they would take more (fewer tiles to fill the chip
// with) and their partial sums could outgrow what the operands save.
struct OzPieces { int batch, rows, cols, K, nsplit; };
inline bool oz_pieces(int digits, int r, int c, int K, int batch, size_t bytes, OzPieces &p) {
  p = {batch, r, c, K, 1};
  for (;;) {
    const OzLayout l = oz_layout(digits, p.rows, p.cols, p.K, p.batch);
    p.nsplit = l.nsplit;
    if (l.total <= bytes) break;
    auto half = [](int n, int unit) { return (n / 2 + unit - 1) / unit * unit; };
    if (p.batch > 1) p.batch = (p.batch + 1) / 2;
    else if (p.K > 2 * kOzMinPieceK) p.K = half(p.K, kOzDrain * kOzStep);
    else if (p.rows >= p.cols && p.rows > 2 * kOzRowsA) p.rows = half(p.rows, kOzRowsA);
    else if (p.cols > 2 * kOzRowsB) p.cols = half(p.cols, kOzRowsB);
    else return false;
  }
  return (p.rows + kOzRowsA - 1) / kOzRowsA <= 65535 && (p.cols + kOzRowsB - 1) / kOzRowsB <= 65535 && p.batch <= 200;
}

// run(b0, r0, c0, k0, nb, nr, nc, nk) for every piece in order, while it returns 0
template <typename F>
int oz_each_piece(int r, int c, int K, int batch, const OzPieces &p, F run) {
  for (int b0 = 0; b0 < batch; b0 += p.batch)
    for (int r0 = 0; r0 < r; r0 += p.rows)
      for (int c0 = 0; c0 < c; c0 += p.cols)
        for (int k0 = 0; k0 < K; k0 += p.K) {
          const int s = run(b0, r0, c0, k0, std::min(p.batch, batch - b0), std::min(p.rows, r - r0),
                            std::min(p.cols, c - c0), std::min(p.K, K - k0));
          if (s != 0) return s;
        }
  return 0;
}

}  // namespace addft
