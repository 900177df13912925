// Complex FP64 GEMM on the tensor cores by digit slicing (ozgemm.cu).
#pragma once
#include "common.cuh"

namespace addft {

// An operand of C[i][j] = sum_k A[i][k] B[j][k] (both indexed row, k): element (r, k) of batch
// entry b at p[b * s_batch + r * s_row + k * s_k], complex128, conjugated when conj != 0.
struct OzMat {
  const void *p;
  long s_row, s_k;
  size_t s_batch;
  int conj;
};

// Scratch that oz_gemm wants with 8 (62 bits) or 7 (55 bits) digits, 256-byte aligned; it
// works in pieces with less, and oz_fits tells whether a buffer is enough for that.
size_t oz_work_bytes(int digits, int M, int N, int K, int batch);
bool oz_fits(int digits, int M, int N, int K, int batch, const void *work, size_t bytes);

// C[b * s_batch + i * s_row + j * s_col] (+)= sum_k A[i][k] B[j][k] for M x N outputs per batch entry.
addft_status oz_gemm(int digits, int M, int N, int K, int batch, const OzMat &A, const OzMat &B, void *C, long s_row,
                     long s_col, size_t s_batch, bool accum, void *work, size_t work_bytes, cudaStream_t st);

// Device-side error bits since the last call (bit 0: a bounded wait ran out), cleared by the read.
unsigned oz_status();
unsigned d64_status();   // the same for dft64.cu

}  // namespace addft
