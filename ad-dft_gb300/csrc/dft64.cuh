// FP64 sphere transforms as digit-slice matrix products on the tensor cores (dft64.cu).
#pragma once
#include <vector>

#include "transforms.cuh"

namespace addft {

// Host side of a plan: the digits of the six transform matrices (x, y, z inverse, then forward)
// appended to `blob`, their geometry in `dm`; dm[a].tiles = 0 where an axis has no form.
void d64_build(int n1, int n2, int n3, const std::vector<int> &xact, const std::vector<int> &yact,
               const std::vector<int> &zact, D64Mat (&dm)[6], std::vector<unsigned char> &blob);

// Whether FP64 transforms of `bands` bands at once go through dft64 (box, size and tuning): local H psi, a
// band density, or a transform one way.
enum class D64Op { kHpsi, kDensity, kField };
bool d64_handles(const PlanDev &pd, D64Op op, int bands);

// Bands at once of a call over nbatch with `bytes` of scratch for them; 0: not one.
int d64_chunk(const PlanDev &pd, int nbatch, size_t bytes);

// Scratch bytes per band in flight, and of the potential in the order the x stage reads it.
size_t d64_band_bytes(const PlanDev &pd);
size_t d64_v_bytes(const PlanDev &pd);

// hpsi = kin psi + FFT^-1[V FFT[psi]] / N for nbatch bands; work holds d64_v_bytes + a multiple of
// d64_band_bytes and the bands go through in chunks.
addft_status d64_hpsi(const PlanDev &pd, int nbatch, const double2 *psi, const double *v_r, double2 *hpsi,
                      const double *kin, int nb_per_k, void *work, size_t bytes, cudaStream_t st);
// rho (+)= dscale sum_b wocc[b] |psi_b(r)|^2
addft_status d64_density(const PlanDev &pd, int nbatch, const double2 *psi, const double *wocc, double dscale, double *rho,
                         void *work, size_t bytes, cudaStream_t st);
// psi_r = scale * inverse transform, complex (or its real part) in (x, y, z) order
addft_status d64_to_real(const PlanDev &pd, int nbatch, const double2 *psi, double scale, void *out, bool real_part,
                         void *work, size_t bytes, cudaStream_t st);
// psi = scale * forward transform of a complex or real field
addft_status d64_from_real(const PlanDev &pd, int nbatch, const void *in, bool in_real, double scale, double2 *psi,
                           void *work, size_t bytes, cudaStream_t st);

}  // namespace addft
