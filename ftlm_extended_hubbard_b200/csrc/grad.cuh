// Krylov moments for the FTLM parameter gradient (grad.cu).
//
// For one chain c with stored (unnormalised) Lanczos vectors W_0..W_{n-1} and a real symmetric
// weight matrix K'_c (scales 1/(b_i b_l) folded in), the kernel returns per chain
//   m0 = sum_il K'_il <W_i| D |W_l>,  m1 = sum_il K'_il <W_i| P |W_l>,  m2 = sum_il K'_il <A W_i|W_l>
// with D = number of doubly occupied sites, P = sum over neighbour pairs of n_i n_j (both
// diagonal, evaluated from the sector tables) and A W_i supplied by the caller (the t' hopping
// operator applied to each W_i).  Vectors are planes over the sector's states: two complex64 chains
// (the batched path) or one complex128 chain (the plain path) per element; plane p of vector i starts
// at W + i * vstride + p * pstride.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace ftlm_b200 {

constexpr int64_t kGradMaxBlocks = 2048;

// Kp: [chains][ld][ld]; used [chains]: the vectors of each chain (those past a plane's longest chain are not read).
// partial: scratch of kGradMaxBlocks * chains * 3 doubles; out: [chains][3].  Shared memory: the ld vectors' entries of a
// block of 32 to 256 states; cudaErrorInvalidValue when that does not fit.
cudaError_t grad_moments(const DevSector& S, const float4* W, const float4* AW, int64_t vstride, int64_t pstride,
                         int chains, const double* Kp, const int* used, int ld, double* partial, double* out,
                         cudaStream_t st);
cudaError_t grad_moments(const DevSector& S, const double2* W, const double2* AW, int64_t vstride, int64_t pstride,
                         int chains, const double* Kp, const int* used, int ld, double* partial, double* out,
                         cudaStream_t st);

}  // namespace ftlm_b200
