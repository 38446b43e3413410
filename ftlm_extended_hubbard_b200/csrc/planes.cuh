// Lanczos chains of one sector on planes of two complex64 chains or one complex128 chain (planes.cu).
//
// A group of `planes` planes is a contiguous block vector W[plane][state]: plane p holds chains 2p and 2p+1 of the group in
// complex64 (float4), or chain p in complex128 (double2), in the sector's spin-ordered basis.  Per-chain scalars (st, alpha, beta, used) are
// indexed by the chain within the group; the arrays have a stride of 32 chains, so a caller that runs the 32 chains
// of a block in several groups passes pointers offset by the group's first chain.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace ftlm_b200 {

// Planes of a sector that one group runs at once (of `planes`): enough that a vector of the group has 256 MB, and two where
// the row pass takes two together.  More planes share the launches and the scalar kernels of a step (4x3
// (6,6), 80 steps of 16 planes: 69.6 ms in one group, 83.6 ms in groups of 2, 109.9 ms plane by plane, although the vectors of
// those stay in L2); past that size they bring nothing (the column pass then loses the slab's locality: 4x4 (5,6), 170 ms
// plane by plane, 177 in groups of 2) and cost memory, all 16 planes of 4x4 (8,8) 127 GB instead of 8.
int pl_group(const DevSector& S, bool c64, int planes);

// Per-chain scalar state and results of a group (kBt* fields of batched.cuh, stride 32), the partial sums of one step
// (kPlPartialDoubles; of large planes also one per item of the column pass, pl_items_doubles), two tiny-entry flags and the
// number of chains that have not ended (kPlFlags ints).
struct PlaneState {
  double* st;
  double* partial;
  double* items;
  double* alpha;  // [M][32]
  double* beta;
  int* used;
  int* flags;
};
int64_t pl_items_doubles(const DevSector& S, bool c64, int planes);
constexpr int kPlFlags = 3;
constexpr int64_t kPlMaxBlocks = 2560;
constexpr int64_t kPlPartialDoubles = kPlMaxBlocks * 32 * 2;

// Whether complex128 chains of the sector run here: a gauge table, a row that fits shared memory, at most 128 up sources.
bool pl_fits(const DevSector& S, int max_up_deg);
// W <- Philox start vectors (chain c of the group: key seed + c*100003) or, with `given`, the vectors that are in W (in the
// sector's order, not normalised) in the gauge basis; norms -> scalar state.  The flags are cleared here.
cudaError_t pl_start(const DevSector& S, float4* W, int planes, unsigned seed, const PlaneState& z, cudaStream_t s);
cudaError_t pl_start(const DevSector& S, double2* W, int planes, unsigned seed, bool given, const PlaneState& z,
                     cudaStream_t s);
// One Lanczos step k of the group's chains: Y <- H W_k, z, W_{k+1} (into Y), beta_k.  The gauge basis has the spectrum
// of the original one and the start vectors are G r, so alpha/beta are those of the original.
cudaError_t pl_step(const DevSector& S, const float4* Wk, const float4* Wkm1, float4* Y, int planes, int k,
                    const PlaneState& z, cudaStream_t s);
cudaError_t pl_step(const DevSector& S, const double2* Wk, const double2* Wkm1, double2* Y, int planes, int k,
                    const PlaneState& z, cudaStream_t s);
// Y = (G H G) X for any number of planes, without Lanczos bookkeeping; flag: an int of scratch.  (complex64: no small-entry
// filter.)
cudaError_t pl_apply(const DevSector& S, const float4* X, float4* Y, int planes, int* flag, cudaStream_t s);
cudaError_t pl_apply(const DevSector& S, const double2* X, double2* Y, int planes, int* flag, cudaStream_t s);

}  // namespace ftlm_b200
