// Batched FTLM kernels of one sector on planes of two chains (planes.cu).
//
// A group of `planes` planes is a contiguous block vector W[plane][state] of float4: plane p holds chains 2p and 2p+1
// of the group in complex64, in the sector's spin-ordered basis.  Per-chain scalars (st, alpha, beta, used) are
// indexed by the chain within the group; the arrays have a stride of 32 chains, so a caller that runs the 32 chains
// of a block in several groups passes pointers offset by the group's first chain.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace ftlm_b200 {

// Planes that one group of a sector runs at once (of `planes`): enough that a vector of the group has 256 MB, and two
// where there are two, which the row pass takes together.  More planes share the launches and the scalar kernels of a
// step (4x3 (6,6), 80 steps of 16 planes: 69.6 ms in one group, 83.6 ms in groups of 2, 109.9 ms plane by plane, although
// the vectors of those stay in L2); past that size they bring nothing (4x4 (5,6): 170 to 172 ms for any group) and cost
// memory, all 16 planes of 4x4 (8,8) 127 GB instead of 16.
int pl_group(int64_t dim, int planes);

// Per-chain scalar state and results of a group (kBt* fields of batched.cuh, stride 32), the partial sums of one step
// (kPlPartialDoubles) and two tiny-entry flags.
struct PlaneState {
  double* st;
  double* partial;
  double* alpha;  // [M][32]
  double* beta;
  int* used;
  int* flags;
};
constexpr int64_t kPlMaxBlocks = 2560;
constexpr int64_t kPlPartialDoubles = kPlMaxBlocks * 32 * 2;

// W <- complex64 Philox start vectors (chain c of the group: key seed + c*100003), norms -> scalar state; the flags
// are cleared here.
cudaError_t pl_start(const DevSector& S, float4* W, int planes, unsigned seed, const PlaneState& z, cudaStream_t s);
// One Lanczos step k of the group's chains: Y <- H W_k, z, W_{k+1} (into Y), beta_k.  The gauge basis has the spectrum
// of the original one and the start vectors are G r, so alpha/beta are those of the original.
cudaError_t pl_step(const DevSector& S, const float4* Wk, const float4* Wkm1, float4* Y, int planes, int k,
                    const PlaneState& z, cudaStream_t s);
// Y = (G H G) X for any number of planes, without Lanczos bookkeeping; zero_flag points to an int 0 (no small-entry
// filter).
cudaError_t pl_apply(const DevSector& S, const float4* X, float4* Y, int planes, int* zero_flag, cudaStream_t s);

}  // namespace ftlm_b200
