// Complex64 Lanczos of a momentum block (batched.cu): 32 chains of the block per vector; the chains' scalars, which the
// planes of a sector (planes.cu) share.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"
#include "orbit.cuh"

namespace ftlm_b200 {

constexpr int kBtBlocksPerSm = 5;
constexpr int kBtBlocks = kBtBlocksPerSm * 148;  // fixed persistent grid: deterministic reductions
constexpr int kBtChains = 32;   // chains per block vector (one warp lane each)
// Per-chain scalar state, st[field * 32 + chain] (doubles).
constexpr int kBtSin = 0;     // 1 / beta_{k-1}: scale of H W_k
constexpr int kBtC1r = 1;     // z / beta_{k-1} (coefficient of W_k), real and imaginary parts
constexpr int kBtC1i = 2;
constexpr int kBtC2 = 3;      // beta_{k-1} / beta_{k-2} (coefficient of W_{k-1})
constexpr int kBtActive = 4;  // 1 while the chain has not broken down
constexpr int kBtFields = 8;
constexpr int kBtPartialDoubles = kBtBlocks * kBtChains * 2;

struct Neu {  // Neumaier-compensated FP64 sum
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double v) {
    const double t = s + v;
    c += (fabs(s) >= fabs(v)) ? ((s - t) + v) : ((v - t) + s);
    s = t;
  }
  __device__ __forceinline__ double value() const { return s + c; }
};

// |v|^2 < 1e-28 in FP32 (squares below FLT_MIN flush towards zero, which is still below the bound).
__device__ __forceinline__ bool tinyf(float2 v) { return fmaf(v.x, v.x, v.y * v.y) < 1e-28f; }

// Totals of nblocks partial sums per chain (partial[(block * 32 + chain) * values]) and the recurrence's scalars for
// the first `lanes` chains.  mode 0: start norms; 1: dot products, alpha_k; 2: norms, beta_k and breakdown.  scaled:
// the dot products are of H q_k (complex128 chains) instead of H W_k.  clear (mode 1): set to 0.  live (or null): counts the
// chains that have not ended, from 0 before mode 0.
void bt_scalars(const double* partial, int nblocks, int mode, int k, int lanes, bool scaled, double* st, double* alpha,
                double* beta, int* used, int* clear, int* live, cudaStream_t s);

// W <- complex64 Philox start vectors of the block's representatives (chain r: key seed + r*100003), norms -> scalar
// state.  flags: 2 ints (tiny-entry flags of the current and next vector, cleared here).
cudaError_t bt_start(float2* W, int64_t dim, unsigned seed, double* st, double* partial, int* used, int* flags,
                     cudaStream_t s);

// One Lanczos step k of 32 chains of an orbit momentum block (block vectors over its dk representatives, 256 bytes
// each): Y <- H_K W_k, z, W_{k+1} (into Y), beta_k; alpha/beta [M][32].  Needs the sector's max up-degree <= 120 and at
// most 256 sources per representative.
cudaError_t bt_orbit_step(const OrbitApplyDev& A, const float2* Wk, const float2* Wkm1, float2* Y, int k, double* st,
                          double* partial, double* alpha, double* beta, int* used, int* flags, cudaStream_t s);

}  // namespace ftlm_b200
