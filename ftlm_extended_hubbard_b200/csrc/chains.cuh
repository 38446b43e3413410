// Fused Lanczos of many small sectors (chains.cu): one block per plane of one sector runs all M steps of the
// src/lanczos.cpp:180-205 recurrence on its own vectors, so a whole sweep of small sectors is a few launches instead of
// M times five kernels per sector.  A plane is two complex64 chains or one complex128 chain of a sector.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace ftlm_b200 {

struct ChainDesc {
  int sector;          // index into the DevSector array
  int out;             // first row of alpha/beta/used/scale written by this plane
  int chains;          // chains of the plane that are wanted (a plane's second complex64 chain may not be)
  unsigned seed;       // Philox key of its first chain
  int rows;            // rows staged at once: all of them where the vector fits shared memory
  int64_t off;         // first element of its three vectors of chain_elements() in the scratch
  int64_t init;        // first element of its start vector in ChainLaunch::init
  int64_t store;       // first element of its stored vectors, and their distance
  int64_t store_step;
};

// Planes of one size class, staging and form of the sectors' gauge tables.
struct ChainLaunch {
  const DevSector* sectors;
  const ChainDesc* descs;
  int blocks;
  int size;             // chain_class of the sectors
  bool smem;            // the gathered vector is in shared memory
  bool phase;           // the tables' coefficients have the phase form
  bool xor_real;        // and the XOR form
  size_t smem_bytes;    // largest chain_smem_bytes of the sectors
  int M;
  void* scratch;
  const double2* init;  // complex128 start vectors, not normalised, in the sector's order; null: Philox
  double* alpha;        // [rows][M], zero-filled by the caller; entries of a chain that broke down at step k: k + 1
  double* beta;         // (beta: k)
  int* used;            // [rows]
  double* scale;        // [rows][M] or null: norm of the stored vector k (1 where the chain has ended)
  void* store;          // or null: the unnormalised vectors W_k in the spin-ordered basis, for a gradient's replay
};

int chain_class(int64_t dim);
// Elements of one vector: rows have a pitch of Dd + 8.
inline size_t chain_elements(const DevSector& S) { return static_cast<size_t>(S.Du) * static_cast<size_t>(S.Dd + 8); }
// Shared memory of a plane of the sector with `rows` rows staged, and the rows that are: all of them where they fit, else
// as many as fit half of it (0: not even one).
size_t chain_smem_bytes(const DevSector& S, bool c64, bool phase, int rows);
int chain_rows(const DevSector& S, bool c64, bool phase);
cudaError_t chains_lanczos(const ChainLaunch& L, bool c64, cudaStream_t st);

}  // namespace ftlm_b200
