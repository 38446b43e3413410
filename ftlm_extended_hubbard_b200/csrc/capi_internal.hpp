// Shared host-side state of the C ABI (capi*.cu): error reporting, device buffers, the Lanczos
// driver, the sector handle and the batched-path workspaces.  Internal; not installed.
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <limits>
#include <memory>
#include <mutex>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../../include/ftlm_gpu.h"
#include "batched.cuh"
#include "chains.cuh"
#include "grad.cuh"
#include "hv.cuh"
#include "lazy_stream.hpp"
#include "orbit.cuh"
#include "planes.cuh"
#include "pool.hpp"
#include "plan.hpp"
#include "symeig.cuh"
#include "tridiag.hpp"

namespace ftlm_b200 {
namespace capi {

// Records msg for ftlm_gpu_last_error() (per host thread) and returns code.
int fail(int code, const std::string& msg);
// The error code of the exception in flight (in a handler): no exception crosses the C ABI.
int caught() noexcept;

#define CU_TRY(expr)                                                                                     \
  do {                                                                                                   \
    cudaError_t e_ = (expr);                                                                             \
    if (e_ != cudaSuccess)                                                                               \
      return ::ftlm_b200::capi::fail(e_ == cudaErrorMemoryAllocation ? FTLM_ERR_NOMEM : FTLM_ERR_CUDA,   \
                  std::string(#expr) + ": " + cudaGetErrorString(e_));                                   \
  } while (0)

// Device buffer that frees itself.
struct DevBuf {
  void* p = nullptr;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { free(); }
  void free() {
    if (p) cudaFree(p);
    p = nullptr;
  }
  cudaError_t alloc(size_t bytes) {
    free();
    cudaError_t e = cudaMalloc(&p, std::max<size_t>(bytes, 16));
    if (e == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      pool_trim();
      e = cudaMalloc(&p, std::max<size_t>(bytes, 16));
    }
    return e;
  }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// Plans of a sweep's sectors by N_up and by N_down, whose tables of that species the other sectors copy (build_plan).
struct PlanParts {
  explicit PlanParts(int n) : up(static_cast<size_t>(n) + 1), dn(static_cast<size_t>(n) + 1) {}
  std::vector<std::shared_ptr<const SectorPlan>> up, dn;
  static const SectorPlan* find(const std::vector<std::shared_ptr<const SectorPlan>>& v, int k) {
    return k >= 0 && k < static_cast<int>(v.size()) ? v[static_cast<size_t>(k)].get() : nullptr;
  }
  void keep(const SectorPlan& P) {
    auto& u = up[static_cast<size_t>(P.nu)];
    auto& d = dn[static_cast<size_t>(P.nd)];
    if (u && d) return;
    auto copy = std::make_shared<const SectorPlan>(P);
    if (!u) u = copy;
    if (!d) d = copy;
  }
};

// Reference start vector (src/lanczos.cpp:140-175): re, im from std::normal_distribution<double>
// over std::mt19937(seed), normalised with a serial sum; falls back to e_0 when ||q|| < 1e-18.
void reference_start(int64_t dim, unsigned seed, std::vector<std::complex<double>>* q);
// R such vectors before normalisation (seed + r*100003), drawn by several threads.
void reference_normals(int64_t dim, int R, unsigned seed, std::vector<std::complex<double>>* out);

struct LanczosWs {
  int64_t n = 0;
  DevBuf q, qp, w, scratch;
  cudaError_t ensure(int64_t dim) {
    if (n == dim && q.p) return cudaSuccess;
    n = dim;
    cudaError_t e;
    if ((e = q.alloc(dim * sizeof(double2))) != cudaSuccess) return e;
    if ((e = qp.alloc(dim * sizeof(double2))) != cudaSuccess) return e;
    if ((e = w.alloc(dim * sizeof(double2))) != cudaSuccess) return e;
    return scratch.alloc(kScratchDoubles * sizeof(double));
  }
};

// Generic Lanczos loop around an operator on device vectors; the recurrence of
// src/lanczos.cpp:180-205 with alpha, ||w||^2 read back once per step for the breakdown test.
template <class Apply>
int run_lanczos(int64_t dim, Apply&& apply, LanczosWs& ws, int max_steps, unsigned seed, int start_mode,
                cudaStream_t st, std::vector<double>* alpha, std::vector<double>* beta, double2* store = nullptr) {
  alpha->clear();
  beta->clear();
  if (dim <= 0 || max_steps <= 0) return FTLM_OK;
  CU_TRY(ws.ensure(dim));
  double* scr = ws.scratch.as<double>();
  if (start_mode == FTLM_START_PHILOX) {
    CU_TRY(lz_philox_start(ws.q.as<double2>(), dim, seed, scr, st));
    CU_TRY(lz_normalise_start(ws.q.as<double2>(), dim, scr, st));
  } else if (start_mode == FTLM_START_REFERENCE) {
    std::vector<std::complex<double>> h;
    reference_start(dim, seed, &h);
    CU_TRY(cudaMemcpyAsync(ws.q.p, h.data(), dim * sizeof(double2), cudaMemcpyHostToDevice, st));
    CU_TRY(cudaStreamSynchronize(st));
  } else {
    return fail(FTLM_ERR_INVALID, "unknown start_mode");
  }
  double2* q = ws.q.as<double2>();
  double2* qp = ws.qp.as<double2>();
  double2* w = ws.w.as<double2>();
  double bprev = 0.0;
  double res[4];
  for (int k = 0; k < max_steps; ++k) {
    if (store)  // keep q_k (gradient replay)
      CU_TRY(cudaMemcpyAsync(store + static_cast<int64_t>(k) * dim, q, dim * sizeof(double2), cudaMemcpyDeviceToDevice,
                             st));
    const int rc = apply(q, w, st);
    if (rc != FTLM_OK) return rc;
    CU_TRY(lz_dotc(q, w, dim, scr, st));
    CU_TRY(lz_update(w, q, qp, bprev, k > 0, dim, scr, st));
    // Next q into the old q_prev buffer (harmless if this step turns out to be the last).
    CU_TRY(lz_scale_by_norm(qp, w, dim, scr, st));
    CU_TRY(cudaMemcpyAsync(res, scr + kResZ, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    const double a_k = res[0];
    const double nw2 = res[2];
    alpha->push_back(a_k);
    if (nw2 < 1e-24) break;
    const double b_k = std::sqrt(nw2);
    beta->push_back(b_k);
    std::swap(q, qp);  // q_prev <- q ; q <- w / b_k (already written)
    bprev = b_k;
  }
  return FTLM_OK;
}

}  // namespace capi
}  // namespace ftlm_b200

namespace ftlm_b200 {
namespace capi {

// Vectors and scalars of Lanczos chains on planes (or of a momentum block's 32 chains), kept between calls.
struct BtWs {
  size_t cap = 0;
  int mcap = 0;
  int64_t icap = 0;
  PoolBuf buf[3], st, partial, items, alpha, beta, used, flags;
  // three vectors of `bytes` each, the scalars of 32 chains of M steps, n_items partial sums of the column pass's items
  cudaError_t ensure(size_t bytes, int M, int64_t n_items = 0) {
    cudaError_t e = cudaSuccess;
    if (bytes > cap) {
      release();
      for (auto& b : buf)
        if ((e = b.alloc(bytes)) != cudaSuccess) return e;
      cap = bytes;
    }
    if (n_items > icap) {
      icap = 0;
      if ((e = items.alloc(static_cast<size_t>(n_items) * sizeof(double))) != cudaSuccess) return e;
      icap = n_items;
    }
    if (!st.p) {
      if ((e = partial.alloc(std::max<int64_t>(kBtPartialDoubles, kPlPartialDoubles) * sizeof(double))) != cudaSuccess) return e;
      if ((e = used.alloc(kBtChains * sizeof(int))) != cudaSuccess) return e;
      if ((e = flags.alloc(kPlFlags * sizeof(int))) != cudaSuccess) return e;
      if ((e = st.alloc(kBtFields * kBtChains * sizeof(double))) != cudaSuccess) return e;
    }
    if (M > mcap) {
      mcap = 0;
      if ((e = alpha.alloc(static_cast<size_t>(M) * kBtChains * sizeof(double))) != cudaSuccess) return e;
      if ((e = beta.alloc(static_cast<size_t>(M) * kBtChains * sizeof(double))) != cudaSuccess) return e;
      mcap = M;
    }
    return e;
  }
  // the scalar state of a group whose first chain is c0 of the block
  PlaneState state(int c0) const {
    return PlaneState{st.as<double>() + c0,   partial.as<double>(),  items.as<double>(),   alpha.as<double>() + c0,
                      beta.as<double>() + c0, used.as<int>() + c0, flags.as<int>()};
  }
  void release() {  // before growing, too
    for (auto& b : buf) b.free();
    cap = 0;
  }
  void free_all(bool idle) {
    for (PoolBuf* b : {&buf[0], &buf[1], &buf[2], &st, &partial, &items, &alpha, &beta, &used, &flags}) b->free(idle);
    cap = 0;
    mcap = 0;
    icap = 0;
  }
};

}  // namespace capi
}  // namespace ftlm_b200

struct OrbitSectorData;

// The opaque C handle: a sector plan, its device tables and per-sector workspaces.
struct ftlm_sector {
  ftlm_b200::SectorPlan plan;
  int Lx = 0, Ly = 0;  // lattice (sectors built from ftlm_params); 0 when built from hop lists
  std::shared_ptr<OrbitSectorData> orbit_data;
  bool on_device = false;
  int device = -1;
  ftlm_b200::DevSector dev{};
  void* tables = nullptr;  // one block of the pool
  size_t tables_bytes = 0;
  ftlm_b200::capi::BtWs planes;  // vectors and scalars of its complex128 Lanczos chains
  int apply_path = 0;    // 0 auto, 1 generic, 2 rows+cols, 3 rows (register coefficient classes)+cols
  bool pinned = false;   // apply_path comes from ftlm_gpu_set_apply_path: the chains keep to it too
  bool use_once = true;  // H v in one pass where it can be (until a path is set)
  int cols_variant = 0;  // column slab 256/128/512 (0/1/2); 3/4/5: the same over the packed up list (path 3)
  ftlm_b200::capi::LanczosWs ws;
  ftlm_b200::capi::DevBuf hx, hy;  // staging for the host-buffer apply
  ftlm_b200::capi::LazyStream stream;
  ~ftlm_sector() {
    if (!tables) return;
    // as a free would wait: a caller's H v may still read the tables
    const bool idle = ftlm_b200::capi::device_idle(device);
    ftlm_b200::capi::pool_give(tables, tables_bytes, idle);
    planes.free_all(idle);
  }
  // Kernel choice for H·v: 1 = generic gather; 2 = row pass with the per-row coefficient table +
  // column-slab pass over the CSR up list; 3 = row pass in the gauge basis (register-held real
  // coefficients) + column-slab pass, over the packed up list when cols_variant >= 3 and the sector
  // has one.  Automatic: one pass (hv_once) for small sectors, else 3, else 2, else 1.
  bool path_available(int path) const {
    if (path == 1) return true;
    if (path == 3 && !dev.dn_g.ent) return false;
    return (path == 2 || path == 3) && ftlm_b200::hv_fast_path_ok(dev_for(path), plan.max_up_deg);
  }
  int effective_path() const {
    if (apply_path >= 1 && apply_path <= 3) return (apply_path == 3 && !dev.dn_g.ent) ? 2 : apply_path;
    if (path_available(3)) return 3;
    return path_available(2) ? 2 : 1;
  }
  // The device view a launch of `path` with column variant cv uses (the row pass reads dn_g on path
  // 3 only, the column pass up_pk on path 3 with cv >= 3 only).
  ftlm_b200::DevSector dev_for(int path, int cv = -1) const {
    ftlm_b200::DevSector d = dev;
    if (cv < 0) cv = cols_variant;
    if (path != 3) d.dn_g.ent = nullptr;
    if (path != 3 || cv < 3) d.up_pk = nullptr;
    return d;
  }
  bool once() const { return use_once && ftlm_b200::hv_once_ok(dev, plan.max_up_deg); }
  bool cols_chosen = false;  // cols_variant was set or timed: the slab of the complex128 chains on planes, too
  // How complex128 chains run: all steps in one kernel, on planes (gauge row pass + column slabs, so also where path 3 is
  // pinned), or step by step on apply().
  enum class Chains { fused, planes, steps };
  Chains chains(int R) const;  // of R of them
  ftlm_b200::DevSector planes_dev() const {
    ftlm_b200::DevSector d = dev;
    if (cols_chosen) d.bt_cols = cols_variant % 3;
    return d;
  }
  int apply(const double2* x, double2* y, cudaStream_t st) {
    if (once()) {
      CU_TRY(ftlm_b200::hv_launch_once(dev, x, y, st));
      return FTLM_OK;
    }
    const int path = effective_path();
    const ftlm_b200::DevSector d = dev_for(path);
    if (path >= 2 && ftlm_b200::hv_rows_smem_bytes(d) > 227 * 1024)
      return ftlm_b200::capi::fail(FTLM_ERR_UNSUPPORTED, "row pass does not fit in shared memory for this sector");
    CU_TRY(ftlm_b200::hv_launch(d, x, y, path == 3 ? 2 : path, st, cols_variant));
    return FTLM_OK;
  }
};

namespace ftlm_b200 {
namespace capi {

int need_device(const ftlm_sector* s);
// Sectors that go with the scope.
struct OwnedSectors {
  std::vector<ftlm_sector*> v;
  OwnedSectors() = default;
  OwnedSectors(const OwnedSectors&) = delete;
  OwnedSectors& operator=(const OwnedSectors&) = delete;
  ~OwnedSectors() {
    for (ftlm_sector* s : v) delete s;
  }
};
// ftlm_gpu_sector_create, with the tables that a sweep's sectors share (parts may be null).
int sector_create(const ftlm_params* p, int n_up, int n_dn, PlanParts* parts, ftlm_sector** out);

// ---- batched complex64 path (capi_batched.cu) ------------------------------------------------
extern BtWs g_bt;
extern std::mutex g_bt_mu;

// Krylov vector store of the gradient replay (grows to the largest piece seen), kept between calls.
struct GradWs {
  DevBuf Q, AQ, flag;
  size_t qcap = 0, acap = 0;
  cudaError_t grow(DevBuf& b, size_t& cap, size_t bytes) {
    if (bytes <= cap && b.p) return cudaSuccess;
    cap = 0;
    const cudaError_t e = b.alloc(bytes);
    if (e == cudaSuccess) cap = bytes;
    return e;
  }
  void release() {
    Q.alloc(0);
    AQ.alloc(0);
    qcap = acap = 0;
  }
};
extern GradWs g_grad;


// Runs ceil(R/32) blocks of 32 chains of a momentum block of dim states, the M steps of a block as one graph; A/B
// [R][M] (beta zero-padded), used [R].
template <class Step>
int bt_run_chains_impl(int64_t dim, cudaStream_t st, Step&& step, int R, int M, unsigned seed, std::vector<double>* A,
                       std::vector<double>* B, std::vector<int>* used) {
  A->assign(static_cast<size_t>(R) * M, 0.0);
  B->assign(static_cast<size_t>(R) * M, 0.0);
  used->assign(static_cast<size_t>(R), 0);
  std::lock_guard<std::mutex> lock(g_bt_mu);
  CU_TRY(g_bt.ensure(static_cast<size_t>(dim) * kBtChains * sizeof(float2), M));
  float2* bufs[3] = {g_bt.buf[0].as<float2>(), g_bt.buf[1].as<float2>(), g_bt.buf[2].as<float2>()};
  double* sd = g_bt.st.as<double>();
  double* part = g_bt.partial.as<double>();
  double* al = g_bt.alpha.as<double>();
  double* be = g_bt.beta.as<double>();
  int* us = g_bt.used.as<int>();
  int* fl = g_bt.flags.as<int>();
  std::vector<double> ha(static_cast<size_t>(M) * kBtChains), hb(static_cast<size_t>(M) * kBtChains);
  std::vector<int> hu(kBtChains);
  for (int blk = 0; blk * kBtChains < R; ++blk) {
    const unsigned seed_b = seed + static_cast<unsigned>(blk * kBtChains) * 100003u;
    CU_TRY(cudaMemsetAsync(al, 0, static_cast<size_t>(M) * kBtChains * sizeof(double), st));
    CU_TRY(cudaMemsetAsync(be, 0, static_cast<size_t>(M) * kBtChains * sizeof(double), st));
    CU_TRY(bt_start(bufs[0], dim, seed_b, sd, part, us, fl, st));
    cudaGraph_t graph = nullptr;
    CU_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    float2 *wk = bufs[0], *y = bufs[1], *wkm1 = bufs[2];
    cudaError_t ce = cudaSuccess;
    for (int k = 0; k < M && ce == cudaSuccess; ++k) {
      ce = step(wk, wkm1, y, k, sd, part, al, be, us, fl);
      float2* t = wkm1;
      wkm1 = wk;
      wk = y;
      y = t;
    }
    const cudaError_t ee = cudaStreamEndCapture(st, &graph);
    if (ce != cudaSuccess || ee != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      return fail(FTLM_ERR_CUDA, std::string("batched step capture: ") +
                                     cudaGetErrorString(ce != cudaSuccess ? ce : ee));
    }
    cudaGraphExec_t exec = nullptr;
    ce = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) return fail(FTLM_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(ce));
    ce = cudaGraphLaunch(exec, st);
    const cudaError_t se = cudaStreamSynchronize(st);
    cudaGraphExecDestroy(exec);
    if (ce != cudaSuccess || se != cudaSuccess)
      return fail(FTLM_ERR_CUDA, std::string("batched steps: ") + cudaGetErrorString(ce != cudaSuccess ? ce : se));
    CU_TRY(cudaMemcpy(ha.data(), al, ha.size() * sizeof(double), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(hb.data(), be, hb.size() * sizeof(double), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(hu.data(), us, hu.size() * sizeof(int), cudaMemcpyDeviceToHost));
    for (int r = 0; r < kBtChains; ++r) {
      const int ch = blk * kBtChains + r;
      if (ch >= R) break;
      (*used)[static_cast<size_t>(ch)] = hu[static_cast<size_t>(r)];
      for (int k = 0; k < M; ++k) {
        (*A)[static_cast<size_t>(ch) * M + k] = ha[static_cast<size_t>(k) * kBtChains + r];
        (*B)[static_cast<size_t>(ch) * M + k] = hb[static_cast<size_t>(k) * kBtChains + r];
      }
    }
  }
  return FTLM_OK;
}

// Per-chain log quadrature and energy (layout of ftlm_gpu_tridiag_quadrature) with the reference's
// rotation-capped Jacobi (converged == false) or the converged GPU eigen-decomposition.
int chain_quadrature(const double* A, const double* B, const int* n, int nc, int ld, const double* bts, int n_bt,
                     double* lq, double* eq, bool converged);
// The quadrature of the complex128 sector path (ftlm_gpu_set_quadrature; the reference's Jacobi by default).
bool plain_quadrature_converged();
// ftlm_gpu_ftlm_sector with an explicit quadrature choice.
int plain_sector_ftlm(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed, int start_mode,
                      bool converged, double* lnz, double* energy);

// The fused chains of many sectors (capi_chains.cu), results on the device: rows [sector][chain] of alpha/beta [M]
// (zero-padded), steps used and, with keep_scale, the norms of the stored vectors.
struct ChainRun {
  Scratch mem;
  double *alpha = nullptr, *beta = nullptr, *scale = nullptr;
  int* used = nullptr;
};
// c64: complex64 chains (Philox starts), else complex128.  store: the chains' vectors W_k go to store + store_base[i] +
// (k * planes + p) * dim for plane p (two chains of complex64, one of complex128) of sector i.
int chains_run(const std::vector<ftlm_sector*>& secs, int R, int M, unsigned seed, int start_mode, bool c64,
               ChainRun* run, void* store = nullptr, const std::vector<int64_t>* store_base = nullptr,
               bool keep_scale = false);
// ln Z and energy of each sector on the temperature grid, [sector][n_bt].
int chains_ftlm(const std::vector<ftlm_sector*>& secs, int R, int M, unsigned seed, int start_mode, bool c64,
                const double* bts, int n_bt, bool converged, double* lnz, double* energy);
// The same into rows out_idx[i] of lnz_s / e_s.
int fused_sectors_ftlm(const std::vector<ftlm_sector*>& secs, const std::vector<int>& out_idx, int R, int M,
                       unsigned seed, int start_mode, bool c64, const double* bts, int n_bt, double* lnz_s, double* e_s,
                       bool converged);

// Whether a single sector's own chains run fused, by the lanes that a step of its block has to go through.  A step on planes
// takes 27 us for sectors of any shape up to 50,000 states; fused, 28 us at 3,456 lanes, 37 at 6,336, 55 at 8,064 (3x3
// (2,3), 4x3 (2,2), 3x3 (3,3), complex128).  Sectors of one row are slower on planes (47 us at 5,005 strings, 58 at 8,008; fused 31 and
// 48).  A vector that is not staged whole is read from the block's scratch: 4x4 (6,0), 8,008 rows of one string and 8 of padding,
// 275 us a step fused, 52 on planes.
inline bool fused_alone(const DevSector& S) {
  const int64_t lanes = S.Dd <= 16 ? S.Du / (32 / S.Dd) * 32 : S.Du * ((S.Dd + 31) / 32 * 32);
  return lanes <= (S.Du == 1 ? 8192 : 4096) && chain_rows(S, false, false) == S.Du;
}
// Sectors with very few strings of one species and many of the other: few or short work items for the passes on planes.
inline bool thin_sector(const DevSector& S) { return std::min(S.Du, S.Dd) <= 16 && std::max(S.Du, S.Dd) > 10000; }

}  // namespace capi
}  // namespace ftlm_b200

inline ftlm_sector::Chains ftlm_sector::chains(int R) const {
  if (!pinned && ftlm_b200::capi::fused_alone(dev)) return Chains::fused;
  // one chain of a thin sector whose H v is the generic kernel (by rule or by timing): 4x4 (0,8) 64 us a step, 82 on planes;
  // (8,1) 66 and 76; (1,8) timed 78 and 88.  From two chains on the planes share their launches: 82 us a step of both.
  if (!pinned && R == 1 && ftlm_b200::capi::thin_sector(dev) && effective_path() == 1 && !once()) return Chains::steps;
  if ((!pinned || effective_path() == 3) && ftlm_b200::pl_fits(dev, plan.max_up_deg)) return Chains::planes;
  return Chains::steps;
}

namespace ftlm_b200 {
namespace capi {

// Largest sector that joins the fused launch of a sweep; a larger one fills the GPU by itself.
constexpr int64_t kFusedSweepMax = 1 << 14;

// R complex128 chains of one sector (seed + r*100003) in groups of planes (planes.cu; pl_fits), layout as below.
int planes_lanczos(ftlm_sector* s, int R, int M, unsigned seed, int start_mode, std::vector<double>* A,
                   std::vector<double>* B, std::vector<int>* used);

// The complex64 chains of one sector in groups of planes (planes.cu), alpha/beta [R][M] (beta zero-padded), used [R].
int bt_run_chains(ftlm_sector* s, int R, int M, unsigned seed, std::vector<double>* A, std::vector<double>* B,
                  std::vector<int>* used);

}  // namespace capi
}  // namespace ftlm_b200
