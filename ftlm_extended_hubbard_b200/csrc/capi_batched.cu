// C ABI of the batched complex64 FTLM of a sector (planes.cu): blocks of 32 chains in groups of planes, the M Lanczos
// steps of a block launched without host synchronisation.
#include <map>

#include "capi_internal.hpp"

using namespace ftlm_b200;
using namespace ftlm_b200::capi;

namespace ftlm_b200 {
namespace capi {

BtWs g_bt;
std::mutex g_bt_mu;
GradWs g_grad;

int bt_run_chains(ftlm_sector* s, int R, int M, unsigned seed, std::vector<double>* A, std::vector<double>* B,
                  std::vector<int>* used) {
  A->assign(static_cast<size_t>(R) * M, 0.0);
  B->assign(static_cast<size_t>(R) * M, 0.0);
  used->assign(static_cast<size_t>(R), 0);
  const int64_t dim = s->plan.dim;
  const DevSector& S = s->dev;
  cudaStream_t st = s->stream;
  const int group = pl_group(S, true, (std::min(R, kBtChains) + 1) / 2);
  std::lock_guard<std::mutex> lock(g_bt_mu);
  CU_TRY(g_bt.ensure(static_cast<size_t>(group) * dim * sizeof(float4), M, pl_items_doubles(S, true, group)));
  const size_t tab = static_cast<size_t>(M) * kBtChains * sizeof(double);
  std::vector<double> ha(static_cast<size_t>(M) * kBtChains), hb(static_cast<size_t>(M) * kBtChains);
  std::vector<int> hu(kBtChains);
  for (int blk = 0; blk * kBtChains < R; ++blk) {
    const int nc = std::min(kBtChains, R - blk * kBtChains), planes = (nc + 1) / 2;
    CU_TRY(cudaMemsetAsync(g_bt.alpha.p, 0, tab, st));
    CU_TRY(cudaMemsetAsync(g_bt.beta.p, 0, tab, st));
    for (int p0 = 0; p0 < planes; p0 += group) {
      const int np = std::min(group, planes - p0);
      const PlaneState z = g_bt.state(2 * p0);
      float4 *wk = g_bt.buf[0].as<float4>(), *y = g_bt.buf[1].as<float4>(), *wkm1 = g_bt.buf[2].as<float4>();
      CU_TRY(pl_start(S, wk, np, seed + static_cast<unsigned>(blk * kBtChains + 2 * p0) * 100003u, z, st));
      for (int k = 0; k < M; ++k) {
        CU_TRY(pl_step(S, wk, wkm1, y, np, k, z, st));
        float4* t = wkm1;
        wkm1 = wk;
        wk = y;
        y = t;
      }
    }
    CU_TRY(cudaMemcpyAsync(ha.data(), g_bt.alpha.p, tab, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hb.data(), g_bt.beta.p, tab, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hu.data(), g_bt.used.p, hu.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    for (int r = 0; r < nc; ++r) {
      const size_t ch = static_cast<size_t>(blk * kBtChains + r);
      (*used)[ch] = hu[static_cast<size_t>(r)];
      for (int k = 0; k < M; ++k) {
        (*A)[ch * M + k] = ha[static_cast<size_t>(k) * kBtChains + r];
        (*B)[ch * M + k] = hb[static_cast<size_t>(k) * kBtChains + r];
      }
    }
  }
  return FTLM_OK;
}

}  // namespace capi
}  // namespace ftlm_b200

extern "C" {

int ftlm_gpu_batched_set_cols_variant(ftlm_sector* s, int variant) {
  if (!s || variant < 0 || variant > 2) return fail(FTLM_ERR_INVALID, "batched cols variant must be 0, 1 or 2");
  s->dev.bt_cols = variant;
  return FTLM_OK;
}

int ftlm_gpu_batched_autotune(ftlm_sector* s, int reps, int* variant, float* ms) try {
  int rc = need_device(s);
  if (rc) return rc;
  if (s->plan.max_up_deg > 120)
    return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
  reps = std::max(1, reps);
  const SectorPlan& P = s->plan;
  static std::mutex mu;
  static std::map<std::string, int> cache;  // one timing per sector shape and process
  char key[160];
  std::snprintf(key, sizeof(key), "%d/%d/%d/%zu/%zu/%d/%d", P.n, P.nu, P.nd, P.hu.size(), P.hd.size(), P.max_up_deg,
                P.max_dn_deg);
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      s->dev.bt_cols = it->second;
      if (variant) *variant = it->second;
      if (ms) *ms = -1.0f;
      return FTLM_OK;
    }
  }
  cudaStream_t st = s->stream;
  int best_v = 0;
  float best = 3.4e38f;
  {
    std::lock_guard<std::mutex> lock(g_bt_mu);
    const int planes = pl_group(s->dev, true, kBtChains / 2);
    CU_TRY(g_bt.ensure(static_cast<size_t>(planes) * P.dim * sizeof(float4), 1));
    float4* W = g_bt.buf[0].as<float4>();
    float4* Y = g_bt.buf[1].as<float4>();
    int* fl = g_bt.flags.as<int>();
    CU_TRY(pl_start(s->dev, W, planes, 7u, g_bt.state(0), st));
    CU_TRY(cudaMemsetAsync(fl, 0, sizeof(int), st));
    cudaEvent_t e0, e1;
    CU_TRY(cudaEventCreate(&e0));
    CU_TRY(cudaEventCreate(&e1));
    cudaError_t ce = cudaSuccess;
    for (int v = 0; v < 3 && ce == cudaSuccess; ++v) {
      DevSector d = s->dev;
      d.bt_cols = v;
      ce = pl_apply(d, W, Y, planes, fl, st);  // warm-up
      if (ce == cudaSuccess) ce = cudaEventRecord(e0, st);
      for (int r = 0; r < reps && ce == cudaSuccess; ++r) ce = pl_apply(d, W, Y, planes, fl, st);
      if (ce == cudaSuccess) ce = cudaEventRecord(e1, st);
      if (ce == cudaSuccess) ce = cudaEventSynchronize(e1);
      float t = 0.0f;
      if (ce == cudaSuccess) ce = cudaEventElapsedTime(&t, e0, e1);
      if (ce == cudaSuccess && t < best) {
        best = t;
        best_v = v;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    CU_TRY(ce);
  }
  s->dev.bt_cols = best_v;
  {
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = best_v;
  }
  if (variant) *variant = best_v;
  if (ms) *ms = best / static_cast<float>(reps);
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_batched_lanczos(ftlm_sector* s, int R, int M, unsigned seed, double* alpha, double* beta, int* used) try {
  int rc = need_device(s);
  if (rc) return rc;
  if (s->plan.max_up_deg > 120)
    return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
  if (R <= 0 || M <= 0 || !alpha || !beta || !used) return fail(FTLM_ERR_INVALID, "bad arguments");
  std::vector<double> A, B;
  std::vector<int> u;
  rc = bt_run_chains(s, R, M, seed, &A, &B, &u);
  if (rc) return rc;
  std::copy(A.begin(), A.end(), alpha);
  std::copy(B.begin(), B.end(), beta);
  std::copy(u.begin(), u.end(), used);
  return FTLM_OK;
} catch (...) {
  return caught();
}

namespace {

// The batched sector estimate, and (n_check > 0) its rounding-error estimate against complex128:
// chains r < n_check are rerun with complex128 vectors from the same Philox start, and
// lnz_err[b] = max_r |L_r(c64) - L_r(c128)| over them, L_r the chain's log quadrature at bts[b].
// Since ln Z_s = ln dim + log mean_r e^{L_r}, a common bound d on |dL_r| bounds |d ln Z_s| by d.
int batched_sector(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed, int n_check, double* lnz,
                   double* energy, double* lnz_err) {
  int rc = need_device(s);
  if (rc) return rc;
  if (n_bt < 0 || (n_bt > 0 && (!bts || !lnz || !energy)) || (n_check > 0 && n_bt > 0 && !lnz_err))
    return fail(FTLM_ERR_INVALID, "bad arguments");
  R = std::max(1, R);
  M = std::max(1, M);
  if (M > 160) return fail(FTLM_ERR_UNSUPPORTED, "more than 160 Lanczos steps for the on-chip Jacobi");
  const int64_t dim = s->plan.dim;
  if (lnz_err) std::fill(lnz_err, lnz_err + n_bt, 0.0);
  // Sectors whose Krylov space the chain can exhaust stay on the complex128 path (same Philox
  // start vectors), where the reference's breakdown test is meaningful; their error is zero.
  if (dim <= 2 * static_cast<int64_t>(M))
    return plain_sector_ftlm(s, bts, n_bt, R, M, seed, FTLM_START_PHILOX, true, lnz, energy);
  if (s->plan.max_up_deg > 120)
    return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
  if (n_check <= 0 && fused_alone(s->dev))
    return chains_ftlm({s}, R, M, seed, FTLM_START_PHILOX, true, bts, n_bt, true, lnz, energy);
  std::vector<double> A, B;
  std::vector<int> used;
  rc = bt_run_chains(s, R, M, seed, &A, &B, &used);
  if (rc) return rc;
  std::vector<double> lq(static_cast<size_t>(R) * n_bt), eq(static_cast<size_t>(R) * n_bt);
  rc = chain_quadrature(A.data(), B.data(), used.data(), R, M, bts, n_bt, lq.data(), eq.data(), true);
  if (rc) return rc;
  rc = ftlm_gpu_ftlm_combine(lq.data(), eq.data(), used.data(), R, n_bt, std::log(static_cast<double>(dim)), lnz, energy);
  if (rc || n_check <= 0 || n_bt == 0) return rc;
  const int nc = std::min(n_check, R);
  std::vector<double> a(static_cast<size_t>(M), 0.0), b(static_cast<size_t>(M), 0.0), q1(static_cast<size_t>(n_bt)),
      e1(static_cast<size_t>(n_bt));
  for (int r = 0; r < nc; ++r) {
    std::fill(a.begin(), a.end(), 0.0);
    std::fill(b.begin(), b.end(), 0.0);
    int nb = 0, u = 0;
    rc = ftlm_gpu_lanczos(s, M, seed + static_cast<unsigned>(r) * 100003u, FTLM_START_PHILOX, a.data(), b.data(), &nb, &u);
    if (rc) return rc;
    rc = chain_quadrature(a.data(), b.data(), &u, 1, M, bts, n_bt, q1.data(), e1.data(), true);
    if (rc) return rc;
    for (int k = 0; k < n_bt; ++k) {
      const double d = std::fabs(lq[static_cast<size_t>(r) * n_bt + k] - q1[static_cast<size_t>(k)]);
      lnz_err[k] = std::max(lnz_err[k], std::isfinite(d) ? d : std::numeric_limits<double>::infinity());
    }
  }
  return FTLM_OK;
}

}  // namespace

int ftlm_gpu_batched_ftlm_sector(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed, double* lnz,
                                 double* energy) try {
  return batched_sector(s, bts, n_bt, R, M, seed, 0, lnz, energy, nullptr);
} catch (...) {
  return caught();
}

int ftlm_gpu_batched_ftlm_sector_checked(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed,
                                         int n_check, double* lnz, double* energy, double* lnz_err) try {
  if (n_check < 1) return fail(FTLM_ERR_INVALID, "n_check must be >= 1");
  return batched_sector(s, bts, n_bt, R, M, seed, n_check, lnz, energy, lnz_err);
} catch (...) {
  return caught();
}

namespace {

int batched_sweep(const ftlm_params* p, int R, int M, unsigned seed, const double* bts, int n_bt, const double* mus,
                  int n_mu, int n_check, double* lnz_s, double* e_s, double* lnz_gc, double* n_avg, double* e_avg,
                  double* lnz_s_err);

}  // namespace

int ftlm_gpu_batched_sweep(const ftlm_params* p, int R, int M, unsigned seed, const double* bts, int n_bt,
                           const double* mus, int n_mu, double* lnz_s, double* e_s, double* lnz_gc, double* n_avg,
                           double* e_avg) try {
  return batched_sweep(p, R, M, seed, bts, n_bt, mus, n_mu, 0, lnz_s, e_s, lnz_gc, n_avg, e_avg, nullptr);
} catch (...) {
  return caught();
}

int ftlm_gpu_batched_sweep_checked(const ftlm_params* p, int R, int M, unsigned seed, const double* bts, int n_bt,
                                   const double* mus, int n_mu, int n_check, double* lnz_s, double* e_s, double* lnz_gc,
                                   double* n_avg, double* e_avg, double* lnz_s_err, double* lnz_gc_err,
                                   double* n_err) try {
  if (n_check < 1) return fail(FTLM_ERR_INVALID, "n_check must be >= 1");
  if (!p || !lnz_s_err || !lnz_gc || !n_avg || !e_avg || !lnz_gc_err || !n_err)
    return fail(FTLM_ERR_INVALID, "null argument");
  int rc = batched_sweep(p, R, M, seed, bts, n_bt, mus, n_mu, n_check, lnz_s, e_s, lnz_gc, n_avg, e_avg, lnz_s_err);
  if (rc) return rc;
  // First-order propagation of the sector errors through the grand-canonical combination:
  // d ln Z_GC = sum_s w_s d ln Z_s and d<n> = sum_s w_s (N_s/n - <n>) d ln Z_s.
  const int n = p->Lx * p->Ly;
  for (int b = 0; b < n_bt; ++b)
    for (int m = 0; m < n_mu; ++m) {
      const size_t o = static_cast<size_t>(b) * n_mu + m;
      double eg = 0.0, en = 0.0;
      for (int nu = 0; nu <= n; ++nu)
        for (int nd = 0; nd <= n; ++nd) {
          const size_t sidx = static_cast<size_t>(nu * (n + 1) + nd);
          const double lz = lnz_s[sidx * n_bt + b];
          if (!std::isfinite(lz)) continue;
          const double w = std::exp(lz + bts[b] * mus[m] * static_cast<double>(nu + nd) - lnz_gc[o]);
          const double d = lnz_s_err[sidx * n_bt + b];
          eg += w * d;
          en += w * std::fabs(static_cast<double>(nu + nd) / n - n_avg[o]) * d;
        }
      lnz_gc_err[o] = eg;
      n_err[o] = en;
    }
  return FTLM_OK;
} catch (...) {
  return caught();
}

namespace {

int batched_sweep(const ftlm_params* p, int R, int M, unsigned seed, const double* bts, int n_bt, const double* mus,
                  int n_mu, int n_check, double* lnz_s, double* e_s, double* lnz_gc, double* n_avg, double* e_avg,
                  double* lnz_s_err) {
  if (!p || !lnz_s || !e_s) return fail(FTLM_ERR_INVALID, "null argument");
  const int n = p->Lx * p->Ly;
  if (n <= 0 || n > 32) return fail(FTLM_ERR_INVALID, "FockBasis: require 1 <= n_sites <= 32 (bit packing)");
  const int nsec = (n + 1) * (n + 1);
  std::vector<int> N(static_cast<size_t>(nsec));
  // small sectors go to fused launches: those the batched path runs in complex128 (dim <= 2M, Philox starts), and
  // those whose complex64 chains need no check against complex128
  PlanParts parts(n);
  OwnedSectors owned[2];
  std::vector<ftlm_sector*>&small = owned[0].v, &mid = owned[1].v;
  std::vector<int> small_idx, mid_idx;
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const int idx = nu * (n + 1) + nd;
      N[static_cast<size_t>(idx)] = nu + nd;
      ftlm_sector* s = nullptr;
      int rc = sector_create(p, nu, nd, &parts, &s);
      if (rc) return rc;
      if (s->plan.dim >= 2 && s->plan.dim <= 2 * static_cast<int64_t>(std::max(1, M)) && M <= 160) {  // a row fits: <= 320
        small.push_back(s);
        small_idx.push_back(idx);
        continue;
      }
      if (n_check <= 0 && M <= 160 && s->plan.dim >= 2 && s->plan.dim <= kFusedSweepMax && s->plan.max_up_deg <= 120 &&
          chain_rows(s->dev, true, false) > 0) {
        mid.push_back(s);
        mid_idx.push_back(idx);
        continue;
      }
      rc = batched_sector(s, bts, n_bt, R, M, seed, n_check, lnz_s + static_cast<size_t>(idx) * n_bt,
                          e_s + static_cast<size_t>(idx) * n_bt,
                          lnz_s_err ? lnz_s_err + static_cast<size_t>(idx) * n_bt : nullptr);
      ftlm_gpu_sector_destroy(s);
      if (rc) return rc;
    }
  int rcf = fused_sectors_ftlm(small, small_idx, std::max(1, R), std::max(1, M), seed, FTLM_START_PHILOX, false, bts, n_bt,
                               lnz_s, e_s, true);
  if (!rcf)
    rcf = fused_sectors_ftlm(mid, mid_idx, std::max(1, R), std::max(1, M), seed, FTLM_START_PHILOX, true, bts, n_bt, lnz_s,
                             e_s, true);
  if (rcf) return rcf;
  if (lnz_s_err)  // the fused small sectors ran in complex128
    for (int i : small_idx) std::fill(lnz_s_err + static_cast<size_t>(i) * n_bt, lnz_s_err + static_cast<size_t>(i + 1) * n_bt, 0.0);
  if (lnz_gc && n_avg && e_avg)
    return ftlm_gpu_gc_reduce(lnz_s, e_s, N.data(), nsec, bts, n_bt, mus, n_mu, n, lnz_gc, n_avg, e_avg);
  return FTLM_OK;
}

}  // namespace

int ftlm_gpu_batched_release(void) try {
  std::lock_guard<std::mutex> lock(g_bt_mu);
  g_bt.release();
  g_grad.release();
  pool_trim();
  return FTLM_OK;
} catch (...) {
  return caught();
}

}  // extern "C"

