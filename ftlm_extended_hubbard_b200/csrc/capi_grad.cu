#include <type_traits>

#include "capi_internal.hpp"

using namespace ftlm_b200;
using namespace ftlm_b200::capi;

// ---------------------------------------------------------------------------------------------
// Parameter gradient of the sector FTLM estimate (no reference counterpart).
//
// For one chain with normalised start vector r, Lanczos vectors q_i and tridiagonal T, the
// estimator term is g = e_1^T e^{-bT T} e_1 and, with r fixed, its exact derivative in the Krylov
// space is dg/dtheta = -sum_il K_il <q_i| dH/dtheta |q_l> (Duhamel; K from duhamel_weights).  The
// chains are replayed from their seed with the forward's kernels (bit-identical alpha/beta), the
// vectors kept on the device, and the three moments of dH/dU (double occupancy), dH/dV (neighbour
// pair density) and dH/dt' (the t' hopping operator) reduced by grad.cu.
namespace {

struct ChainGrad {
  bool ok = false;
  double lmin = 0.0, g = 0.0, m[3] = {0.0, 0.0, 0.0};
};

// The moments of nc chains of one sector: tridiagonals, lengths and stored vectors' norms on the device, the vectors at Q
// (Q + i * vstride + p * pstride: plane p of vector i) and their images under the operator at AQ (or null).
template <class T>
struct SectorChains {
  ftlm_sector* s;
  int nc;
  const T* Q;
  const T* AQ;
  int64_t vstride, pstride;
};

// Weights K = Z P Z^T of all chains (eigen-decomposition of each chain's tridiagonal, Duhamel's formula), then the
// moments sector by sector; everything stays on the device until the end.
template <class T>
int chain_moments(const std::vector<SectorChains<T>>& v, int ld, double bT, const double* alpha, const double* beta,
                  const int* used, const double* scale, cudaStream_t st, std::vector<ChainGrad>* out) {
  int nc = 0, most = 0;
  for (const auto& x : v) {
    nc += x.nc;
    most = std::max(most, x.nc);
  }
  const size_t mat = static_cast<size_t>(nc) * ld;
  Scratch mem;
  const size_t o_l = mem.array<double>(mat), o_v = mem.array<double>(mat * ld), o_y = mem.array<double>(mat * ld);
  const size_t o_k = mem.array<double>(mat * ld), o_g = mem.array<double>(5 * static_cast<size_t>(nc));
  const size_t o_i = mem.array<int>(2 * static_cast<size_t>(nc));
  const size_t o_p = mem.array<double>(static_cast<size_t>(kGradMaxBlocks) * most * 3);
  CU_TRY(mem.commit());
  double *g = mem.at<double>(o_g), *lmin = g + nc, *m = lmin + nc;
  CU_TRY(symeig_tridiag(alpha, beta, used, nc, ld, mem.at<double>(o_l), nullptr, mem.at<double>(o_v), mem.at<int>(o_i), st));
  CU_TRY(duhamel_weights_dev(mem.at<double>(o_l), mem.at<double>(o_v), used, nc, ld, bT, scale, mem.at<double>(o_y),
                             mem.at<double>(o_k), g, lmin, st));
  int c0 = 0;
  for (const auto& x : v) {
    const cudaError_t e = grad_moments(x.s->dev, x.Q, x.AQ ? x.AQ : x.Q, x.vstride, x.pstride, x.nc,
                                       mem.at<double>(o_k) + static_cast<size_t>(c0) * ld * ld, used + c0, ld,
                                       mem.at<double>(o_p), m + 3 * c0, st);
    if (e == cudaErrorInvalidValue)
      return fail(FTLM_ERR_UNSUPPORTED, "gradient: Lanczos vectors of one block do not fit in shared memory");
    CU_TRY(e);
    c0 += x.nc;
  }
  std::vector<double> h(5 * static_cast<size_t>(nc));
  std::vector<int> info(static_cast<size_t>(nc)), n(static_cast<size_t>(nc));
  CU_TRY(cudaMemcpyAsync(h.data(), g, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaMemcpyAsync(info.data(), mem.at<void>(o_i), info.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaMemcpyAsync(n.data(), used, n.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  mem.idle();
  out->assign(static_cast<size_t>(nc), ChainGrad{});
  for (size_t c = 0; c < out->size(); ++c) {
    if (n[c] <= 0) continue;
    if (info[c] != 0) return fail(FTLM_ERR_NUMERIC, "GPU eigen-solver did not converge");
    ChainGrad& cg = (*out)[c];
    cg.ok = true;
    cg.g = h[c];
    cg.lmin = h[static_cast<size_t>(nc) + c];
    for (int q = 0; q < 3; ++q) cg.m[q] = h[2 * static_cast<size_t>(nc) + 3 * c + q];
  }
  return FTLM_OK;
}

// Bytes of stored vectors (and as many of their images under the operator) of one piece of a replay.  A replay whose
// device memory does not suffice is tried again with half, down to one plane.
constexpr size_t kGradStore = size_t(6) << 30;

// One piece of grad_fused: chains r0 .. r0 + R - 1 of the sectors, their vectors at the elements `base` of the store of
// `total` elements; out: [sector][R].
template <class T>
int grad_piece(const std::vector<ftlm_sector*>& secs, const std::vector<ftlm_sector*>& op, double bT, int r0, int R, int M,
               unsigned seed, int start_mode, const std::vector<int64_t>& base, int64_t total, std::vector<ChainGrad>* out) {
  constexpr bool c64 = std::is_same<T, float4>::value;
  const int planes = c64 ? (R + 1) / 2 : R;
  CU_TRY(g_grad.grow(g_grad.Q, g_grad.qcap, static_cast<size_t>(total) * sizeof(T)));
  CU_TRY(g_grad.grow(g_grad.AQ, g_grad.acap, static_cast<size_t>(total) * sizeof(T)));
  ChainRun run;
  const unsigned seed0 = seed + static_cast<unsigned>(r0) * 100003u;
  int rc = chains_run(secs, R, M, seed0, start_mode, c64, &run, g_grad.Q.p, &base, true);
  if (rc) return rc;
  cudaStream_t st = secs[0]->stream;
  run.mem.busy();
  std::vector<SectorChains<T>> v;
  for (size_t i = 0; i < secs.size(); ++i) {
    const int64_t dim = secs[i]->plan.dim;
    const T* Q = g_grad.Q.as<T>() + base[i];
    T* AQ = op[i] ? g_grad.AQ.as<T>() + base[i] : nullptr;
    // the operator on every stored vector: the planes of all steps are contiguous
    if (AQ) CU_TRY(pl_apply(op[i]->dev, Q, AQ, M * planes, g_grad.flag.as<int>(), st));
    v.push_back(SectorChains<T>{secs[i], R, Q, AQ, planes * dim, dim});
  }
  rc = chain_moments(v, M, bT, run.alpha, run.beta, run.used, run.scale, st, out);
  if (!rc) run.mem.idle();
  return rc;
}

// Chains of small sectors (chains_run), replayed with their vectors kept; op[i] (may be null) is the operator's sector.
// Pieces of a bounded store: several whole sectors, or a range of one sector's chains where all of them do not fit (a
// plane's two complex64 chains stay together, so each chain is the forward's).  out: [sector][R].
template <class T>
int grad_fused(const std::vector<ftlm_sector*>& secs, const std::vector<ftlm_sector*>& op, double bT, int R, int M,
               unsigned seed, int start_mode, std::vector<std::vector<ChainGrad>>* out) {
  constexpr int kC = std::is_same<T, float4>::value ? 2 : 1;
  out->assign(secs.size(), {});
  std::lock_guard<std::mutex> lock(g_bt_mu);
  if (!g_grad.flag.p) CU_TRY(g_grad.flag.alloc(sizeof(int)));
  size_t store = kGradStore;
  auto vectors = [&](size_t i, int chains) {  // elements of the stored vectors of so many chains
    return static_cast<int64_t>(M) * ((chains + kC - 1) / kC) * secs[i]->plan.dim;
  };
  const size_t weights = static_cast<size_t>(M) * M * sizeof(double) * 3;  // of a chain, at most half a store of them
  for (size_t i0 = 0; i0 < secs.size();) {
    const int r0 = static_cast<int>((*out)[i0].size());
    const size_t plane = static_cast<size_t>(vectors(i0, 1)) * sizeof(T);
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>(store / plane, store / 2 / (weights * kC)));  // planes
    const int n = static_cast<int>(std::min<int64_t>(R - r0, most * kC));
    std::vector<ftlm_sector*> piece{secs[i0]}, ops{op[i0]};
    std::vector<int64_t> base{0};
    int64_t total = vectors(i0, n);
    size_t i1 = i0 + 1;
    if (n == R)
      for (; i1 < secs.size(); ++i1) {
        const int64_t add = vectors(i1, R);
        if (static_cast<size_t>(total + add) * sizeof(T) > store || (piece.size() + 1) * R * weights > store / 2) break;
        piece.push_back(secs[i1]);
        ops.push_back(op[i1]);
        base.push_back(total);
        total += add;
      }
    std::vector<ChainGrad> cg;
    const int rc = grad_piece<T>(piece, ops, bT, r0, n, M, seed, start_mode, base, total, &cg);
    if (rc == FTLM_ERR_NOMEM && store > plane) {
      cudaGetLastError();
      g_grad.release();
      store /= 2;
      continue;
    }
    if (rc) return rc;
    for (size_t i = 0; i < piece.size(); ++i)
      (*out)[i0 + i].insert((*out)[i0 + i].end(), cg.begin() + static_cast<long>(i) * n, cg.begin() + static_cast<long>(i + 1) * n);
    if (r0 + n == R) i0 = i1;
  }
  return FTLM_OK;
}

// Chains of one sector on the whole GPU (planes.cu), replayed step by step with the vectors kept: the forward's groups and
// kernels, so its alpha and beta.
template <class T>
int grad_planes(ftlm_sector* s, ftlm_sector* op, double bT, int R, int M, unsigned seed, int start_mode,
                std::vector<ChainGrad>* out) {
  constexpr bool c64 = std::is_same<T, float4>::value;
  constexpr int kC = c64 ? 2 : 1;
  const int64_t dim = s->plan.dim;
  const int most = (std::min(R, kBtChains) + kC - 1) / kC;
  int group = pl_group(s->dev, c64, most);
  // Complex64 chains replay in the forward's groups, at most a block's 16 planes: a group of another size adds its sums
  // in another order, which their FP32 vectors do not forgive.  Complex128 chains take as many as the store holds.
  if (!c64)
    group = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(group, kGradStore / ((M + 1) * dim * sizeof(T)))));
  std::lock_guard<std::mutex> lock(g_bt_mu);
  auto room = [&]() -> int {
    const size_t vector = static_cast<size_t>(dim) * group * sizeof(T);
    CU_TRY(g_bt.ensure(0, M, pl_items_doubles(s->dev, c64, group)));
    CU_TRY(g_grad.grow(g_grad.Q, g_grad.qcap, static_cast<size_t>(M + 1) * vector));
    if (op) CU_TRY(g_grad.grow(g_grad.AQ, g_grad.acap, static_cast<size_t>(M) * vector));
    if (!g_grad.flag.p) CU_TRY(g_grad.flag.alloc(sizeof(int)));
    return FTLM_OK;
  };
  for (;;) {
    const int rc = room();
    if (!rc) break;
    if (rc != FTLM_ERR_NOMEM || c64 || group == 1) return rc;
    cudaGetLastError();
    g_grad.release();
    group = (group + 1) / 2;
  }
  cudaStream_t st = s->stream;
  T* Q = g_grad.Q.as<T>();
  T* AQ = op ? g_grad.AQ.as<T>() : nullptr;
  const size_t tab = static_cast<size_t>(M) * kBtChains;
  std::vector<double> ha(tab), hb(tab), hs(kBtChains);  // hs: 1 / ||raw start||
  std::vector<int> hu(kBtChains);
  std::vector<std::complex<double>> start;
  out->clear();
  for (int r0 = 0; r0 < R;) {
    // as the forward: blocks of 32 chains (complex64), groups of planes within them
    const int left = c64 ? std::min(kBtChains - r0 % kBtChains, R - r0) : R - r0;
    const int nc = std::min(group * kC, left), np = (nc + kC - 1) / kC;
    const unsigned seed_g = seed + static_cast<unsigned>(r0) * 100003u;
    const PlaneState z = g_bt.state(0);
    CU_TRY(cudaMemsetAsync(z.alpha, 0, tab * sizeof(double), st));
    CU_TRY(cudaMemsetAsync(z.beta, 0, tab * sizeof(double), st));
    if constexpr (c64) {
      CU_TRY(pl_start(s->dev, Q, np, seed_g, z, st));
    } else {
      const bool given = start_mode == FTLM_START_REFERENCE;
      if (given) {
        reference_normals(dim, np, seed_g, &start);
        CU_TRY(cudaMemcpyAsync(Q, start.data(), start.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
      }
      CU_TRY(pl_start(s->dev, Q, np, seed_g, given, z, st));
    }
    CU_TRY(cudaMemcpyAsync(hs.data(), z.st + kBtSin * kBtChains, kBtChains * sizeof(double), cudaMemcpyDeviceToHost, st));
    const int64_t step = dim * np;
    for (int k = 0; k < M; ++k)
      CU_TRY(pl_step(s->dev, Q + k * step, Q + (k > 0 ? k - 1 : 0) * step, Q + (k + 1) * step, np, k, z, st));
    CU_TRY(cudaMemcpyAsync(ha.data(), z.alpha, tab * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hb.data(), z.beta, tab * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hu.data(), z.used, hu.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    int steps = 0;  // of the group's longest chain: no vector is written after it
    for (int c = 0; c < nc; ++c) steps = std::max(steps, hu[static_cast<size_t>(c)]);
    if (op && steps > 0) CU_TRY(pl_apply(op->dev, Q, AQ, steps * np, g_grad.flag.as<int>(), st));
    // chain-major tables: alpha, beta, norms of the stored vectors (W_0 = ||raw|| q_0, W_i = beta_{i-1} q_i)
    const size_t row = static_cast<size_t>(nc) * M;
    std::vector<double> t(3 * row, 0.0);
    std::vector<int> n(static_cast<size_t>(nc));
    for (int c = 0; c < nc; ++c) {
      n[static_cast<size_t>(c)] = hs[static_cast<size_t>(c)] > 0.0 ? hu[static_cast<size_t>(c)] : 0;
      for (int k = 0; k < M; ++k) {
        const size_t o = static_cast<size_t>(c) * M + k, h = static_cast<size_t>(k) * kBtChains + c;
        t[o] = ha[h];
        t[row + o] = hb[h];
        double norm = 1.0;
        if (k < n[static_cast<size_t>(c)]) norm = k == 0 ? 1.0 / hs[static_cast<size_t>(c)] : hb[h - kBtChains];
        t[2 * row + o] = norm;
      }
    }
    Scratch mem;
    const size_t o_t = mem.array<double>(t.size()), o_n = mem.array<int>(n.size());
    CU_TRY(mem.commit());
    CU_TRY(cudaMemcpyAsync(mem.at<void>(o_t), t.data(), t.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    CU_TRY(cudaMemcpyAsync(mem.at<void>(o_n), n.data(), n.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    const double* dt = mem.at<double>(o_t);
    std::vector<ChainGrad> cg;
    const int rc = chain_moments<T>({SectorChains<T>{s, nc, Q, AQ, step, dim}}, M, bT, dt, dt + row, mem.at<int>(o_n),
                                    dt + 2 * row, st, &cg);
    if (rc) return rc;
    mem.idle();
    out->insert(out->end(), cg.begin(), cg.end());
    r0 += nc;
  }
  return FTLM_OK;
}

// Complex128 chains one at a time with the sector's own H v (sectors without a gauge table).
int grad_serial(ftlm_sector* s, ftlm_sector* op, double bT, int R, int M, unsigned seed, int start_mode,
                std::vector<ChainGrad>* out) {
  const int64_t dim = s->plan.dim;
  std::lock_guard<std::mutex> lock(g_bt_mu);
  CU_TRY(g_grad.grow(g_grad.Q, g_grad.qcap, static_cast<size_t>(M) * dim * sizeof(double2)));
  if (op) CU_TRY(g_grad.grow(g_grad.AQ, g_grad.acap, static_cast<size_t>(M) * dim * sizeof(double2)));
  double2* Q = g_grad.Q.as<double2>();
  double2* AQ = op ? g_grad.AQ.as<double2>() : nullptr;
  out->assign(static_cast<size_t>(R), ChainGrad{});
  for (int r = 0; r < R; ++r) {
    std::vector<double> a, b;
    int rc = run_lanczos(
        dim, [s](const double2* x, double2* y, cudaStream_t st) { return s->apply(x, y, st); }, s->ws, M,
        seed + static_cast<unsigned>(r) * 100003u, start_mode, s->stream, &a, &b, Q);
    if (rc) return rc;
    const int n = static_cast<int>(a.size());
    if (n <= 0) continue;
    if (op)
      for (int i = 0; i < n; ++i) {
        rc = op->apply(Q + static_cast<int64_t>(i) * dim, AQ + static_cast<int64_t>(i) * dim, s->stream);
        if (rc) return rc;
      }
    std::vector<double> t(3 * static_cast<size_t>(M), 0.0);
    std::copy(a.begin(), a.end(), t.begin());
    std::copy(b.begin(), b.begin() + std::min<size_t>(b.size(), static_cast<size_t>(M)), t.begin() + M);
    std::fill(t.begin() + 2 * M, t.end(), 1.0);
    cudaStream_t st = s->stream;
    Scratch mem;
    const size_t o_t = mem.array<double>(t.size()), o_n = mem.array<int>(1);
    CU_TRY(mem.commit());
    CU_TRY(cudaMemcpyAsync(mem.at<void>(o_t), t.data(), t.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    CU_TRY(cudaMemcpyAsync(mem.at<void>(o_n), &n, sizeof(int), cudaMemcpyHostToDevice, st));
    const double* dt = mem.at<double>(o_t);
    std::vector<ChainGrad> cg;
    rc = chain_moments<double2>({SectorChains<double2>{s, 1, Q, AQ, dim, dim}}, M, bT, dt, dt + M, mem.at<int>(o_n),
                                dt + 2 * M, st, &cg);
    if (rc) return rc;
    mem.idle();
    (*out)[static_cast<size_t>(r)] = cg[0];
  }
  return FTLM_OK;
}

// ln Z = ln dim + log mean_r g_r, g_r = e^{-bT lmin_r} ghat_r; d ln Z = -sum_r e^{-bT lmin_r} m_r / sum_r g_r
void sector_gradient(const std::vector<ChainGrad>& cg, int64_t dim, double bT, bool has_op, double* lnz, double* dlnz) {
  double mx = -std::numeric_limits<double>::infinity();
  int used = 0;
  for (const auto& c : cg)
    if (c.ok) {
      mx = std::max(mx, -bT * c.lmin + std::log(c.g));
      ++used;
    }
  dlnz[0] = dlnz[1] = dlnz[2] = 0.0;
  if (used == 0) {
    *lnz = -std::numeric_limits<double>::infinity();
    return;
  }
  double zs = 0.0, d[3] = {0.0, 0.0, 0.0};
  for (const auto& c : cg) {
    if (!c.ok) continue;
    const double w = std::exp(-bT * c.lmin - mx);
    zs += w * c.g;
    for (int q = 0; q < 3; ++q) d[q] -= w * c.m[q];
  }
  *lnz = std::log(static_cast<double>(dim)) + mx + std::log(zs / static_cast<double>(used));
  for (int q = 0; q < (has_op ? 3 : 2); ++q) dlnz[q] = d[q] / zs;
}

// The path of a sector's chains in the gradient, which is the forward's: fused, on planes, or (complex128 without a gauge
// table) not available.
bool grad_is_c64(const ftlm_sector* s, int M, int method) { return method == 1 && s->plan.dim > 2 * static_cast<int64_t>(M); }
bool grad_is_fused(const ftlm_sector* s, const ftlm_sector* op, bool c64) {
  if (op && !c64 && !pl_fits(op->dev, op->plan.max_up_deg)) return false;  // complex128 planes of it do not run
  return s->plan.dim <= kFusedSweepMax && chain_rows(s->dev, c64, false) > 0 && s->plan.max_up_deg <= 120;
}

int grad_one(ftlm_sector* s, ftlm_sector* op, double bT, int R, int M, unsigned seed, int method, int start_mode,
             std::vector<ChainGrad>* cg) {
  const bool c64 = grad_is_c64(s, M, method);
  const int mode = method == 1 ? FTLM_START_PHILOX : start_mode;
  if (grad_is_fused(s, op, c64)) {
    std::vector<std::vector<ChainGrad>> v;
    const int rc = c64 ? grad_fused<float4>({s}, {op}, bT, R, M, seed, mode, &v)
                       : grad_fused<double2>({s}, {op}, bT, R, M, seed, mode, &v);
    if (!rc) *cg = v[0];
    return rc;
  }
  if (c64) return grad_planes<float4>(s, op, bT, R, M, seed, mode, cg);
  if (!pl_fits(s->dev, s->plan.max_up_deg) || (op && !pl_fits(op->dev, op->plan.max_up_deg)))
    return grad_serial(s, op, bT, R, M, seed, mode, cg);
  return grad_planes<double2>(s, op, bT, R, M, seed, mode, cg);
}

}  // namespace

extern "C" {

int ftlm_gpu_grad_sector(ftlm_sector* s, ftlm_sector* op_tp, double bT, int R, int M, unsigned seed, int method,
                         int start_mode, double* lnz, double* dlnz) try {
  int rc = need_device(s);
  if (rc) return rc;
  if (op_tp) {
    rc = need_device(op_tp);
    if (rc) return rc;
    if (op_tp->plan.n != s->plan.n || op_tp->plan.nu != s->plan.nu || op_tp->plan.nd != s->plan.nd)
      return fail(FTLM_ERR_INVALID, "gradient operator sector has a different (n_sites, N_up, N_dn)");
  }
  if (!lnz || !dlnz || method < 0 || method > 1) return fail(FTLM_ERR_INVALID, "bad arguments");
  R = std::max(1, R);
  M = std::max(1, M);
  if (M > kMaxEig) return fail(FTLM_ERR_UNSUPPORTED, "more than 160 Lanczos steps for the GPU eigen-solver");
  if (method == 1 && s->plan.dim > 2 * static_cast<int64_t>(M) &&
      (s->plan.max_up_deg > 120 || (op_tp && op_tp->plan.max_up_deg > 120)))
    return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
  std::vector<ChainGrad> cg;
  rc = grad_one(s, op_tp, bT, R, M, seed, method, start_mode, &cg);
  if (rc) return rc;
  sector_gradient(cg, s->plan.dim, bT, op_tp != nullptr, lnz, dlnz);
  return FTLM_OK;
} catch (...) {
  return caught();
}

// ---- differentiable grand-canonical ln Z at one (T, mu) ----------------------------------------
// Forward: every sector's chains as the FTLM entry points make them (the small sectors' chains in
// one fused launch), the converged tridiagonal quadrature, the sector combine
// (src/ftlm_thermo.cpp:246-256) and the grand-canonical log-sum-exp of
// benchmarks/bench_ftlm_nmu_rect.cpp:186-219 at a single (T, mu).  Backward: d/dmu = bT <N>,
// d/dbT = <mu N - E>, and d/d(U, V, t') = sum_s w_s d ln Z_s/dtheta from ftlm_gpu_grad_sector
// (sectors with weight w_s < 1e-13 skipped).
namespace {

constexpr double kGcWeightCutoff = 1e-13;
constexpr long long kGcFusedPlainMax = kFusedSweepMax;

struct SectorDeleter {
  void operator()(ftlm_sector* s) const { ftlm_gpu_sector_destroy(s); }
};
using SectorPtr = std::unique_ptr<ftlm_sector, SectorDeleter>;

int gc_check(const ftlm_params* p, double bT, int R, int M, int method, int start_mode) {
  if (!p) return fail(FTLM_ERR_INVALID, "null params");
  const int n = p->Lx * p->Ly;
  if (p->Lx <= 0 || p->Ly <= 0 || n > 32) return fail(FTLM_ERR_INVALID, "FockBasis: require 1 <= n_sites <= 32");
  if (R <= 0 || M <= 0 || M > 160) return fail(FTLM_ERR_INVALID, "require R > 0 and 0 < M <= 160");
  if (method < 0 || method > 1) return fail(FTLM_ERR_INVALID, "method must be 0 (plain) or 1 (batched)");
  if (start_mode != FTLM_START_REFERENCE && start_mode != FTLM_START_PHILOX)
    return fail(FTLM_ERR_INVALID, "unknown start_mode");
  if (!(bT > 0.0) || !std::isfinite(bT)) return fail(FTLM_ERR_INVALID, "inverse temperature must be finite and > 0");
  return FTLM_OK;
}

// ln Z_s, E_s at bT from R chains (alpha/beta [R][M], used [R]) of a sector of size dim.
int gc_quadrature(const double* A, const double* B, const int* used, int R, int M, double bT, int64_t dim,
                  double* lnz, double* en) {
  std::vector<double> lq(static_cast<size_t>(R)), eq(static_cast<size_t>(R));
  int rc = ftlm_gpu_tridiag_quadrature_exact(A, B, used, R, M, &bT, 1, lq.data(), eq.data());
  if (rc) return rc;
  return ftlm_gpu_ftlm_combine(lq.data(), eq.data(), used, R, 1, std::log(static_cast<double>(dim)), lnz, en);
}

double gc_lse(const std::vector<double>& x) {
  double mx = -std::numeric_limits<double>::infinity();
  for (double v : x) mx = std::max(mx, v);
  if (!std::isfinite(mx)) return mx;
  double s = 0.0;
  for (double v : x) s += std::exp(v - mx);
  return mx + std::log(s);
}

}  // namespace

int ftlm_gpu_gc_logz(const ftlm_params* p, double mu, double bT, int R, int M, unsigned seed, int method,
                     int start_mode, double* lnz_s, double* e_s, double* lnz_gc) try {
  int rc = gc_check(p, bT, R, M, method, start_mode);
  if (rc) return rc;
  if (!lnz_s || !e_s || !lnz_gc) return fail(FTLM_ERR_INVALID, "null output");
  const int n = p->Lx * p->Ly;
  const int nsec = (n + 1) * (n + 1);
  const int st_mode = method == 1 ? FTLM_START_PHILOX : start_mode;
  const long long limit = method == 1 ? 2LL * M : kGcFusedPlainMax;
  PlanParts parts(n);
  std::vector<SectorPtr> small, mid;  // chains in fused launches below: complex128 and complex64
  std::vector<int> small_idx, mid_idx;
  std::vector<double> A, B;
  std::vector<int> used;
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const int idx = nu * (n + 1) + nd;
      ftlm_sector* raw = nullptr;
      rc = sector_create(p, nu, nd, &parts, &raw);
      if (rc) return rc;
      SectorPtr s(raw);
      const int64_t dim = s->plan.dim;
      if (dim <= limit && chain_rows(s->dev, false, false) > 0) {
        small.push_back(std::move(s));
        small_idx.push_back(idx);
        continue;
      }
      if (method == 1 && dim <= kFusedSweepMax && s->plan.max_up_deg <= 120 && chain_rows(s->dev, true, false) > 0) {
        mid.push_back(std::move(s));
        mid_idx.push_back(idx);
        continue;
      }
      if (method == 1) {
        rc = need_device(s.get());
        if (rc) return rc;
        if (s->plan.max_up_deg > 120)
          return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
        rc = bt_run_chains(s.get(), R, M, seed, &A, &B, &used);
        if (rc) return rc;
      } else {
        if (s->chains(R) == ftlm_sector::Chains::planes) {
          rc = planes_lanczos(s.get(), R, M, seed, st_mode, &A, &B, &used);
          if (rc) return rc;
        } else {
          A.assign(static_cast<size_t>(R) * M, 0.0);
          B.assign(static_cast<size_t>(R) * M, 0.0);
          used.assign(static_cast<size_t>(R), 0);
          for (int r = 0; r < R; ++r) {
            int nb = 0, u = 0;
            rc = ftlm_gpu_lanczos(s.get(), M, seed + static_cast<unsigned>(r) * 100003u, st_mode,
                                  A.data() + static_cast<size_t>(r) * M, B.data() + static_cast<size_t>(r) * M, &nb, &u);
            if (rc) return rc;
            used[static_cast<size_t>(r)] = u;
          }
        }
      }
      rc = gc_quadrature(A.data(), B.data(), used.data(), R, M, bT, dim, lnz_s + idx, e_s + idx);
      if (rc) return rc;
    }
  auto fused = [&](const std::vector<SectorPtr>& v, const std::vector<int>& at, bool c64) {
    std::vector<ftlm_sector*> hs;
    for (const auto& s : v) hs.push_back(s.get());
    return fused_sectors_ftlm(hs, at, R, M, seed, st_mode, c64, &bT, 1, lnz_s, e_s, true);
  };
  rc = fused(small, small_idx, false);
  if (!rc) rc = fused(mid, mid_idx, true);
  if (rc) return rc;
  std::vector<double> x(static_cast<size_t>(nsec));
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const int idx = nu * (n + 1) + nd;
      x[static_cast<size_t>(idx)] = lnz_s[idx] + bT * mu * static_cast<double>(nu + nd);
    }
  *lnz_gc = gc_lse(x);
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_gc_logz_grad(const ftlm_params* p, double mu, double bT, int R, int M, unsigned seed, int method,
                          int start_mode, const double* lnz_s, const double* e_s, double* grad) try {
  int rc = gc_check(p, bT, R, M, method, start_mode);
  if (rc) return rc;
  if (!lnz_s || !e_s || !grad) return fail(FTLM_ERR_INVALID, "null argument");
  const int n = p->Lx * p->Ly;
  const int nsec = (n + 1) * (n + 1);
  std::vector<double> x(static_cast<size_t>(nsec)), N(static_cast<size_t>(nsec));
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const int idx = nu * (n + 1) + nd;
      N[static_cast<size_t>(idx)] = static_cast<double>(nu + nd);
      x[static_cast<size_t>(idx)] = lnz_s[idx] + bT * mu * N[static_cast<size_t>(idx)];
    }
  const double lnZ = gc_lse(x);
  if (!std::isfinite(lnZ)) return fail(FTLM_ERR_NUMERIC, "grand-canonical ln Z is not finite");
  double d[3] = {0.0, 0.0, 0.0}, dmu = 0.0, dbeta = 0.0;
  ftlm_params pop = *p;  // dH/dt': the t' hopping operator alone
  pop.t = 0.0;
  pop.tp = 1.0;
  pop.U = 0.0;
  pop.V = 0.0;
  PlanParts parts(n), op_parts(n);
  struct Term {
    SectorPtr s, op;
    size_t idx;
    double w;
  };
  std::vector<Term> fused[2];  // small sectors, complex128 and complex64: their chains together
  auto add = [&](const Term& t, const std::vector<ChainGrad>& cg) {
    double lz = 0.0, g[3] = {0.0, 0.0, 0.0};
    sector_gradient(cg, t.s->plan.dim, bT, true, &lz, g);
    if (!(std::fabs(lz - lnz_s[t.idx]) <= 1e-9 * std::max(1.0, std::fabs(lz))))
      return fail(FTLM_ERR_NUMERIC, "gradient replay of sector (" + std::to_string(t.s->plan.nu) + "," +
                                        std::to_string(t.s->plan.nd) + ") did not reproduce the forward ln Z");
    for (int q = 0; q < 3; ++q) d[q] += t.w * g[q];
    return static_cast<int>(FTLM_OK);
  };
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const size_t idx = static_cast<size_t>(nu * (n + 1) + nd);
      const double w = std::exp(x[idx] - lnZ);
      if (!(w > 0.0)) continue;
      dmu += bT * w * N[idx];
      dbeta += w * (mu * N[idx] - e_s[idx]);
      if (!(w >= kGcWeightCutoff)) continue;
      ftlm_sector *rs = nullptr, *ro = nullptr;
      rc = sector_create(p, nu, nd, &parts, &rs);
      if (rc) return rc;
      Term t{SectorPtr(rs), nullptr, idx, w};
      rc = sector_create(&pop, nu, nd, &op_parts, &ro);
      if (rc) return rc;
      t.op.reset(ro);
      const bool c64 = grad_is_c64(rs, M, method);
      if (c64 && (rs->plan.max_up_deg > 120 || ro->plan.max_up_deg > 120))
        return fail(FTLM_ERR_UNSUPPORTED, "batched path: more than 120 up-hop sources per string");
      if (grad_is_fused(rs, ro, c64)) {
        fused[c64 ? 1 : 0].push_back(std::move(t));
        continue;
      }
      std::vector<ChainGrad> cg;
      rc = grad_one(rs, ro, bT, R, M, seed, method, start_mode, &cg);
      if (!rc) rc = add(t, cg);
      if (rc) return rc;
    }
  for (int c64 = 0; c64 < 2; ++c64) {
    std::vector<ftlm_sector*> hs, ho;
    for (const Term& t : fused[c64]) {
      hs.push_back(t.s.get());
      ho.push_back(t.op.get());
    }
    if (hs.empty()) continue;
    std::vector<std::vector<ChainGrad>> cg;
    const int mode = method == 1 ? FTLM_START_PHILOX : start_mode;
    rc = c64 ? grad_fused<float4>(hs, ho, bT, R, M, seed, mode, &cg) : grad_fused<double2>(hs, ho, bT, R, M, seed, mode, &cg);
    for (size_t i = 0; !rc && i < hs.size(); ++i) rc = add(fused[c64][i], cg[i]);
    if (rc) return rc;
  }
  grad[0] = d[0];
  grad[1] = d[1];
  grad[2] = d[2];
  grad[3] = dmu;
  grad[4] = dbeta;
  return FTLM_OK;
} catch (...) {
  return caught();
}

// Per-chain log quadrature and energy ratio with a converged eigen-decomposition (implicit QL
// on the GPU, symeig.cu), the quadrature the gradient differentiates; same layout as
// ftlm_gpu_tridiag_quadrature.
int ftlm_gpu_tridiag_quadrature_exact(const double* alpha, const double* beta, const int* n, int nc, int ld,
                                      const double* bts, int n_bt, double* logq, double* energy) try {
  if (nc < 0 || ld <= 0 || n_bt < 0 || !alpha || !beta || !n || (n_bt > 0 && (!bts || !logq || !energy)))
    return fail(FTLM_ERR_INVALID, "bad arguments");
  if (ld > kMaxEig) return fail(FTLM_ERR_UNSUPPORTED, "tridiagonal size > 160 is not supported by the GPU eigen-solver");
  for (int c = 0; c < nc; ++c)
    if (n[c] < 0 || n[c] > ld) return fail(FTLM_ERR_INVALID, "chain length outside [0, ld]");
  if (static_cast<long long>(nc) * n_bt > 0x7fffffffLL) return fail(FTLM_ERR_INVALID, "n_chains * n_bt exceeds 2^31 - 1");
  if (nc == 0 || n_bt == 0) return FTLM_OK;
  const size_t mat = static_cast<size_t>(nc) * ld * sizeof(double);
  const size_t outb = static_cast<size_t>(nc) * n_bt * sizeof(double);
  Scratch mem;
  const size_t o_da = mem.add(mat), o_db = mem.add(mat), o_dn = mem.add(nc * sizeof(int)), o_dl = mem.add(mat);
  const size_t o_dw = mem.add(mat), o_dbt = mem.add(n_bt * sizeof(double)), o_dq = mem.add(outb);
  const size_t o_de = mem.add(outb), o_di = mem.add(nc * sizeof(int));
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_da), alpha, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_db), beta, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dn), n, nc * sizeof(int), cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dbt), bts, n_bt * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(symeig_tridiag(mem.at<double>(o_da), mem.at<double>(o_db), mem.at<int>(o_dn), nc, ld, mem.at<double>(o_dl), mem.at<double>(o_dw),
                        nullptr, mem.at<int>(o_di), nullptr));
  CU_TRY(quad_eval(mem.at<double>(o_dl), mem.at<double>(o_dw), mem.at<int>(o_dn), nc, ld, mem.at<double>(o_dbt), n_bt, mem.at<double>(o_dq),
                   mem.at<double>(o_de), nullptr));
  std::vector<int> info(static_cast<size_t>(nc));
  CU_TRY(cudaMemcpy(info.data(), mem.at<void>(o_di), nc * sizeof(int), cudaMemcpyDeviceToHost));
  for (int c = 0; c < nc; ++c)
    if (n[c] > 0 && info[static_cast<size_t>(c)] != 0) return fail(FTLM_ERR_NUMERIC, "GPU eigen-solver did not converge");
  CU_TRY(cudaMemcpy(logq, mem.at<void>(o_dq), outb, cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(energy, mem.at<void>(o_de), outb, cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

// Host-only helper exposed for tests: eigenvalues/eigenvectors of a symmetric tridiagonal.
int ftlm_gpu_tridiag_eigvec(const double* alpha, const double* beta, int n, double* lam, double* Z) try {
  if (n < 0 || (n > 0 && (!alpha || !lam || !Z || (n > 1 && !beta)))) return fail(FTLM_ERR_INVALID, "bad arguments");
  const std::string err = tridiag_eigvec(n, alpha, beta, lam, Z);
  if (!err.empty()) return fail(FTLM_ERR_NUMERIC, err);
  return FTLM_OK;
} catch (...) {
  return caught();
}

// Host-only helper exposed for tests: the Duhamel weight matrix of one tridiagonal.
int ftlm_gpu_duhamel_weights(const double* alpha, const double* beta, int n, double bT, double* K, double* g,
                             double* lam_min) try {
  if (n < 0 || (n > 0 && (!alpha || !K || !g || (n > 1 && !beta)))) return fail(FTLM_ERR_INVALID, "bad arguments");
  const std::string err = duhamel_weights(n, alpha, beta, bT, K, g, lam_min);
  if (!err.empty()) return fail(FTLM_ERR_NUMERIC, err);
  return FTLM_OK;
} catch (...) {
  return caught();
}

}  // extern "C"

