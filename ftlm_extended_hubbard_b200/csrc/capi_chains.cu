// Host side of the fused Lanczos chains of many sectors (chains.cu): launches by size class, and the sectors' ln Z and
// energy with the chains' tridiagonals never leaving the device.
#include <thread>

#include "capi_internal.hpp"
#include "workers.hpp"

using namespace ftlm_b200;
using namespace ftlm_b200::capi;

namespace ftlm_b200 {
namespace capi {

// The reference's start vectors (src/lanczos.cpp:140-175) before normalisation.  The entries of a shorter vector are
// the first ones of a longer vector of the same seed, so the longest of each seed serves every sector.
void reference_normals(int64_t dim, int R, unsigned seed, std::vector<std::complex<double>>* out) {
  out->resize(static_cast<size_t>(R) * dim);
  const int hw = static_cast<int>(std::max(1u, std::min(32u, std::thread::hardware_concurrency())));
  share_out(static_cast<int64_t>(R) * dim < 4096 ? 1 : hw, R, [&](int64_t r) {
    std::mt19937 rng(seed + static_cast<unsigned>(r) * 100003u);
    std::normal_distribution<double> gauss(0.0, 1.0);
    std::complex<double>* v = out->data() + static_cast<size_t>(r) * dim;
    for (int64_t i = 0; i < dim; ++i) {
      const double re = gauss(rng);
      const double im = gauss(rng);
      v[i] = {re, im};
    }
  });
}

int chains_run(const std::vector<ftlm_sector*>& secs, int R, int M, unsigned seed, int start_mode, bool c64,
               ChainRun* run, void* store, const std::vector<int64_t>* store_base, bool keep_scale) {
  if (start_mode != FTLM_START_REFERENCE && start_mode != FTLM_START_PHILOX)
    return fail(FTLM_ERR_INVALID, "unknown start_mode");
  const int ns = static_cast<int>(secs.size());
  const int per = c64 ? 2 : 1, planes = (R + per - 1) / per;
  struct Item {
    ChainDesc d;
    int size;
    bool smem, phase, xor_real;
    int64_t dim;
    size_t bytes;
    int group() const { return size * 8 + (smem ? 4 : 0) + (phase ? 2 : 0) + (xor_real ? 1 : 0); }
  };
  std::vector<DevSector> devs;
  std::vector<Item> items;
  int64_t max_dim = 0;
  for (int i = 0; i < ns; ++i) {
    const DevSector& S = secs[static_cast<size_t>(i)]->dev;
    devs.push_back(S);
    max_dim = std::max(max_dim, S.dim);
    const bool phase = S.dn_g.ent && S.dn_g.phase, xor_real = S.dn_g.ent && S.dn_g.xor_real;  // forms of its table entries
    const int rows = chain_rows(S, c64, phase);
    const bool smem = rows == static_cast<int>(S.Du);
    if (rows == 0) return fail(FTLM_ERR_UNSUPPORTED, "fused chains: a row of the sector does not fit shared memory");
    for (int p = 0; p < planes; ++p) {
      ChainDesc d{};
      d.sector = i;
      d.out = i * R + per * p;
      d.chains = std::min(per, R - per * p);
      d.seed = seed + static_cast<unsigned>(per * p) * 100003u;
      d.rows = rows;
      if (store_base) {
        d.store = (*store_base)[static_cast<size_t>(i)] + static_cast<int64_t>(p) * S.dim;
        d.store_step = static_cast<int64_t>(planes) * S.dim;
      }
      items.push_back(Item{d, chain_class(S.dim), smem, phase, xor_real, S.dim, chain_elements(S) * 16 * 3});
    }
  }
  std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) {
    if (a.group() != b.group()) return a.group() < b.group();
    return a.dim > b.dim;
  });
  cudaStream_t st = secs[0]->stream;
  const size_t nc = static_cast<size_t>(ns) * R;
  const size_t o_a = run->mem.array<double>(nc * M), o_b = run->mem.array<double>(nc * M);
  const size_t o_u = run->mem.array<int>(nc);
  const size_t o_s = keep_scale ? run->mem.array<double>(nc * M) : 0;
  CU_TRY(run->mem.commit());
  run->alpha = run->mem.at<double>(o_a);
  run->beta = run->mem.at<double>(o_b);
  run->used = run->mem.at<int>(o_u);
  CU_TRY(cudaMemsetAsync(run->alpha, 0, nc * M * sizeof(double), st));
  CU_TRY(cudaMemsetAsync(run->beta, 0, nc * M * sizeof(double), st));
  std::vector<double> ones;
  if (keep_scale) {
    ones.assign(nc * M, 1.0);
    run->scale = run->mem.at<double>(o_s);
    CU_TRY(cudaMemcpyAsync(run->scale, ones.data(), nc * M * sizeof(double), cudaMemcpyHostToDevice, st));
  }
  std::vector<std::complex<double>> host;
  if (start_mode == FTLM_START_REFERENCE) {
    reference_normals(max_dim, R, seed, &host);
    for (auto& it : items) it.d.init = static_cast<int64_t>(it.d.out % R) * max_dim;
  }
  // The planes in pieces whose vectors fit a bounded scratch; the classes of a piece run side by side.
  constexpr size_t kScratch = size_t(16) << 30;
  size_t largest = 0, total = 0;
  for (const auto& it : items) {
    largest = std::max(largest, it.bytes);
    total += it.bytes;
  }
  Scratch mem;
  const size_t o_sec = mem.array<DevSector>(devs.size()), o_desc = mem.array<ChainDesc>(items.size());
  const size_t o_init = mem.array<double2>(host.size());
  const size_t o_scr = mem.add(std::min(total, std::max(kScratch, largest)));
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpyAsync(mem.at<void>(o_sec), devs.data(), devs.size() * sizeof(DevSector), cudaMemcpyHostToDevice, st));
  if (!host.empty())
    CU_TRY(cudaMemcpyAsync(mem.at<void>(o_init), host.data(), host.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
  std::vector<ChainDesc> descs(items.size());
  const size_t room = std::max(kScratch, largest);
  std::vector<size_t> piece{0};  // first items of the pieces
  {
    size_t at = 0;
    for (size_t i = 0; i < items.size(); ++i) {
      if (at + items[i].bytes > room) {
        piece.push_back(i);
        at = 0;
      }
      items[i].d.off = static_cast<int64_t>(at / 16);
      at += items[i].bytes;
      descs[i] = items[i].d;
    }
  }
  piece.push_back(items.size());
  CU_TRY(cudaMemcpyAsync(mem.at<void>(o_desc), descs.data(), descs.size() * sizeof(ChainDesc), cudaMemcpyHostToDevice, st));
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaError_t ce = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
  if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
  for (size_t pc = 0; pc + 1 < piece.size() && ce == cudaSuccess; ++pc) {
    ce = cudaEventRecord(ev[0], st);
    int stream = 0;
    for (size_t i = piece[pc]; i < piece[pc + 1] && ce == cudaSuccess;) {
      size_t j = i;
      size_t smem_bytes = 0;
      for (; j < piece[pc + 1] && items[j].group() == items[i].group(); ++j)
        smem_bytes = std::max(smem_bytes, chain_smem_bytes(devs[static_cast<size_t>(items[j].d.sector)], c64, items[j].phase, items[j].d.rows));
      cudaStream_t s2 = secs[static_cast<size_t>(std::min(stream, ns - 1))]->stream;
      ++stream;
      if (s2 != st) ce = cudaStreamWaitEvent(s2, ev[0], 0);
      ChainLaunch L{};
      L.sectors = mem.at<DevSector>(o_sec);
      L.descs = mem.at<ChainDesc>(o_desc) + i;
      L.blocks = static_cast<int>(j - i);
      L.size = items[i].size;
      L.smem = items[i].smem;
      L.phase = items[i].phase;
      L.xor_real = items[i].xor_real;
      L.smem_bytes = smem_bytes;
      L.M = M;
      L.scratch = mem.at<void>(o_scr);
      L.init = host.empty() ? nullptr : mem.at<double2>(o_init);
      L.alpha = run->alpha;
      L.beta = run->beta;
      L.used = run->used;
      L.scale = run->scale;
      L.store = store;
      if (ce == cudaSuccess) ce = chains_lanczos(L, c64, s2);
      if (s2 != st && ce == cudaSuccess) {
        ce = cudaEventRecord(ev[1], s2);
        if (ce == cudaSuccess) ce = cudaStreamWaitEvent(st, ev[1], 0);
      }
      i = j;
    }
  }
  const cudaError_t se = cudaStreamSynchronize(st);
  for (auto& e : ev)
    if (e) cudaEventDestroy(e);
  CU_TRY(ce);
  CU_TRY(se);
  mem.idle();
  run->mem.idle();
  return FTLM_OK;
}

int chains_ftlm(const std::vector<ftlm_sector*>& secs, int R, int M, unsigned seed, int start_mode, bool c64,
                const double* bts, int n_bt, bool converged, double* lnz, double* energy) {
  if (secs.empty() || n_bt == 0) return FTLM_OK;
  if (M > 160) return fail(FTLM_ERR_UNSUPPORTED, "tridiagonal size > 160 is not supported by the on-chip eigen-solver");
  const int ns = static_cast<int>(secs.size()), nc = ns * R;
  if (static_cast<long long>(nc) * n_bt > 0x7fffffffLL) return fail(FTLM_ERR_INVALID, "n_chains * n_bt exceeds 2^31 - 1");
  ChainRun run;
  int rc = chains_run(secs, R, M, seed, start_mode, c64, &run);
  if (rc) return rc;
  cudaStream_t st = secs[0]->stream;
  const size_t outb = static_cast<size_t>(nc) * n_bt * sizeof(double);
  std::vector<double> logd;
  for (const ftlm_sector* s : secs) logd.push_back(std::log(static_cast<double>(s->plan.dim)));
  Scratch mem;
  const size_t mat = static_cast<size_t>(nc) * M;
  const size_t o_l = mem.array<double>(mat), o_w = mem.array<double>(mat), o_q = mem.add(outb), o_e = mem.add(outb);
  const size_t o_i = mem.array<int>(nc), o_in = mem.array<double>(n_bt + logd.size());
  const size_t o_out = mem.array<double>(2 * ns * n_bt);
  CU_TRY(mem.commit());
  std::vector<double> in(bts, bts + n_bt), out(2 * static_cast<size_t>(ns) * n_bt);
  in.insert(in.end(), logd.begin(), logd.end());
  CU_TRY(cudaMemcpyAsync(mem.at<void>(o_in), in.data(), in.size() * sizeof(double), cudaMemcpyHostToDevice, st));
  const double *bt = mem.at<double>(o_in), *ld = bt + n_bt;
  double *lam = mem.at<double>(o_l), *w = mem.at<double>(o_w), *lq = mem.at<double>(o_q), *eq = mem.at<double>(o_e);
  double *z = mem.at<double>(o_out), *e = z + static_cast<size_t>(ns) * n_bt;
  if (converged)
    CU_TRY(symeig_tridiag(run.alpha, run.beta, run.used, nc, M, lam, w, nullptr, mem.at<int>(o_i), st));
  else
    CU_TRY(quad_jacobi(run.alpha, run.beta, run.used, nc, M, 0, 1e-14, lam, w, st));
  run.mem.busy();
  CU_TRY(quad_eval(lam, w, run.used, nc, M, bt, n_bt, lq, eq, st));
  CU_TRY(quad_sectors(lq, eq, run.used, ns, R, n_bt, ld, z, e, st));
  CU_TRY(cudaMemcpyAsync(out.data(), z, out.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  std::vector<int> bad(static_cast<size_t>(nc), 0);
  if (converged) CU_TRY(cudaMemcpyAsync(bad.data(), mem.at<void>(o_i), nc * sizeof(int), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  mem.idle();
  run.mem.idle();
  std::copy(out.begin(), out.begin() + ns * n_bt, lnz);
  std::copy(out.begin() + ns * n_bt, out.end(), energy);
  for (int b : bad)
    if (b == 1) return fail(FTLM_ERR_NUMERIC, "GPU eigen-solver did not converge");
  return FTLM_OK;
}

}  // namespace capi
}  // namespace ftlm_b200
