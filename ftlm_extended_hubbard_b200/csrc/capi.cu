// C ABI (include/ftlm_gpu.h): sector handles, H·v, Lanczos, quadrature, grand-canonical sweep.
// Host orchestration only; every floating-point operation on sector vectors runs in the
// kernels of hv.cu / lanczos.cu / quad.cu.  No exception crosses the ABI.  The batched path,
// the parameter gradient and the momentum blocks are in capi_batched.cu, capi_grad.cu and
// capi_orbit.cu.
#include <atomic>
#include <map>

#include "capi_internal.hpp"

using namespace ftlm_b200;
using namespace ftlm_b200::capi;

// Quadrature of the complex128 sector path (ftlm_gpu_set_quadrature).
static std::atomic<bool> g_quad_converged{false};

namespace {
thread_local std::string g_err;
}  // namespace

int ftlm_b200::capi::fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

int ftlm_b200::capi::caught() noexcept {
  try {
    try {
      throw;
    } catch (const std::bad_alloc&) {
      return fail(FTLM_ERR_NOMEM, "host allocation failed");
    } catch (const std::exception& e) {  // a size that no vector can have
      return fail(FTLM_ERR_NOMEM, e.what());
    }
  } catch (...) {  // not even the message
  }
  return FTLM_ERR_NOMEM;
}

int ftlm_b200::set_error(int code, const char* msg) { return fail(code, msg); }

namespace ftlm_b200 {
namespace capi {

void reference_start(int64_t dim, unsigned seed, std::vector<std::complex<double>>* q) {
  std::mt19937 rng(seed);
  std::normal_distribution<double> gauss(0.0, 1.0);
  q->resize(static_cast<size_t>(dim));
  auto& v = *q;
  for (int64_t i = 0; i < dim; ++i) {
    const double re = gauss(rng);
    const double im = gauss(rng);
    v[static_cast<size_t>(i)] = {re, im};
  }
  double n0 = 0.0;
  for (const auto& z : v) n0 += std::norm(z);
  n0 = std::sqrt(n0);
  if (n0 < 1e-18) {
    std::fill(v.begin(), v.end(), std::complex<double>(0.0, 0.0));
    v[0] = {1.0, 0.0};
  } else {
    const std::complex<double> sc(1.0 / n0, 0.0);
    for (auto& z : v) z *= sc;
  }
}

}  // namespace capi
}  // namespace ftlm_b200

namespace {

// A sector's tables in one block: laid out in a host image, copied at once.
class TableArena {
 public:
  template <class T>
  size_t add(const std::vector<T>& v) {
    const size_t at = (image_.size() + 255) / 256 * 256, bytes = std::max<size_t>(v.size(), 1) * sizeof(T);
    image_.resize(at + bytes);
    if (!v.empty()) std::memcpy(image_.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
  cudaError_t upload(void** block, size_t* got) {
    const cudaError_t e = pool_take(image_.size(), block, got);
    if (e != cudaSuccess) return e;
    base_ = static_cast<char*>(*block);
    const cudaError_t c = cudaMemcpy(base_, image_.data(), image_.size(), cudaMemcpyHostToDevice);
    return c == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : c;  // other streams may read it now
  }
  template <class T>
  const T* at(size_t off) const {
    return reinterpret_cast<const T*>(base_ + off);
  }

 private:
  std::vector<char> image_;
  char* base_ = nullptr;
};

int upload_plan(ftlm_sector* s) {
  const SectorPlan& P = s->plan;
  DevSector& D = s->dev;
  CU_TRY(cudaGetDevice(&s->device));
  s->stream.set_device(s->device);
  D.n = P.n;
  D.Du = P.up.D;
  D.Dd = P.dn.D;
  D.dim = P.dim;
  D.U = P.U;
  D.V = P.V;
  std::vector<float2> upc32(P.up_src.size()), dnc32s(P.dn_coef.size());
  for (size_t i = 0; i < upc32.size(); ++i)
    upc32[i] = make_float2(static_cast<float>(P.up_coef[2 * i]), static_cast<float>(P.up_coef[2 * i + 1]));
  for (size_t i = 0; i < dnc32s.size() / 2; ++i) {
    const float x = static_cast<float>(P.dn_coef[2 * i]), y = static_cast<float>(P.dn_coef[2 * i + 1]);
    dnc32s[2 * i] = make_float2(x, y);
    dnc32s[2 * i + 1] = make_float2(-x, -y);
  }
  TableArena A;
  const size_t um = A.add(P.up.masks), dm = A.add(P.dn.masks), cuu = A.add(P.cnt_uu), cdd = A.add(P.cnt_dd);
  const size_t wp = A.add(P.wpl), uptr = A.add(P.up_ptr), usrc = A.add(P.up_src), ucf = A.add(P.up_coef);
  const size_t ulh = A.add(P.up_lohi), ucf32 = A.add(upc32), gptr = A.add(P.dn_gptr), dent = A.add(P.dn_ent);
  const size_t cptr = A.add(P.dn_csr_ptr), cent = A.add(P.dn_csr_ent), dcf = A.add(P.dn_coef), dcf32s = A.add(dnc32s);
  const size_t dnm = A.add(P.dn_nmask), fl = A.add(std::vector<int>(4, 0));
  const GaugeTable& G = P.dn_g;
  const size_t gent = G.ok ? A.add(G.ent) : 0, ggrp = G.ok ? A.add(G.grp) : 0, gperm = G.ok ? A.add(G.perm) : 0;
  const size_t gtab = G.ok && !G.tab.empty() ? A.add(G.tab) : 0, upk = P.up_pk_ok ? A.add(P.up_pk) : 0;
  CU_TRY(A.upload(&s->tables, &s->tables_bytes));
  D.bt_cols = 1;  // 128-column slabs of the batched column pass (ftlm_gpu_batched_autotune times the others)
  D.dn_g = DevGauge{};
  D.dn_g.real2[0] = G.real2[0];
  D.dn_g.real2[1] = G.real2[1];
  if (G.ok) {
    D.dn_g.ent = A.at<uint32_t>(gent);
    D.dn_g.grp = A.at<int4>(ggrp);
    D.dn_g.perm = A.at<uint8_t>(gperm);
    D.dn_g.nt = static_cast<int>(G.tab.size() / 2);
    D.dn_g.phase = G.phase ? 1 : 0;
    D.dn_g.xor_real = G.xor_real ? 1 : 0;
    D.dn_g.pc = G.pc;
    D.dn_g.ps = G.ps;
    if (D.dn_g.nt > 0) D.dn_g.tab = A.at<double2>(gtab);
  }
  D.up_pk = P.up_pk_ok ? A.at<uint32_t>(upk) : nullptr;
  D.up_real2[0] = P.up_real2[0];
  D.up_real2[1] = P.up_real2[1];
  D.up_pc = P.up_pc;
  D.up_ps = P.up_ps;
  D.umask = A.at<uint32_t>(um);
  D.dmask = A.at<uint32_t>(dm);
  D.cnt_uu = A.at<int32_t>(cuu);
  D.cnt_dd = A.at<int32_t>(cdd);
  D.wpl = A.at<uint4>(wp);
  D.up_ptr = A.at<int32_t>(uptr);
  D.up_src = A.at<int32_t>(usrc);
  D.up_coef = A.at<double2>(ucf);
  D.up_lohi = A.at<uint32_t>(ulh);
  D.dn_gptr = A.at<int64_t>(gptr);
  D.dn_ent = A.at<uint32_t>(dent);
  D.dn_csr_ptr = A.at<int64_t>(cptr);
  D.up_coef32 = A.at<float2>(ucf32);
  D.dn_coef32s = A.at<float2>(dcf32s);
  D.dn_csr_ent = A.at<uint32_t>(cent);
  D.dn_coef = A.at<double2>(dcf);
  D.dn_nmask = A.at<uint32_t>(dnm);
  D.n_dn_hops = P.dn_pad_hop;
  D.flags = const_cast<int*>(A.at<int>(fl));
  s->on_device = true;
  return FTLM_OK;
}

int create_common(int n_sites, int n_up, int n_dn, double U, double V, const ftlm_hop* hops, int n_hops,
                  const ftlm_pair* pairs, int n_pairs, bool device, ftlm_sector** out, PlanParts* parts = nullptr) {
  if (!out) return fail(FTLM_ERR_INVALID, "null output handle");
  *out = nullptr;
  if (n_hops < 0 || n_pairs < 0 || (n_hops > 0 && !hops) || (n_pairs > 0 && !pairs))
    return fail(FTLM_ERR_INVALID, "bad hopping/pair arrays");
  auto* s = new (std::nothrow) ftlm_sector();
  if (!s) return fail(FTLM_ERR_NOMEM, "host allocation failed");
  std::string err;
  try {
    std::vector<HopIn> hv(static_cast<size_t>(n_hops));
    for (int i = 0; i < n_hops; ++i) hv[i] = HopIn{hops[i].from, hops[i].to, hops[i].spin, hops[i].coeff_re, hops[i].coeff_im};
    std::vector<PairIn> pv(static_cast<size_t>(n_pairs));
    for (int i = 0; i < n_pairs; ++i) pv[i] = PairIn{pairs[i].i, pairs[i].j};
    err = build_plan(n_sites, n_up, n_dn, U, V, hv, pv, &s->plan, parts ? parts->find(parts->up, n_up) : nullptr,
                     parts ? parts->find(parts->dn, n_dn) : nullptr);
    if (parts && err.empty()) parts->keep(s->plan);
    if (device && err.empty()) {
      const int rc = upload_plan(s);
      if (rc != FTLM_OK) {
        delete s;
        return rc;
      }
    }
  } catch (const std::bad_alloc&) {
    delete s;
    return fail(FTLM_ERR_NOMEM, "host allocation failed while building the sector plan");
  }
  if (!err.empty()) {
    delete s;
    const bool unsup = err.find("not supported") != std::string::npos || err.find("2^31") != std::string::npos;
    return fail(unsup ? FTLM_ERR_UNSUPPORTED : FTLM_ERR_INVALID, err);
  }
  *out = s;
  return FTLM_OK;
}


}  // namespace

int ftlm_b200::capi::need_device(const ftlm_sector* s) {
  if (!s) return fail(FTLM_ERR_INVALID, "null sector");
  if (!s->on_device) return fail(FTLM_ERR_INVALID, "sector was created host-only");
  return FTLM_OK;
}

int ftlm_b200::capi::sector_create(const ftlm_params* p, int n_up, int n_dn, PlanParts* parts, ftlm_sector** out) {
  if (!p) return fail(FTLM_ERR_INVALID, "null params");
  if (p->Lx <= 0 || p->Ly <= 0) return fail(FTLM_ERR_INVALID, "Lx, Ly must be positive");
  std::vector<HopIn> hv;
  std::vector<PairIn> pv;
  build_geometry(p->Lx, p->Ly, p->t, p->tp, p->phi_x, p->phi_y, &hv, &pv);
  std::vector<ftlm_hop> h(hv.size());
  for (size_t i = 0; i < hv.size(); ++i) h[i] = ftlm_hop{hv[i].from, hv[i].to, hv[i].spin, hv[i].cre, hv[i].cim};
  std::vector<ftlm_pair> q(pv.size());
  for (size_t i = 0; i < pv.size(); ++i) q[i] = ftlm_pair{pv[i].i, pv[i].j};
  const int rc = create_common(p->Lx * p->Ly, n_up, n_dn, p->U, p->V, h.data(), static_cast<int>(h.size()), q.data(),
                               static_cast<int>(q.size()), true, out, parts);
  if (rc == FTLM_OK) {
    (*out)->Lx = p->Lx;
    (*out)->Ly = p->Ly;
  }
  return rc;
}

extern "C" {

const char* ftlm_gpu_last_error(void) { return g_err.c_str(); }

const char* ftlm_gpu_version_string(void) { return "ftlm_extended_hubbard_b200 0.1.0 (sm_100a)"; }

int ftlm_gpu_device_count(int* n) {
  if (!n) return fail(FTLM_ERR_INVALID, "null");
  *n = 0;
  const cudaError_t e = cudaGetDeviceCount(n);
  if (e != cudaSuccess) {
    *n = 0;
    return fail(FTLM_ERR_CUDA, std::string("cudaGetDeviceCount: ") + cudaGetErrorString(e));
  }
  return FTLM_OK;
}

int ftlm_gpu_build_geometry(const ftlm_params* p, ftlm_hop* hops, int max_hops, int* n_hops, ftlm_pair* pairs,
                            int max_pairs, int* n_pairs) try {
  if (!p || !n_hops || !n_pairs) return fail(FTLM_ERR_INVALID, "null argument");
  if (p->Lx <= 0 || p->Ly <= 0) return fail(FTLM_ERR_INVALID, "Lx, Ly must be positive");
  std::vector<HopIn> hv;
  std::vector<PairIn> pv;
  build_geometry(p->Lx, p->Ly, p->t, p->tp, p->phi_x, p->phi_y, &hv, &pv);
  *n_hops = static_cast<int>(hv.size());
  *n_pairs = static_cast<int>(pv.size());
  for (int i = 0; i < *n_hops && i < max_hops && hops; ++i)
    hops[i] = ftlm_hop{hv[i].from, hv[i].to, hv[i].spin, hv[i].cre, hv[i].cim};
  for (int i = 0; i < *n_pairs && i < max_pairs && pairs; ++i) pairs[i] = ftlm_pair{pv[i].i, pv[i].j};
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_sector_create_hops(int n_sites, int n_up, int n_dn, double U, double V, const ftlm_hop* hops, int n_hops,
                                const ftlm_pair* pairs, int n_pairs, ftlm_sector** out) {
  return create_common(n_sites, n_up, n_dn, U, V, hops, n_hops, pairs, n_pairs, true, out);
}

int ftlm_gpu_sector_create_host(int n_sites, int n_up, int n_dn, double U, double V, const ftlm_hop* hops, int n_hops,
                                const ftlm_pair* pairs, int n_pairs, ftlm_sector** out) {
  return create_common(n_sites, n_up, n_dn, U, V, hops, n_hops, pairs, n_pairs, false, out);
}

int ftlm_gpu_sector_create(const ftlm_params* p, int n_up, int n_dn, ftlm_sector** out) try {
  return sector_create(p, n_up, n_dn, nullptr, out);
} catch (...) {
  return caught();
}

int ftlm_gpu_sector_destroy(ftlm_sector* s) {
  delete s;
  return FTLM_OK;
}

int ftlm_gpu_sector_dim(const ftlm_sector* s, long long* dim) {
  if (!s || !dim) return fail(FTLM_ERR_INVALID, "null argument");
  *dim = s->plan.dim;
  return FTLM_OK;
}

int ftlm_gpu_sector_masks(const ftlm_sector* s, uint64_t* up, uint64_t* dn) {
  if (!s || !up || !dn) return fail(FTLM_ERR_INVALID, "null argument");
  const auto& P = s->plan;
  for (int64_t r = 0; r < P.up.D; ++r)
    for (int64_t c = 0; c < P.dn.D; ++c) {
      up[r * P.dn.D + c] = P.up.masks[static_cast<size_t>(r)];
      dn[r * P.dn.D + c] = P.dn.masks[static_cast<size_t>(c)];
    }
  return FTLM_OK;
}

int ftlm_gpu_sector_index_of(const ftlm_sector* s, uint64_t up, uint64_t dn, long long* index) {
  if (!s || !index) return fail(FTLM_ERR_INVALID, "null argument");
  *index = -1;
  if ((up >> 32) != 0 || (dn >> 32) != 0) return FTLM_OK;
  const int64_t ru = s->plan.up.rank(static_cast<uint32_t>(up));
  const int64_t rd = s->plan.dn.rank(static_cast<uint32_t>(dn));
  if (ru >= 0 && rd >= 0) *index = ru * s->plan.dn.D + rd;
  return FTLM_OK;
}

int ftlm_gpu_sector_state(const ftlm_sector* s, long long index, uint64_t* up, uint64_t* dn) {
  if (!s || !up || !dn) return fail(FTLM_ERR_INVALID, "null argument");
  if (index < 0 || index >= s->plan.dim) return fail(FTLM_ERR_INVALID, "FockBasis index out of range");
  *up = s->plan.up.masks[static_cast<size_t>(index / s->plan.dn.D)];
  *dn = s->plan.dn.masks[static_cast<size_t>(index % s->plan.dn.D)];
  return FTLM_OK;
}

int ftlm_gpu_sector_down_table_gauge(const ftlm_sector* s, int* available, long long* n_groups, long long* n_entries,
                                     int* n_table, int* groups, uint32_t* entries, double* table, double* real2) {
  if (!s || !available || !n_groups || !n_entries || !n_table) return fail(FTLM_ERR_INVALID, "null argument");
  const GaugeTable& G = s->plan.dn_g;
  *available = G.ok ? 1 : 0;
  *n_groups = G.ok ? static_cast<long long>(G.grp.size() / 4) : 0;
  *n_entries = G.ok ? static_cast<long long>(G.ent.size()) : 0;
  *n_table = G.ok ? static_cast<int>(G.tab.size() / 2) : 0;
  if (!G.ok) return FTLM_OK;
  if (groups) std::copy(G.grp.begin(), G.grp.end(), groups);
  if (entries) std::copy(G.ent.begin(), G.ent.end(), entries);
  if (table) std::copy(G.tab.begin(), G.tab.end(), table);
  if (real2) std::copy(G.real2, G.real2 + 2, real2);
  return FTLM_OK;
}

int ftlm_gpu_sector_down_table_form(const ftlm_sector* s, int* phase, double* pc_ps, int* xor_real,
                                    unsigned char* lane_perm) {
  if (!s || !phase) return fail(FTLM_ERR_INVALID, "null argument");
  const GaugeTable& G = s->plan.dn_g;
  *phase = (G.ok && G.phase) ? 1 : 0;
  if (xor_real) *xor_real = (G.ok && G.xor_real) ? 1 : 0;
  if (lane_perm && G.ok) std::copy(G.perm.begin(), G.perm.end(), lane_perm);
  if (pc_ps) {
    pc_ps[0] = G.pc;
    pc_ps[1] = G.ps;
  }
  return FTLM_OK;
}

int ftlm_gpu_sector_up_table_packed(const ftlm_sector* s, int* available, long long* n_entries, int32_t* ptr,
                                    uint32_t* entries, double* real2, double* pc_ps) {
  if (!s || !available || !n_entries) return fail(FTLM_ERR_INVALID, "null argument");
  const SectorPlan& P = s->plan;
  *available = P.up_pk_ok ? 1 : 0;
  *n_entries = P.up_pk_ok ? static_cast<long long>(P.up_pk.size()) : 0;
  if (!P.up_pk_ok) return FTLM_OK;
  if (ptr) std::copy(P.up_ptr.begin(), P.up_ptr.end(), ptr);
  if (entries) std::copy(P.up_pk.begin(), P.up_pk.end(), entries);
  if (real2) std::copy(P.up_real2, P.up_real2 + 2, real2);
  if (pc_ps) {
    pc_ps[0] = P.up_pc;
    pc_ps[1] = P.up_ps;
  }
  return FTLM_OK;
}

int ftlm_gpu_sector_stats(const ftlm_sector* s, double* mean_up, double* mean_dn, long long* du, long long* dd) {
  if (!s) return fail(FTLM_ERR_INVALID, "null sector");
  if (mean_up) *mean_up = s->plan.mean_up_sources;
  if (mean_dn) *mean_dn = s->plan.mean_dn_sources;
  if (du) *du = s->plan.up.D;
  if (dd) *dd = s->plan.dn.D;
  return FTLM_OK;
}

int ftlm_gpu_sector_down_table(const ftlm_sector* s, long long* n_groups, long long* n_entries, long long* gptr,
                               uint32_t* entries, int* pad_hop) {
  if (!s || !n_groups || !n_entries) return fail(FTLM_ERR_INVALID, "null argument");
  *n_groups = static_cast<long long>(s->plan.dn_gptr.size()) - 1;
  *n_entries = static_cast<long long>(s->plan.dn_ent.size());
  if (gptr) std::copy(s->plan.dn_gptr.begin(), s->plan.dn_gptr.end(), gptr);
  if (entries) std::copy(s->plan.dn_ent.begin(), s->plan.dn_ent.end(), entries);
  if (pad_hop) *pad_hop = s->plan.dn_pad_hop;
  return FTLM_OK;
}

int ftlm_gpu_sector_diag(const ftlm_sector* s, long long index, double* value) {
  if (!s || !value) return fail(FTLM_ERR_INVALID, "null argument");
  if (index < 0 || index >= s->plan.dim) return fail(FTLM_ERR_INVALID, "index out of range");
  *value = plan_diag(s->plan, index / s->plan.dn.D, index % s->plan.dn.D);
  return FTLM_OK;
}

int ftlm_gpu_set_apply_path(ftlm_sector* s, int path) {
  if (!s || path < 0 || path > 3) return fail(FTLM_ERR_INVALID, "bad path");
  s->apply_path = path;
  s->pinned = path != 0;
  s->use_once = path == 0;
  return FTLM_OK;
}

int ftlm_gpu_apply(ftlm_sector* s, const double* x, double* y, void* stream) {
  int rc = need_device(s);
  if (rc) return rc;
  if (!x || !y) return fail(FTLM_ERR_INVALID, "null vector");
  if (x == y) return fail(FTLM_ERR_INVALID, "x and y must not alias");
  return s->apply(reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), static_cast<cudaStream_t>(stream));
}

int ftlm_gpu_apply_profiled(ftlm_sector* s, const double* x, double* y, void* stream, float* ms_passes, int* n_passes) {
  int rc = need_device(s);
  if (rc) return rc;
  if (!x || !y || !ms_passes || !n_passes) return fail(FTLM_ERR_INVALID, "null argument");
  if (x == y) return fail(FTLM_ERR_INVALID, "x and y must not alias");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int path = s->effective_path();
  const DevSector d = s->dev_for(path);
  cudaEvent_t ev[3];
  for (auto& e : ev) CU_TRY(cudaEventCreate(&e));
  CU_TRY(cudaEventRecord(ev[0], st));
  const bool once = s->once();
  if (once) {
    CU_TRY(hv_launch_once(s->dev, reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), st));
    CU_TRY(cudaEventRecord(ev[1], st));
  } else if (path >= 2) {
    CU_TRY(hv_launch_pass(d, reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), 0, st,
                          s->cols_variant));
    CU_TRY(cudaEventRecord(ev[1], st));
    CU_TRY(hv_launch_pass(d, reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), 1, st,
                          s->cols_variant));
  } else {
    CU_TRY(hv_launch(d, reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), path, st));
    CU_TRY(cudaEventRecord(ev[1], st));
  }
  CU_TRY(cudaEventRecord(ev[2], st));
  CU_TRY(cudaEventSynchronize(ev[2]));
  CU_TRY(cudaEventElapsedTime(&ms_passes[0], ev[0], ev[1]));
  *n_passes = 1;
  if (path >= 2 && !once) {
    CU_TRY(cudaEventElapsedTime(&ms_passes[1], ev[1], ev[2]));
    *n_passes = 2;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  return FTLM_OK;
}

int ftlm_gpu_apply_host(ftlm_sector* s, const double* x, double* y) {
  int rc = need_device(s);
  if (rc) return rc;
  if (!x || !y) return fail(FTLM_ERR_INVALID, "null vector");
  const size_t bytes = static_cast<size_t>(s->plan.dim) * sizeof(double2);
  if (!s->hx.p) {
    CU_TRY(s->hx.alloc(bytes));
    CU_TRY(s->hy.alloc(bytes));
  }
  CU_TRY(cudaMemcpyAsync(s->hx.p, x, bytes, cudaMemcpyHostToDevice, s->stream));
  rc = s->apply(s->hx.as<double2>(), s->hy.as<double2>(), s->stream);
  if (rc) return rc;
  CU_TRY(cudaMemcpyAsync(y, s->hy.p, bytes, cudaMemcpyDeviceToHost, s->stream));
  CU_TRY(cudaStreamSynchronize(s->stream));
  return FTLM_OK;
}

}  // extern "C"

int ftlm_b200::capi::planes_lanczos(ftlm_sector* s, int R, int M, unsigned seed, int start_mode, std::vector<double>* A,
                                    std::vector<double>* B, std::vector<int>* used) {
  if (start_mode != FTLM_START_REFERENCE && start_mode != FTLM_START_PHILOX)
    return fail(FTLM_ERR_INVALID, "unknown start_mode");
  A->assign(static_cast<size_t>(R) * M, 0.0);
  B->assign(static_cast<size_t>(R) * M, 0.0);
  used->assign(static_cast<size_t>(R), 0);
  const int64_t dim = s->plan.dim;
  const DevSector S = s->planes_dev();
  cudaStream_t st = s->stream;
  BtWs& ws = s->planes;
  const int group = pl_group(S, false, std::min(R, kBtChains));
  CU_TRY(ws.ensure(static_cast<size_t>(group) * dim * sizeof(double2), M, pl_items_doubles(S, false, group)));
  const size_t tab = static_cast<size_t>(M) * kBtChains * sizeof(double);
  std::vector<double> ha(static_cast<size_t>(M) * kBtChains), hb(static_cast<size_t>(M) * kBtChains);
  std::vector<int> hu(kBtChains);
  std::vector<std::complex<double>> start;
  const bool given = start_mode == FTLM_START_REFERENCE;
  for (int r0 = 0; r0 < R; r0 += group) {  // the scalars of a group are read before the next one starts
    const int np = std::min(group, R - r0);
    const unsigned seed_g = seed + static_cast<unsigned>(r0) * 100003u;
    const PlaneState z = ws.state(0);
    double2 *wk = ws.buf[0].as<double2>(), *y = ws.buf[1].as<double2>(), *wkm1 = ws.buf[2].as<double2>();
    CU_TRY(cudaMemsetAsync(ws.alpha.p, 0, tab, st));
    CU_TRY(cudaMemsetAsync(ws.beta.p, 0, tab, st));
    if (given) {
      reference_normals(dim, np, seed_g, &start);
      CU_TRY(cudaMemcpyAsync(wk, start.data(), start.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
    }
    CU_TRY(pl_start(S, wk, np, seed_g, given, z, st));
    for (int k = 0; k < M; ++k) {
      CU_TRY(pl_step(S, wk, wkm1, y, np, k, z, st));
      double2* t = wkm1;
      wkm1 = wk;
      wk = y;
      y = t;
    }
    CU_TRY(cudaMemcpyAsync(ha.data(), ws.alpha.p, tab, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hb.data(), ws.beta.p, tab, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(hu.data(), ws.used.p, hu.size() * sizeof(int), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    for (int r = 0; r < np; ++r) {
      const size_t ch = static_cast<size_t>(r0 + r);
      (*used)[ch] = hu[static_cast<size_t>(r)];
      for (int k = 0; k < M; ++k) {
        (*A)[ch * M + k] = ha[static_cast<size_t>(k) * kBtChains + r];
        (*B)[ch * M + k] = hb[static_cast<size_t>(k) * kBtChains + r];
      }
    }
  }
  // A handle keeps the three vectors of one chain, or what L2 holds of several (given back and taken again, those cost
  // 4x3 (4,5) with four chains 0.4 % of a call); more goes back to the pool, which ftlm_gpu_batched_release empties.
  constexpr size_t kHandleKeep = size_t(40) << 20;  // a vector
  if (group > 1 && ws.cap > kHandleKeep) ws.release();
  return FTLM_OK;
}

namespace {

// A chain's alpha and beta without their padding: one that ended has no last beta (0; one that is not a number counts).
void trim_chain(int n, std::vector<double>* a, std::vector<double>* b) {
  a->resize(static_cast<size_t>(n));
  b->resize(static_cast<size_t>(n > 0 && (*b)[static_cast<size_t>(n) - 1] != 0.0 ? n : std::max(0, n - 1)));
}

}  // namespace

extern "C" {

int ftlm_gpu_lanczos(ftlm_sector* s, int max_steps, unsigned seed, int start_mode, double* alpha, double* beta,
                     int* n_beta, int* used) try {
  int rc = need_device(s);
  if (rc) return rc;
  std::vector<double> a, b;
  if (s->chains(1) == ftlm_sector::Chains::fused && max_steps > 0) {
    // few states: all steps in one kernel
    ChainRun run;
    rc = chains_run({s}, 1, max_steps, seed, start_mode, false, &run);
    if (rc) return rc;
    int n = 0;
    CU_TRY(cudaMemcpy(&n, run.used, sizeof(int), cudaMemcpyDeviceToHost));
    a.resize(static_cast<size_t>(max_steps));
    b.resize(static_cast<size_t>(max_steps));
    CU_TRY(cudaMemcpy(a.data(), run.alpha, a.size() * sizeof(double), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(b.data(), run.beta, b.size() * sizeof(double), cudaMemcpyDeviceToHost));
    trim_chain(n, &a, &b);
  } else if (s->chains(1) == ftlm_sector::Chains::planes && max_steps > 0) {
    std::vector<int> u;
    rc = planes_lanczos(s, 1, max_steps, seed, start_mode, &a, &b, &u);
    if (rc) return rc;
    trim_chain(u[0], &a, &b);
  } else {
    rc = run_lanczos(
        s->plan.dim, [s](const double2* x, double2* y, cudaStream_t st) { return s->apply(x, y, st); }, s->ws,
        max_steps, seed, start_mode, s->stream, &a, &b);
  }
  if (rc) return rc;
  if (alpha) std::copy(a.begin(), a.end(), alpha);
  if (beta) std::copy(b.begin(), b.end(), beta);
  if (n_beta) *n_beta = static_cast<int>(b.size());
  if (used) *used = static_cast<int>(a.size());
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_lanczos_op(long long dim, ftlm_apply_fn fn, void* ctx, int max_steps, unsigned seed, int start_mode,
                        double* alpha, double* beta, int* n_beta, int* used) {
  if (!fn) return fail(FTLM_ERR_INVALID, "null operator");
  LanczosWs ws;
  std::vector<double> a, b;
  const int rc = run_lanczos(
      dim,
      [fn, ctx](const double2* x, double2* y, cudaStream_t st) {
        if (cudaStreamSynchronize(st) != cudaSuccess) return fail(FTLM_ERR_CUDA, "stream sync before operator");
        fn(reinterpret_cast<const double*>(x), reinterpret_cast<double*>(y), ctx);
        if (cudaDeviceSynchronize() != cudaSuccess) return fail(FTLM_ERR_CUDA, "operator callback failed");
        return FTLM_OK;
      },
      ws, max_steps, seed, start_mode, nullptr, &a, &b);
  if (rc) return rc;
  if (alpha) std::copy(a.begin(), a.end(), alpha);
  if (beta) std::copy(b.begin(), b.end(), beta);
  if (n_beta) *n_beta = static_cast<int>(b.size());
  if (used) *used = static_cast<int>(a.size());
  return FTLM_OK;
}

int ftlm_gpu_lanczos_host_op(long long dim, ftlm_host_apply_fn fn, void* ctx, int max_steps, unsigned seed,
                             int start_mode, double* alpha, double* beta, int* n_beta, int* used) {
  if (!fn) return fail(FTLM_ERR_INVALID, "null operator");
  LanczosWs ws;
  std::vector<double> a, b, hx, hy;
  try {
    hx.resize(static_cast<size_t>(std::max(0LL, dim)) * 2);
    hy.resize(static_cast<size_t>(std::max(0LL, dim)) * 2);
  } catch (const std::bad_alloc&) {
    return fail(FTLM_ERR_NOMEM, "host staging buffers");
  }
  const int rc = run_lanczos(
      dim,
      [&](const double2* x, double2* y, cudaStream_t st) {
        CU_TRY(cudaMemcpyAsync(hx.data(), x, dim * sizeof(double2), cudaMemcpyDeviceToHost, st));
        CU_TRY(cudaStreamSynchronize(st));
        fn(hx.data(), hy.data(), ctx);
        CU_TRY(cudaMemcpyAsync(y, hy.data(), dim * sizeof(double2), cudaMemcpyHostToDevice, st));
        CU_TRY(cudaStreamSynchronize(st));
        return FTLM_OK;
      },
      ws, max_steps, seed, start_mode, nullptr, &a, &b);
  if (rc) return rc;
  if (alpha) std::copy(a.begin(), a.end(), alpha);
  if (beta) std::copy(b.begin(), b.end(), beta);
  if (n_beta) *n_beta = static_cast<int>(b.size());
  if (used) *used = static_cast<int>(a.size());
  return FTLM_OK;
}

int ftlm_gpu_ftlm_combine(const double* logq, const double* energy_r, const int* used, int R, int n_bt, double log_dim,
                          double* lnz, double* energy) try {
  if (R <= 0 || n_bt < 0 || !logq || !energy_r || !used || !lnz || !energy) return fail(FTLM_ERR_INVALID, "bad arguments");
  if (n_bt == 0) return FTLM_OK;
  const size_t qb = static_cast<size_t>(R) * n_bt * sizeof(double);
  Scratch mem;
  const size_t o_dq = mem.add(qb), o_de = mem.add(qb), o_dn = mem.add(R * sizeof(int));
  const size_t o_dz = mem.add(n_bt * sizeof(double)), o_den = mem.add(n_bt * sizeof(double));
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_dq), logq, qb, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_de), energy_r, qb, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dn), used, R * sizeof(int), cudaMemcpyHostToDevice));
  CU_TRY(quad_sector(mem.at<double>(o_dq), mem.at<double>(o_de), mem.at<int>(o_dn), R, n_bt, log_dim, mem.at<double>(o_dz),
                     mem.at<double>(o_den), nullptr));
  CU_TRY(cudaMemcpy(lnz, mem.at<void>(o_dz), n_bt * sizeof(double), cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(energy, mem.at<void>(o_den), n_bt * sizeof(double), cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_tridiag_eig(const double* alpha, const double* beta, const int* n, int nc, int ld, int max_rot, double tol,
                         double* lam, double* w0) try {
  if (nc < 0 || ld <= 0 || !alpha || !beta || !n || !lam || !w0) return fail(FTLM_ERR_INVALID, "bad arguments");
  if (ld > 160) return fail(FTLM_ERR_UNSUPPORTED, "tridiagonal size > 160 is not supported by the on-chip Jacobi");
  for (int c = 0; c < nc; ++c)
    if (n[c] < 0 || n[c] > ld) return fail(FTLM_ERR_INVALID, "chain length outside [0, ld]");
  if (nc == 0) return FTLM_OK;
  const size_t mat = static_cast<size_t>(nc) * ld * sizeof(double);
  Scratch mem;
  const size_t o_da = mem.add(mat), o_db = mem.add(mat), o_dn = mem.add(nc * sizeof(int)), o_dl = mem.add(mat);
  const size_t o_dw = mem.add(mat);
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_da), alpha, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_db), beta, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dn), n, nc * sizeof(int), cudaMemcpyHostToDevice));
  CU_TRY(quad_jacobi(mem.at<double>(o_da), mem.at<double>(o_db), mem.at<int>(o_dn), nc, ld, max_rot, tol, mem.at<double>(o_dl),
                     mem.at<double>(o_dw), nullptr));
  CU_TRY(cudaMemcpy(lam, mem.at<void>(o_dl), mat, cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(w0, mem.at<void>(o_dw), mat, cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_tridiag_quadrature(const double* alpha, const double* beta, const int* n, int nc, int ld,
                                const double* bts, int n_bt, double* logq, double* energy) try {
  if (nc < 0 || ld <= 0 || n_bt < 0 || !alpha || !beta || !n || !bts || !logq || !energy)
    return fail(FTLM_ERR_INVALID, "bad arguments");
  if (ld > 160) return fail(FTLM_ERR_UNSUPPORTED, "tridiagonal size > 160 is not supported by the on-chip Jacobi");
  for (int c = 0; c < nc; ++c)
    if (n[c] < 0 || n[c] > ld) return fail(FTLM_ERR_INVALID, "chain length outside [0, ld]");
  if (static_cast<long long>(nc) * n_bt > 0x7fffffffLL) return fail(FTLM_ERR_INVALID, "n_chains * n_bt exceeds 2^31 - 1");
  if (nc == 0 || n_bt == 0) return FTLM_OK;
  const size_t mat = static_cast<size_t>(nc) * ld * sizeof(double);
  const size_t outb = static_cast<size_t>(nc) * n_bt * sizeof(double);
  Scratch mem;
  const size_t o_da = mem.add(mat), o_db = mem.add(mat), o_dn = mem.add(nc * sizeof(int)), o_dl = mem.add(mat);
  const size_t o_dw = mem.add(mat), o_dbt = mem.add(n_bt * sizeof(double)), o_dq = mem.add(outb);
  const size_t o_de = mem.add(outb);
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_da), alpha, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_db), beta, mat, cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dn), n, nc * sizeof(int), cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dbt), bts, n_bt * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(quad_jacobi(mem.at<double>(o_da), mem.at<double>(o_db), mem.at<int>(o_dn), nc, ld, 0, 1e-14, mem.at<double>(o_dl), mem.at<double>(o_dw),
                     nullptr));
  CU_TRY(quad_eval(mem.at<double>(o_dl), mem.at<double>(o_dw), mem.at<int>(o_dn), nc, ld, mem.at<double>(o_dbt), n_bt, mem.at<double>(o_dq),
                   mem.at<double>(o_de), nullptr));
  CU_TRY(cudaMemcpy(logq, mem.at<void>(o_dq), outb, cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(energy, mem.at<void>(o_de), outb, cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_ritz_values(const double* alpha, const double* beta, int n, int k, double* ritz) try {
  if (n <= 0 || k <= 0 || !alpha || !ritz || (n > 1 && !beta)) return fail(FTLM_ERR_INVALID, "bad arguments");
  k = std::min(k, n);
  Scratch mem;
  const size_t o_da = mem.add(n * sizeof(double)), o_db = mem.add(n * sizeof(double));
  const size_t o_dr = mem.add(k * sizeof(double));
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_da), alpha, n * sizeof(double), cudaMemcpyHostToDevice));
  if (n > 1) CU_TRY(cudaMemcpy(mem.at<void>(o_db), beta, (n - 1) * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(ritz_bisect(mem.at<double>(o_da), mem.at<double>(o_db), n, k, mem.at<double>(o_dr), nullptr));
  CU_TRY(cudaMemcpy(ritz, mem.at<void>(o_dr), k * sizeof(double), cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_lanczos_extrema(ftlm_sector* s, int max_steps, unsigned seed, int start_mode, double* mn, double* mx,
                             int* steps_used) try {
  if (!mn || !mx) return fail(FTLM_ERR_INVALID, "null output");
  *mn = 0.0;
  *mx = 0.0;
  if (steps_used) *steps_used = 0;
  std::vector<double> a(std::max(1, max_steps)), b(std::max(1, max_steps));
  int nb = 0, used = 0;
  int rc = ftlm_gpu_lanczos(s, max_steps, seed, start_mode, a.data(), b.data(), &nb, &used);
  if (rc) return rc;
  if (steps_used) *steps_used = used;
  if (used == 0) return FTLM_OK;
  // src/lanczos.cpp:106-123, 211-231: 120 Jacobi rotations, tol 1e-15, on beta[0..used-2].
  if (used > 160) return fail(FTLM_ERR_UNSUPPORTED, "more than 160 Lanczos steps for the on-chip Jacobi");
  std::vector<double> lam(static_cast<size_t>(used)), w(static_cast<size_t>(used));
  std::vector<double> bt(static_cast<size_t>(used), 0.0);
  for (int i = 0; i + 1 < used && i < nb; ++i) bt[static_cast<size_t>(i)] = b[static_cast<size_t>(i)];
  int n1 = used;
  if (used == 1) {
    *mn = a[0];
    *mx = a[0];
    return FTLM_OK;
  }
  rc = ftlm_gpu_tridiag_eig(a.data(), bt.data(), &n1, 1, used, 120, 1e-15, lam.data(), w.data());
  if (rc) return rc;
  *mn = *std::min_element(lam.begin(), lam.end());
  *mx = *std::max_element(lam.begin(), lam.end());
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_set_quadrature(int mode) {
  if (mode != FTLM_QUAD_REFERENCE && mode != FTLM_QUAD_CONVERGED) return fail(FTLM_ERR_INVALID, "unknown quadrature");
  g_quad_converged.store(mode == FTLM_QUAD_CONVERGED);
  return FTLM_OK;
}

int ftlm_gpu_ftlm_sector(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed, int start_mode,
                         double* lnz, double* energy) try {
  return plain_sector_ftlm(s, bts, n_bt, R, M, seed, start_mode, plain_quadrature_converged(), lnz, energy);
} catch (...) {
  return caught();
}

}  // extern "C"

namespace ftlm_b200 {
namespace capi {

int plain_sector_ftlm(ftlm_sector* s, const double* bts, int n_bt, int R, int M, unsigned seed, int start_mode,
                      bool converged, double* lnz, double* energy) {
  int rc = need_device(s);
  if (rc) return rc;
  if (n_bt < 0 || (n_bt > 0 && (!bts || !lnz || !energy))) return fail(FTLM_ERR_INVALID, "bad arguments");
  const int64_t dim = s->plan.dim;
  R = std::max(1, R);
  M = std::max(1, M);
  if (M > 160) return fail(FTLM_ERR_UNSUPPORTED, "more than 160 Lanczos steps for the on-chip Jacobi");
  if (dim == 1) {  // src/ftlm_thermo.cpp:219-223: apply H to e_0.
    const double one[2] = {1.0, 0.0};
    double h00[2] = {0.0, 0.0};
    rc = ftlm_gpu_apply_host(s, one, h00);
    if (rc) return rc;
    for (int b = 0; b < n_bt; ++b) {
      lnz[b] = -bts[b] * h00[0];
      energy[b] = h00[0];
    }
    return FTLM_OK;
  }
  if (s->chains(R) == ftlm_sector::Chains::fused)
    return chains_ftlm({s}, R, M, seed, start_mode, false, bts, n_bt, converged, lnz, energy);
  std::vector<double> A(static_cast<size_t>(R) * M, 0.0), B(static_cast<size_t>(R) * M, 0.0);
  std::vector<int> nv(static_cast<size_t>(R), 0);
  if (s->chains(R) == ftlm_sector::Chains::planes) {
    rc = planes_lanczos(s, R, M, seed, start_mode, &A, &B, &nv);
    if (rc) return rc;
  } else {
    for (int r = 0; r < R; ++r) {
      const unsigned seed_r = seed + static_cast<unsigned>(r) * 100003u;
      int nb = 0, used = 0;
      rc = ftlm_gpu_lanczos(s, M, seed_r, start_mode, &A[static_cast<size_t>(r) * M], &B[static_cast<size_t>(r) * M], &nb,
                            &used);
      if (rc) return rc;
      nv[static_cast<size_t>(r)] = used;
    }
  }
  std::vector<double> lq(static_cast<size_t>(R) * n_bt), eq(static_cast<size_t>(R) * n_bt);
  rc = chain_quadrature(A.data(), B.data(), nv.data(), R, M, bts, n_bt, lq.data(), eq.data(), converged);
  if (rc) return rc;
  Scratch mem;
  const size_t o_dq = mem.add(lq.size() * sizeof(double)), o_de = mem.add(eq.size() * sizeof(double));
  const size_t o_dn = mem.add(nv.size() * sizeof(int)), o_dz = mem.add(n_bt * sizeof(double));
  const size_t o_den = mem.add(n_bt * sizeof(double));
  CU_TRY(mem.commit());
  CU_TRY(cudaMemcpy(mem.at<void>(o_dq), lq.data(), lq.size() * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_de), eq.data(), eq.size() * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dn), nv.data(), nv.size() * sizeof(int), cudaMemcpyHostToDevice));
  CU_TRY(quad_sector(mem.at<double>(o_dq), mem.at<double>(o_de), mem.at<int>(o_dn), R, n_bt, std::log(static_cast<double>(dim)),
                     mem.at<double>(o_dz), mem.at<double>(o_den), nullptr));
  CU_TRY(cudaMemcpy(lnz, mem.at<void>(o_dz), n_bt * sizeof(double), cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(energy, mem.at<void>(o_den), n_bt * sizeof(double), cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
}

int chain_quadrature(const double* A, const double* B, const int* n, int nc, int ld, const double* bts, int n_bt,
                     double* lq, double* eq, bool converged) {
  return converged ? ftlm_gpu_tridiag_quadrature_exact(A, B, n, nc, ld, bts, n_bt, lq, eq)
                   : ftlm_gpu_tridiag_quadrature(A, B, n, nc, ld, bts, n_bt, lq, eq);
}

bool plain_quadrature_converged() { return g_quad_converged.load(); }

}  // namespace capi
}  // namespace ftlm_b200

extern "C" {

int ftlm_gpu_gc_reduce(const double* lnz_s, const double* e_s, const int* N_s, int n_sec, const double* bts, int n_bt,
                       const double* mus, int n_mu, int n_sites, double* lnz_gc, double* n_avg, double* e_avg) try {
  if (n_sec < 0 || n_bt < 0 || n_mu < 0 || !lnz_s || !e_s || !N_s || !bts || !mus || !lnz_gc || !n_avg || !e_avg)
    return fail(FTLM_ERR_INVALID, "bad arguments");
  if (n_bt == 0 || n_mu == 0) return FTLM_OK;
  const size_t sb = static_cast<size_t>(std::max(n_sec, 1)) * n_bt * sizeof(double);
  const size_t gb = static_cast<size_t>(n_bt) * n_mu * sizeof(double);
  Scratch mem;
  const size_t o_dl = mem.add(sb), o_de = mem.add(sb), o_dN = mem.add(std::max(n_sec, 1) * sizeof(int));
  const size_t o_db = mem.add(n_bt * sizeof(double)), o_dm = mem.add(n_mu * sizeof(double)), o_o1 = mem.add(gb);
  const size_t o_o2 = mem.add(gb), o_o3 = mem.add(gb);
  CU_TRY(mem.commit());
  if (n_sec > 0) {
    CU_TRY(cudaMemcpy(mem.at<void>(o_dl), lnz_s, static_cast<size_t>(n_sec) * n_bt * sizeof(double), cudaMemcpyHostToDevice));
    CU_TRY(cudaMemcpy(mem.at<void>(o_de), e_s, static_cast<size_t>(n_sec) * n_bt * sizeof(double), cudaMemcpyHostToDevice));
    CU_TRY(cudaMemcpy(mem.at<void>(o_dN), N_s, n_sec * sizeof(int), cudaMemcpyHostToDevice));
  }
  CU_TRY(cudaMemcpy(mem.at<void>(o_db), bts, n_bt * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(cudaMemcpy(mem.at<void>(o_dm), mus, n_mu * sizeof(double), cudaMemcpyHostToDevice));
  CU_TRY(gc_reduce_dev(mem.at<double>(o_dl), mem.at<double>(o_de), mem.at<int>(o_dN), n_sec, mem.at<double>(o_db), n_bt, mem.at<double>(o_dm),
                       n_mu, n_sites, mem.at<double>(o_o1), mem.at<double>(o_o2), mem.at<double>(o_o3), nullptr));
  CU_TRY(cudaMemcpy(lnz_gc, mem.at<void>(o_o1), gb, cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(n_avg, mem.at<void>(o_o2), gb, cudaMemcpyDeviceToHost));
  CU_TRY(cudaMemcpy(e_avg, mem.at<void>(o_o3), gb, cudaMemcpyDeviceToHost));
  mem.idle();
  return FTLM_OK;
} catch (...) {
  return caught();
}

}  // extern "C"

namespace ftlm_b200 {
namespace capi {

int64_t g_fused_max_dim = kFusedSweepMax;

int fused_sectors_ftlm(const std::vector<ftlm_sector*>& secs, const std::vector<int>& out_idx, int R, int M,
                       unsigned seed, int start_mode, bool c64, const double* bts, int n_bt, double* lnz_s, double* e_s,
                       bool converged) {
  if (secs.empty()) return FTLM_OK;
  const size_t n = static_cast<size_t>(n_bt);
  std::vector<double> lz(secs.size() * n), en(secs.size() * n);
  const int rc = chains_ftlm(secs, R, M, seed, start_mode, c64, bts, n_bt, converged, lz.data(), en.data());
  if (rc) return rc;
  for (size_t i = 0; i < secs.size(); ++i) {
    const size_t dst = static_cast<size_t>(out_idx[i]) * n;
    std::copy(lz.begin() + i * n, lz.begin() + (i + 1) * n, lnz_s + dst);
    std::copy(en.begin() + i * n, en.begin() + (i + 1) * n, e_s + dst);
  }
  return FTLM_OK;
}

}  // namespace capi
}  // namespace ftlm_b200

extern "C" {

int ftlm_gpu_lanczos_sectors(ftlm_sector* const* secs, int n_sectors, int R, int M, unsigned seed, int start_mode,
                             double* alpha, double* beta, int* used) try {
  if (!secs || n_sectors < 0 || R <= 0 || M <= 0 || !alpha || !beta || !used) return fail(FTLM_ERR_INVALID, "bad arguments");
  // Sectors far beyond the fused path's range, or with rows too long for it, run their chains one at a time.
  constexpr int64_t kFusedMost = int64_t(1) << 22;
  std::vector<ftlm_sector*> v;
  std::vector<int> at;
  for (int i = 0; i < n_sectors; ++i) {
    int rc = need_device(secs[i]);
    if (rc) return rc;
    if (secs[i]->plan.dim <= kFusedMost && chain_rows(secs[i]->dev, false, false) > 0) {
      v.push_back(secs[i]);
      at.push_back(i);
      continue;
    }
    for (int r = 0; r < R; ++r) {
      const size_t row = static_cast<size_t>(i) * R + r;
      std::fill(alpha + row * M, alpha + (row + 1) * M, 0.0);
      std::fill(beta + row * M, beta + (row + 1) * M, 0.0);
      int nb = 0;
      rc = ftlm_gpu_lanczos(secs[i], M, seed + static_cast<unsigned>(r) * 100003u, start_mode, alpha + row * M,
                            beta + row * M, &nb, used + row);
      if (rc) return rc;
    }
  }
  if (v.empty()) return FTLM_OK;
  ChainRun run;
  const int rc = chains_run(v, R, M, seed, start_mode, false, &run);
  if (rc) return rc;
  const size_t rows = static_cast<size_t>(R), tab = rows * M;
  for (size_t i = 0; i < v.size(); ++i) {
    const size_t o = static_cast<size_t>(at[i]) * rows;
    CU_TRY(cudaMemcpy(alpha + o * M, run.alpha + i * tab, tab * sizeof(double), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(beta + o * M, run.beta + i * tab, tab * sizeof(double), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(used + o, run.used + i * rows, rows * sizeof(int), cudaMemcpyDeviceToHost));
  }
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_set_cols_variant(ftlm_sector* s, int variant) {
  if (!s || variant < 0 || variant > 5) return fail(FTLM_ERR_INVALID, "cols variant must be in [0, 6)");
  s->cols_variant = variant;
  s->cols_chosen = true;
  return FTLM_OK;
}

int ftlm_gpu_autotune_apply(ftlm_sector* s, int reps, int* path, int* cols_variant, float* ms) try {
  int rc = need_device(s);
  if (rc) return rc;
  reps = std::max(1, reps);
  const SectorPlan& P = s->plan;
  // one timing per sector shape and process
  static std::mutex mu;
  struct Choice {
    int path, variant;
    bool once;
  };
  static std::map<std::string, Choice> cache;
  auto take = [s](const Choice& c) {
    s->apply_path = c.path;
    s->cols_variant = c.variant;
    s->use_once = c.once;
    s->pinned = false;
    s->cols_chosen = c.path >= 2 && !c.once;  // else no slab was timed
  };
  char key[160];
  std::snprintf(key, sizeof(key), "%d/%d/%d/%zu/%zu/%d/%d", P.n, P.nu, P.nd, P.hu.size(), P.hd.size(), P.max_up_deg,
                P.max_dn_deg);
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      take(it->second);
      if (path) *path = s->apply_path;
      if (cols_variant) *cols_variant = s->cols_variant;
      if (ms) *ms = -1.0f;
      return FTLM_OK;
    }
  }
  const int64_t dim = P.dim;
  DevBuf x, y;
  CU_TRY(x.alloc(static_cast<size_t>(dim) * sizeof(double2)));
  CU_TRY(y.alloc(static_cast<size_t>(dim) * sizeof(double2)));
  cudaStream_t st = s->stream;
  CU_TRY(cudaMemsetAsync(x.p, 0, static_cast<size_t>(dim) * sizeof(double2), st));
  const double one[2] = {1.0, 0.0};
  CU_TRY(cudaMemcpyAsync(x.p, one, sizeof(double2), cudaMemcpyHostToDevice, st));
  cudaEvent_t e0, e1;
  CU_TRY(cudaEventCreate(&e0));
  CU_TRY(cudaEventCreate(&e1));
  int best_p = 1, best_v = 0;
  float best = 3.4e38f;
  const bool fast = hv_fast_path_ok(s->dev_for(2), P.max_up_deg);
  bool best_once = false;
  const int variants[11][2] = {{0, 0}, {1, 0}, {2, 0}, {2, 1}, {2, 2}, {3, 0}, {3, 1}, {3, 2}, {3, 3}, {3, 4}, {3, 5}};
  cudaError_t ce = cudaSuccess;
  for (const auto& v : variants) {
    const bool once = v[0] == 0;  // H v in one pass; reported as path 3, whose row pass it has
    if (once && !hv_once_ok(s->dev, P.max_up_deg)) continue;
    if (v[0] >= 2 && !fast) continue;
    if (v[0] == 3 && !s->path_available(3)) continue;
    if (v[1] >= 3 && !s->dev.up_pk) continue;
    const DevSector d = s->dev_for(v[0], v[1]);
    const int lp = v[0] == 3 ? 2 : v[0];
    auto run = [&]() {
      return once ? hv_launch_once(s->dev, x.as<double2>(), y.as<double2>(), st)
                  : hv_launch(d, x.as<double2>(), y.as<double2>(), lp, st, v[1]);
    };
    ce = run();  // warm-up
    if (ce == cudaSuccess) ce = cudaEventRecord(e0, st);
    for (int r = 0; r < reps && ce == cudaSuccess; ++r) ce = run();
    if (ce == cudaSuccess) ce = cudaEventRecord(e1, st);
    if (ce == cudaSuccess) ce = cudaEventSynchronize(e1);
    float t = 0.0f;
    if (ce == cudaSuccess) ce = cudaEventElapsedTime(&t, e0, e1);
    if (ce != cudaSuccess) break;
    if (t < best) {
      best = t;
      best_p = once ? 3 : v[0];
      best_v = v[1];
      best_once = once;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  CU_TRY(ce);
  take(Choice{best_p, best_v, best_once});
  {
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = Choice{best_p, best_v, best_once};
  }
  if (path) *path = best_p;
  if (cols_variant) *cols_variant = best_v;
  if (ms) *ms = best / static_cast<float>(reps);
  return FTLM_OK;
} catch (...) {
  return caught();
}

int ftlm_gpu_set_fused_max_dim(long long max_dim) {
  if (max_dim < 0) return fail(FTLM_ERR_INVALID, "max_dim must be >= 0");
  g_fused_max_dim = max_dim;
  return FTLM_OK;
}

int ftlm_gpu_gc_sweep(const ftlm_params* p, int R, int M, unsigned seed, int start_mode, const double* bts, int n_bt,
                      const double* mus, int n_mu, double* lnz_s, double* e_s, double* lnz_gc, double* n_avg,
                      double* e_avg) try {
  if (!p || !lnz_s || !e_s) return fail(FTLM_ERR_INVALID, "null argument");
  const int n = p->Lx * p->Ly;
  if (n <= 0 || n > 32) return fail(FTLM_ERR_INVALID, "FockBasis: require 1 <= n_sites <= 32 (bit packing)");
  const int nsec = (n + 1) * (n + 1);
  std::vector<int> N(static_cast<size_t>(nsec));
  PlanParts parts(n);
  OwnedSectors owned;
  std::vector<ftlm_sector*>& small = owned.v;  // sectors for the fused small-sector launch
  std::vector<int> small_idx;
  for (int nu = 0; nu <= n; ++nu)
    for (int nd = 0; nd <= n; ++nd) {
      const int idx = nu * (n + 1) + nd;  // benchmarks/bench_ftlm_nmu_rect.cpp:62
      N[static_cast<size_t>(idx)] = nu + nd;
      ftlm_sector* s = nullptr;
      int rc = sector_create(p, nu, nd, &parts, &s);
      if (rc) return rc;
      if (s->plan.dim >= 2 && s->plan.dim <= g_fused_max_dim && M <= 160 && chain_rows(s->dev, false, false) > 0) {  // fused below
        small.push_back(s);
        small_idx.push_back(idx);
        continue;
      }
      rc = ftlm_gpu_ftlm_sector(s, bts, n_bt, R, M, seed, start_mode, lnz_s + static_cast<size_t>(idx) * n_bt,
                                e_s + static_cast<size_t>(idx) * n_bt);
      ftlm_gpu_sector_destroy(s);
      if (rc) return rc;
    }
  const int rcf = fused_sectors_ftlm(small, small_idx, std::max(1, R), std::max(1, M), seed, start_mode, false, bts, n_bt,
                                     lnz_s, e_s, plain_quadrature_converged());
  if (rcf) return rcf;
  if (lnz_gc && n_avg && e_avg)
    return ftlm_gpu_gc_reduce(lnz_s, e_s, N.data(), nsec, bts, n_bt, mus, n_mu, n, lnz_gc, n_avg, e_avg);
  return FTLM_OK;
} catch (...) {
  return caught();
}

}  // extern "C"

