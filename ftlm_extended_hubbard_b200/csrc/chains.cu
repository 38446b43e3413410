// Fused Lanczos of many small sectors; contract in chains.cuh.
//
// One block per plane (chains.cuh) runs all M steps: a warp takes 32 output strings of one row, a lane one state, with
// the row pass's gauge-table walk for the down hops and the row's source list (the same for the whole warp) for the up
// hops; then the dot products, the update and the norm over the block's own vectors.  The vector that the hops gather
// from is staged in shared memory where it fits (14,336 states with their padding), else in the block's scratch.
// Rows have a pitch of Dd + 8 elements whose last 8 stay zero: the target of the table's padding entries, and harmless
// to the flat elementwise passes.  Bound by the latency of the gathers and of four block reductions a step; it exists
// because a step of a small sector otherwise costs five kernel launches, whatever its size: 3x3
// batched sweep (100 sectors, 60 steps) 336 -> 127 ms, most of that in the host's allocations.
// Same FP32 order of operations per element as planes.cu, so complex64 chains agree with that path up to the order of
// the FP64 sums.  Sums are in a fixed order: bitwise repeatable.
#include <algorithm>

#include "chains.cuh"
#include "philox.cuh"
#include "planes_dev.cuh"

namespace ftlm_b200 {

namespace {

constexpr size_t kMaxSmem = 227 * 1024;

// Totals of NV doubles over the block, in every thread.
template <int NV>
__device__ __forceinline__ void all_totals(double (&v)[NV], double* sh /* NV * 33 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    if (lane == 0) sh[i * 33 + warp] = v[i];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double s = lane < nw ? sh[i * 33 + lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
      if (lane == 0) sh[i * 33 + 32] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = sh[i * 33 + 32];
}

// Down hops of string d from the padded per-string list (sectors without the gauge table).
template <class P>
__device__ __forceinline__ typename P::T list_hops(const DevSector& S, const typename P::T* row, int d, typename P::T acc) {
  const int64_t e1 = S.dn_csr_ptr[d + 1];
  for (int64_t e = S.dn_csr_ptr[d]; e < e1; ++e) {
    const uint32_t q = S.dn_csr_ent[e];
    P::cmac(acc, P::dn_coef(S, q), row[q >> 9]);
  }
  return acc;
}

template <class P, bool kSmem, bool kPhase>
__global__ void __launch_bounds__(1024, 1) chains_kernel(const DevSector* __restrict__ sectors,
                                                         const ChainDesc* __restrict__ descs, int M,
                                                         typename P::T* __restrict__ scratch,
                                                         const double2* __restrict__ init, double* __restrict__ alpha,
                                                         double* __restrict__ beta, int* __restrict__ used,
                                                         double* __restrict__ scale, typename P::T* __restrict__ store) {
  using T = typename P::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[2 * P::kC * 33];
  const ChainDesc cd = descs[blockIdx.x];
  const DevSector S = sectors[cd.sector];
  const int Dd = static_cast<int>(S.Dd), Du = static_cast<int>(S.Du), pitch = Dd + 8;
  const int V = Du * pitch, dim = static_cast<int>(S.dim);
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  T* wk = scratch + cd.off;
  T* y = wk + V;
  T* wkm1 = y + V;
  typename P::Cf* tab = reinterpret_cast<typename P::Cf*>(smem_raw);
  const DevGauge G = S.dn_g;
  const size_t tab_bytes = kPhase ? 0 : (G.ent ? static_cast<size_t>(G.nt) * 8 * sizeof(typename P::Cf) : 0);
  T* xs = kSmem ? reinterpret_cast<T*>(smem_raw + ((tab_bytes + 15) & ~size_t(15))) : wkm1 + V;
  const RowCoefs<P> rc(G);
  if (!kPhase && G.ent)
    for (int i = tid; i < G.nt * 8; i += nt) tab[i] = P::coef(G.tab[i >> 3]);
  const bool phase = kPhase && G.phase;
  // padding: zero in every vector
  for (int i = tid; i < Du * 8; i += nt) {
    const int o = (i >> 3) * pitch + Dd + (i & 7);
    wk[o] = y[o] = wkm1[o] = P::zero();
    xs[o] = P::zero();
  }
  // start vector: Philox (chain q: key seed + q * 100003) or the caller's, in the gauge basis
  double n0[P::kC] = {};
  for (int i = tid; i < dim; i += nt) {
    const uint32_t r = static_cast<uint32_t>(i) / static_cast<uint32_t>(Dd), c = static_cast<uint32_t>(i) - r * Dd;
    const double g = gauge_sign(S.umask[r], S.dmask[c]) ? -1.0 : 1.0;
    decltype(P::narrow(0.0, 0.0)) z[P::kC];
#pragma unroll
    for (int q = 0; q < P::kC; ++q) {
      const double2 n = init ? init[cd.init + i] : philox_normal(i, cd.seed + static_cast<unsigned>(q) * 100003u);
      z[q] = P::narrow(g * n.x, g * n.y);
      n0[q] += static_cast<double>(z[q].x) * z[q].x + static_cast<double>(z[q].y) * z[q].y;
    }
    wk[r * pitch + c] = P::make(z);
  }
  all_totals<P::kC>(n0, sh);
  double s_in[P::kC], c2[P::kC];
  bool active[P::kC];
  int steps[P::kC];
#pragma unroll
  for (int q = 0; q < P::kC; ++q) {
    const double n = sqrt(n0[q]);
    active[q] = !(n < 1e-18);
    s_in[q] = active[q] ? 1.0 / n : 0.0;
    c2[q] = 0.0;
    steps[q] = 0;
    if (scale && tid == 0 && q < cd.chains) scale[static_cast<int64_t>(cd.out + q) * M] = active[q] ? n : 1.0;
  }
  const int ng = (Dd + 31) >> 5, items = Du * ng;
  for (int k = 0; k < M; ++k) {
    for (int i = tid; i < V; i += nt) {
      T v = wk[i];
      if (P::kScaled) v = P::times(s_in[0], v);
      xs[i] = P::filtered(v, 1.0);
    }
    if (store) {
      T* out = store + cd.store + static_cast<int64_t>(k) * cd.store_step;
      for (int i = tid; i < dim; i += nt) {
        const uint32_t r = static_cast<uint32_t>(i) / static_cast<uint32_t>(Dd);
        out[i] = wk[i + 8 * r];
      }
    }
    __syncthreads();
    double d[2 * P::kC] = {};
    for (int it = warp; it < items; it += nw) {
      const int r = it / ng, pos = (it - r * ng) * 32 + lane;
      const T* row = xs + r * pitch;
      const bool in = pos < Dd;
      const int c = !in ? 0 : G.ent ? gauge_string(G, pos) : pos;
      const uint32_t u = S.umask[r];
      T acc = P::times(diag_value(S, u, S.dmask[c], S.cnt_uu[r], S.cnt_dd[c], S.wpl[r]), row[c]);
      if (G.ent) {
        if (phase) {
          RowSum<P, 1, kPhase> s;
          s.base = reinterpret_cast<const unsigned char*>(row);
          s.line = 0;
          s.acc[0] = acc;
          s.walk(G, pos, tab, rc);
          acc = s.acc[0];
        } else {
          RowSum<P, 1, false> s;
          s.base = reinterpret_cast<const unsigned char*>(row);
          s.line = 0;
          s.acc[0] = acc;
          s.walk(G, pos, tab, rc);
          acc = s.acc[0];
        }
      } else if (in) {
        acc = list_hops<P>(S, row, c, acc);
      }
      T up = P::zero();
      const T* col = xs + c;
      const int j1 = S.up_ptr[r + 1];
      int j = S.up_ptr[r];
      for (; j + 4 <= j1; j += 4) {
        T v[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) v[t] = col[S.up_src[j + t] * pitch];
#pragma unroll
        for (int t = 0; t < 4; ++t) P::cmac(up, P::up_coef(S, j + t), v[t]);
      }
      for (; j < j1; ++j) P::cmac(up, P::up_coef(S, j), col[S.up_src[j] * pitch]);
      if (in) {
        const T v = P::add_scaled(acc, up, 1.0);
        y[r * pitch + c] = v;
        P::dot(d, wk[r * pitch + c], v, s_in[0]);
      }
    }
    all_totals<2 * P::kC>(d, sh);
    double c1r[P::kC], c1i[P::kC];
#pragma unroll
    for (int q = 0; q < P::kC; ++q) {
      const double f = P::kScaled ? 1.0 : s_in[q] * s_in[q];
      const double zr = d[2 * q] * f, zi = d[2 * q + 1] * f;
      c1r[q] = zr * s_in[q];
      c1i[q] = zi * s_in[q];
      if (active[q] && tid == 0 && q < cd.chains) alpha[static_cast<int64_t>(cd.out + q) * M + k] = zr;
    }
    double n2[P::kC] = {};
    for (int i = tid; i < V; i += nt) {
      const T yv = y[i], av = wk[i], pv = k > 0 ? wkm1[i] : P::zero();
      decltype(P::narrow(0.0, 0.0)) w[P::kC];
#pragma unroll
      for (int q = 0; q < P::kC; ++q) {
        const auto yy = P::get(yv, q), aa = P::get(av, q), pp = P::get(pv, q);
        const double sy = P::kScaled ? 1.0 : s_in[q];
        double wr = sy * static_cast<double>(yy.x) - (c1r[q] * aa.x - c1i[q] * aa.y);
        double wi = sy * static_cast<double>(yy.y) - (c1r[q] * aa.y + c1i[q] * aa.x);
        wr -= c2[q] * pp.x;
        wi -= c2[q] * pp.y;
        w[q] = P::narrow(wr, wi);
        n2[q] += static_cast<double>(w[q].x) * w[q].x + static_cast<double>(w[q].y) * w[q].y;
      }
      y[i] = P::make(w);
    }
    all_totals<P::kC>(n2, sh);
    bool any = false;
#pragma unroll
    for (int q = 0; q < P::kC; ++q) {
      if (active[q]) {
        steps[q] = k + 1;
        if (n2[q] < 1e-24) {  // src/lanczos.cpp:187: alpha_k kept, no beta_k
          active[q] = false;
          s_in[q] = c2[q] = 0.0;
        } else {
          const double b = sqrt(n2[q]);
          if (tid == 0 && q < cd.chains) {
            beta[static_cast<int64_t>(cd.out + q) * M + k] = b;
            if (scale && k + 1 < M) scale[static_cast<int64_t>(cd.out + q) * M + k + 1] = b;
          }
          c2[q] = b * s_in[q];
          s_in[q] = 1.0 / b;
        }
      } else {
        s_in[q] = c2[q] = 0.0;
      }
      any = any || active[q];
    }
    if (!any) break;
    T* t = wkm1;
    wkm1 = wk;
    wk = y;
    y = t;
  }
  if (tid == 0)
    for (int q = 0; q < P::kC && q < cd.chains; ++q) used[cd.out + q] = steps[q];
}

constexpr int kClassThreads[4] = {1024, 512, 256, 64};

}  // namespace

int chain_class(int64_t dim) { return dim > 4096 ? 0 : dim > 1024 ? 1 : dim > 256 ? 2 : 3; }

size_t chain_smem_bytes(const DevSector& S, bool c64, bool phase, bool with_vector) {
  const size_t tab = !S.dn_g.ent || phase ? 0 : static_cast<size_t>(S.dn_g.nt) * 8 * (c64 ? 8 : 16);
  return (tab + 15) / 16 * 16 + (with_vector ? chain_elements(S) * 16 : 0);
}

bool chain_in_smem(const DevSector& S, bool c64, bool phase) {
  return chain_smem_bytes(S, c64, phase, true) + 2048 <= kMaxSmem;  // 2048: the reduction's own
}

namespace {

template <class P>
cudaError_t launch(const ChainLaunch& L, cudaStream_t st) {
  using T = typename P::T;
  using K = void (*)(const DevSector*, const ChainDesc*, int, T*, const double2*, double*, double*, int*, double*, T*);
  const K k = L.smem ? (L.phase ? chains_kernel<P, true, true> : chains_kernel<P, true, false>)
                     : (L.phase ? chains_kernel<P, false, true> : chains_kernel<P, false, false>);
  const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(L.smem_bytes));
  if (e != cudaSuccess) return e;
  k<<<L.blocks, kClassThreads[L.size], L.smem_bytes, st>>>(L.sectors, L.descs, L.M, static_cast<T*>(L.scratch), L.init, L.alpha,
                                                    L.beta, L.used, L.scale, static_cast<T*>(L.store));
  return cudaGetLastError();
}

}  // namespace

cudaError_t chains_lanczos(const ChainLaunch& L, bool c64, cudaStream_t st) {
  if (L.blocks <= 0) return cudaSuccess;
  return c64 ? launch<C64>(L, st) : launch<C128>(L, st);
}

}  // namespace ftlm_b200
