// Fused Lanczos of many small sectors; contract in chains.cuh.
//
// One block per plane (chains.cuh) runs all M steps: a warp takes 32 output strings of one row, a lane one state, with
// the row pass's gauge-table walk for the down hops and the row's source list (the same for the whole warp) for the up
// hops.  The walk serves the 32 strings in the table's order, which spreads its gathers over the shared-memory banks;
// the up hops read 32 neighbouring strings of a row, so they run in the strings' own order (of any 8
// of them in the table's order about 2.5 share the fullest bank group) and the sums change lanes by a shuffle.  Their list is the packed one where
// the sector has it: one word a source instead of three, two real FMAs a component instead of four.  Then the dot
// products, the update and the norm over the block's own vectors.  The vector that the hops gather from is staged in
// shared memory where it fits (14,336 states with their padding); else the rows are, a block of rows at a time, and the
// up hops read the block's scratch: 3x3 (4,4), 15,876 states, 146 us a step of one complex128 chain. Rows have a pitch of Dd + 8 elements whose last 8 stay zero:
// the target of the table's padding entries, and harmless to the flat elementwise passes.  Bound by the shared-memory
// pipe and instruction issue above 4,096 states (60 and 64 % in the 3x3 batched sweep's launch of 320 blocks; 85 % of the
// wavefronts before the lane change and the packed list, 13.4 -> 11.5 ms), by latency below; it exists because a step of a small sector otherwise costs
// five kernel launches, whatever its size: 3x3 batched sweep (100 sectors, 60 steps) 336 ms without it, 27.2 now, the host's
// allocations and tables included.
// Same FP32 order of operations per element as planes.cu, so complex64 chains agree with that path up to the order of
// the FP64 sums.  Sums are in a fixed order: bitwise repeatable.
#include <algorithm>

#include "chains.cuh"
#include "launch.cuh"
#include "philox.cuh"
#include "planes_dev.cuh"

namespace ftlm_b200 {

namespace {

constexpr size_t kMaxSmem = 227 * 1024, kOwnSmem = 2048;  // of which the reductions' own

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

template <class P, int kMost, bool kSmem, bool kPhase, bool kXor>
__global__ void __launch_bounds__(kMost, kMost == 1024 ? 1 : 2) chains_kernel(const DevSector* __restrict__ sectors,
                                                         const ChainDesc* __restrict__ descs, int M,
                                                         typename P::T* __restrict__ scratch,
                                                         const double2* __restrict__ init, double* __restrict__ alpha,
                                                         double* __restrict__ beta, int* __restrict__ used,
                                                         double* __restrict__ scale, typename P::T* __restrict__ store) {
  using T = typename P::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[2 * P::kC * 33];
  __shared__ typename P::Cf uc[16];  // the packed up list's coefficients by its bits 28 to 31
  using Coefs = RowCoefs<P, kXor>;
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
  T* xs = reinterpret_cast<T*>(smem_raw + ((tab_bytes + 15) & ~size_t(15)));
  const Coefs rc(G);
  const auto ua0 = P::coef(make_double2(S.up_real2[0], 0.0)).x, ua1 = P::coef(make_double2(S.up_real2[1], 0.0)).x;
  if (tid < 16) {
    const double cf = (tid & 8 ? -1.0 : 1.0) * (tid & 4 ? S.up_real2[1] : S.up_real2[0]);
    const bool ph = tid & 2;
    uc[tid] = P::coef(make_double2(ph ? cf * S.up_pc : cf, ph ? cf * (tid & 1 ? -S.up_ps : S.up_ps) : 0.0));
  }
  if (!kPhase && G.ent)
    for (int i = tid; i < G.nt * 8; i += nt) tab[i] = P::coef(G.tab[i >> 3]);
  // padding: zero in every vector
  for (int i = tid; i < Du * 8; i += nt) {
    const int o = (i >> 3) * pitch + Dd + (i & 7);
    wk[o] = y[o] = wkm1[o] = P::zero();
  }
  // start vector: Philox (chain q: key seed + q * 100003) or the caller's, in the gauge basis
  double n0[P::kC];
  typename P::Norm acc0[P::kC];
  for (int i = tid; i < dim; i += nt) {
    const uint32_t r = static_cast<uint32_t>(i) / static_cast<uint32_t>(Dd), c = static_cast<uint32_t>(i) - r * Dd;
    const double g = gauge_sign(S.umask[r], S.dmask[c]) ? -1.0 : 1.0;
    decltype(P::narrow(0.0, 0.0)) z[P::kC];
#pragma unroll
    for (int q = 0; q < P::kC; ++q) {
      const double2 n = init ? init[cd.init + i] : philox_normal(i, cd.seed + static_cast<unsigned>(q) * 100003u);
      z[q] = P::narrow(g * n.x, g * n.y);
      acc0[q].add(static_cast<double>(z[q].x) * z[q].x + static_cast<double>(z[q].y) * z[q].y);
    }
    wk[r * pitch + c] = P::make(z);
  }
#pragma unroll
  for (int q = 0; q < P::kC; ++q) n0[q] = acc0[q].value();
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
  // A warp's item is 32 strings of one row, or 32 / Dd whole rows where they are short.
  const int rpw = Dd <= 16 ? 32 / Dd : 1, ng = (Dd + 31) >> 5;
  const int sub = rpw > 1 ? lane / Dd : 0, pos0 = rpw > 1 ? lane - sub * Dd : lane;
  for (int k = 0; k < M; ++k) {
    if (store) {
      T* out = store + cd.store + static_cast<int64_t>(k) * cd.store_step;
      for (int i = tid; i < dim; i += nt) {
        const uint32_t r = static_cast<uint32_t>(i) / static_cast<uint32_t>(Dd);
        out[i] = wk[i + 8 * r];
      }
    }
    double d[2 * P::kC] = {};
    for (int rb = 0; rb < Du; rb += cd.rows) {  // all rows at once where the whole vector is staged
      const int nr = min(cd.rows, Du - rb);
      if (rb > 0) __syncthreads();
      bool saw = false;
      for (int i = tid; i < nr * pitch; i += nt) {
        T v = wk[rb * pitch + i];
        if constexpr (P::kScaled) {
          v = P::times(s_in[0], v);
          saw = saw || P::small(v);
        }
        xs[i] = P::filtered(v, 1.0);
      }
      // Where an entry is skipped as a source the dot product takes it from the vector itself (complex128; beside the
      // rounding of FP32 vectors it is nothing).
      bool filtered = false;
      if constexpr (P::kScaled)
        filtered = __syncthreads_or(saw);
      else
        __syncthreads();
      const int items = (nr + rpw - 1) / rpw * ng;
      for (int it = warp; it < items; it += nw) {
        const int rl = it / ng * rpw + sub, pos = (it - it / ng * ng) * 32 + pos0;
        const bool in = rl < nr && sub < rpw && pos < Dd;
        const int r = rb + (in ? rl : 0);
        const T* row = xs + (in ? rl : 0) * pitch;
        const int tp = in ? pos : 0, c = !G.ent ? tp : gauge_string(G, tp);
        T acc = P::times(diag_value(S, S.umask[r], S.dmask[c], S.cnt_uu[r], S.cnt_dd[c], S.wpl[r]), row[c]);
        if (G.ent) {
          RowSum<P, 1, kPhase, kXor> s;
          s.base = reinterpret_cast<const unsigned char*>(row);
          s.line = 0;
          s.acc[0] = acc;
          s.walk(G, rpw > 1 ? tp : pos, tab, rc);
          acc = s.acc[0];
        } else {
          acc = list_hops<P>(S, row, c, acc);
        }
        T up = P::zero();
        const T* col = (kSmem ? xs : wk) + tp;
        auto source = [&](int src) {
          const T v = col[src * pitch];
          return kSmem ? v : P::filtered(v, s_in[0]);
        };
        const int j0 = S.up_ptr[r], j1 = S.up_ptr[r + 1];
        if (S.up_pk) {
          auto term = [&](uint32_t e, T v) {
            if (e & 0x20000000u)
              P::cmac(up, uc[e >> 28], v);
            else
              Coefs::mac(up, Coefs::flip((e & 0x40000000u) ? ua1 : ua0, e & 0x80000000u), v);
          };
          int j = j0;
          for (; j + 4 <= j1; j += 4) {
            uint32_t e[4];
            T v[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) e[t] = S.up_pk[j + t];
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = source(e[t] & 0x3FFFu);
#pragma unroll
            for (int t = 0; t < 4; ++t) term(e[t], v[t]);
          }
          for (; j < j1; ++j) term(S.up_pk[j], source(S.up_pk[j] & 0x3FFFu));
        } else {
          int j = j0;
          for (; j + 4 <= j1; j += 4) {
            T v[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = source(S.up_src[j + t]);
#pragma unroll
            for (int t = 0; t < 4; ++t) P::cmac(up, P::up_coef(S, j + t), v[t]);
          }
          for (; j < j1; ++j) P::cmac(up, P::up_coef(S, j), source(S.up_src[j]));
        }
        up = P::shuffle(up, rpw > 1 ? sub * Dd + c : c & 31);
        if (in) {
          const T v = P::add_scaled(acc, up, kSmem ? 1.0 : s_in[0]);
          y[r * pitch + c] = v;
          T left = row[c];
          if constexpr (P::kScaled)
            if (filtered) left = P::times(s_in[0], wk[r * pitch + c]);
          P::dot(d, left, v, 1.0);
        }
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
    double n2[P::kC];
    typename P::Norm acc2[P::kC];
    constexpr int kBatch = P::kC == 1 ? 2 : 1;  // two complex64 chains need the registers
    for (int i0 = tid; i0 < V; i0 += kBatch * nt) {
      T yv[kBatch], av[kBatch], pv[kBatch];
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        const int i = i0 + t * nt < V ? i0 + t * nt : i0;
        yv[t] = y[i];
        av[t] = wk[i];
        pv[t] = k > 0 ? wkm1[i] : P::zero();
      }
#pragma unroll
      for (int t = 0; t < kBatch; ++t) {
        if (i0 + t * nt >= V) continue;
        decltype(P::narrow(0.0, 0.0)) w[P::kC];
#pragma unroll
        for (int q = 0; q < P::kC; ++q) {
          const auto yy = P::get(yv[t], q), aa = P::get(av[t], q), pp = P::get(pv[t], q);
          const double sy = P::kScaled ? 1.0 : s_in[q];
          double wr = sy * static_cast<double>(yy.x) - (c1r[q] * aa.x - c1i[q] * aa.y);
          double wi = sy * static_cast<double>(yy.y) - (c1r[q] * aa.y + c1i[q] * aa.x);
          wr -= c2[q] * pp.x;
          wi -= c2[q] * pp.y;
          w[q] = P::narrow(wr, wi);
          acc2[q].add(static_cast<double>(w[q].x) * w[q].x + static_cast<double>(w[q].y) * w[q].y);
        }
        y[i0 + t * nt] = P::make(w);
      }
    }
#pragma unroll
    for (int q = 0; q < P::kC; ++q) n2[q] = acc2[q].value();
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

// Blocks of up to 256 threads have a kernel of their own with 128 registers a thread, without the spills of 64 (grad 3x2,
// chains 1.46 -> 1.23 ms); with 512 or 768 threads and more registers the large classes are slower (27.9 -> 29.0 ms).
constexpr int kClassThreads[4] = {1024, 512, 256, 64};

}  // namespace

int chain_class(int64_t dim) { return dim > 4096 ? 0 : dim > 1024 ? 1 : dim > 256 ? 2 : 3; }

size_t chain_smem_bytes(const DevSector& S, bool c64, bool phase, int rows) {
  const size_t tab = !S.dn_g.ent || phase ? 0 : static_cast<size_t>(S.dn_g.nt) * 8 * (c64 ? 8 : 16);
  return (tab + 15) / 16 * 16 + static_cast<size_t>(rows) * static_cast<size_t>(S.Dd + 8) * 16;
}

int chain_rows(const DevSector& S, bool c64, bool phase) {
  const size_t most = kMaxSmem - kOwnSmem;
  if (chain_smem_bytes(S, c64, phase, static_cast<int>(S.Du)) <= most) return static_cast<int>(S.Du);
  const size_t base = chain_smem_bytes(S, c64, phase, 0), line = static_cast<size_t>(S.Dd + 8) * 16;
  if (base + line > most) return 0;
  return static_cast<int>(std::max<size_t>(1, base < most / 2 ? (most / 2 - base) / line : 1));
}

namespace {

template <class P>
cudaError_t launch(const ChainLaunch& L, cudaStream_t st) {
  using T = typename P::T;
  using K = void (*)(const DevSector*, const ChainDesc*, int, T*, const double2*, double*, double*, int*, double*, T*);
  static const K kernels[12] = {chains_kernel<P, 1024, false, false, false>, chains_kernel<P, 1024, false, false, true>,
                                chains_kernel<P, 1024, false, true, false>,  chains_kernel<P, 1024, false, true, true>,
                                chains_kernel<P, 1024, true, false, false>,  chains_kernel<P, 1024, true, false, true>,
                                chains_kernel<P, 1024, true, true, false>,   chains_kernel<P, 1024, true, true, true>,
                                chains_kernel<P, 256, true, false, false>,   chains_kernel<P, 256, true, false, true>,
                                chains_kernel<P, 256, true, true, false>,    chains_kernel<P, 256, true, true, true>};
  const int form = (L.phase ? 2 : 0) + (L.xor_real ? 1 : 0);
  const K k = kernels[form + (!L.smem ? 0 : kClassThreads[L.size] > 256 ? 4 : 8)];
  const cudaError_t e = allow_shared(k, L.smem_bytes, kOwnSmem);
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
