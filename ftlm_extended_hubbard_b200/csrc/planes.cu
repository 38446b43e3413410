// Lanczos chains of one sector on planes of 16-byte elements; contract in planes.cuh.
//
// A plane is a vector over the sector's states with one 16-byte element per state: two complex64 chains (C64, the
// batched path) or one complex128 chain (C128).  Both passes of H v then have the access pattern of hv.cu: rows staged
// in shared memory whole and contiguous, column slabs of 16-byte elements in L2.  (With the 32 complex64 chains of a
// state side by side instead, 256 bytes a state, a row stage read 16 of every 256 bytes and the column gathers reached
// half the L2 rate: 4x4 (5,6), a step of 32 chains, rows 22.5 and columns 24.6 ms, now 16.8 and 17.3 to 19.4; 4x3 (6,6) 516 and
// 379 us, now 289 and 366.)
// The recurrence, on unnormalised vectors W_k = beta_{k-1} q_k (W_0 = raw start, beta_{-1} = ||raw||):
//       Y = H W_k                              (FP32, unscaled)
//       z = <q_k, H q_k> = <W_k, Y> / beta_{k-1}^2,  alpha_k = Re z
//       W_{k+1} = Y / beta_{k-1} - (z / beta_{k-1}) W_k - (beta_{k-1} / beta_{k-2}) W_{k-1},  beta_k = ||W_{k+1}||
// so no normalisation pass exists and no per-step FP32 rounding of the scale enters alpha.  H v in FP32 (FMA), dot
// products and norms accumulated in FP64, the update evaluated in FP64 and rounded to complex64; fixed grids and
// fixed per-block work order, so the sums are bitwise repeatable.  The vectors live in the spin-ordered (gauge) basis,
// where neither the row nor the column coefficients depend on the other species' string.
#include <algorithm>

#include "batched.cuh"
#include "device.cuh"
#include "launch.cuh"
#include "philox.cuh"
#include "planes.cuh"
#include "planes_dev.cuh"

namespace ftlm_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxDeg = 128;       // up sources of a string
constexpr int kStreamBlocks = 592; // start / update: blocks over all planes (4 per SM of 148, a multiple of 16)
constexpr size_t kMaxSmem = 227 * 1024;

// Whether every chain of the group has ended (live: the count of those that have not; null outside a chain).  The steps
// that are still to come then cost their launches alone: a Hamiltonian with few levels ends all chains early, and the
// host does not wait to learn of it.
__device__ __forceinline__ bool all_ended(const int* live) { return live && *live == 0; }

// Start vectors: given ones (in W already, in the sector's order), or chain c of the group uses Philox4x32-10 with key seed + c*100003 and counter = state index, the
// stream of FTLM_START_PHILOX, rounded to the chains' type and expressed in the gauge basis (W = G r).
template <class P>
__global__ void __launch_bounds__(kThreads) start_kernel(typename P::T* __restrict__ W, int64_t dim, unsigned seed, int nb,
                                                         double* __restrict__ partial, int* __restrict__ flag,
                                                         const uint32_t* __restrict__ umask,
                                                         const uint32_t* __restrict__ dmask, int64_t Dd, bool given) {
  __shared__ double sh[P::kC * kThreads / 32];
  const int plane = blockIdx.x / nb, b = blockIdx.x - plane * nb;
  const unsigned key = seed + static_cast<unsigned>(P::kC * plane) * 100003u;
  typename P::T* out = W + static_cast<int64_t>(plane) * dim;
  Neu acc[P::kC];
  for (int64_t i = static_cast<int64_t>(b) * kThreads + threadIdx.x; i < dim; i += static_cast<int64_t>(nb) * kThreads) {
    const uint32_t r = static_cast<uint32_t>(i) / static_cast<uint32_t>(Dd);
    const double g = gauge_sign(umask[r], dmask[static_cast<uint32_t>(i) - r * static_cast<uint32_t>(Dd)]) ? -1.0 : 1.0;
    decltype(P::narrow(0.0, 0.0)) z[P::kC];
#pragma unroll
    for (int q = 0; q < P::kC; ++q) {
      double2 n;
      if (given) {
        const auto v = P::get(out[i], q);
        n = make_double2(v.x, v.y);
      } else {
        n = philox_normal(i, key + static_cast<unsigned>(q) * 100003u);
      }
      z[q] = P::narrow(g * n.x, g * n.y);
      acc[q].add(static_cast<double>(z[q].x) * z[q].x + static_cast<double>(z[q].y) * z[q].y);
    }
    const typename P::T w = P::make(z);
    if (!P::kScaled && P::small(w)) *flag = 1;
    out[i] = w;
  }
  double v[P::kC];
#pragma unroll
  for (int q = 0; q < P::kC; ++q) v[q] = acc[q].value();
  block_totals<P::kC, kThreads>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < P::kC; ++q) partial[b * 32 + P::kC * plane + q] = v[q];
  }
}

// Warm L2 with bytes that this block reads next (bulk prefetch, no completion to wait on).
__device__ __forceinline__ void prefetch_l2(const void* from, uint32_t bytes) {
  const char* p = static_cast<const char*>(from);
  for (uint32_t off = 0; off < bytes; off += 32768u)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p + off), "r"(min(32768u, bytes - off)) : "memory");
}

// Row pass: one work item is row u of kP planes, staged in shared memory (each plane a line of Dd + 8 elements: the
// gauge table's byte offsets and bank-group schedule address any of them), y = diag o x + down hops.  The table entries
// and coefficients of a string are read once for the kP planes; their order is the table's, so the FP32 sums do not
// depend on kP.  Bound by the shared-memory pipe (a 16-byte load per hop and plane, plus the entries' loads):
// 4x4 (5,5), one plane, 0.57 ms with 87 % of its wavefronts, in either type.
template <class P, int kP, bool kPhase, bool kXor>
__global__ void __launch_bounds__(1024, 1) rows_kernel(DevSector S, const typename P::T* __restrict__ W,
                                                       typename P::T* __restrict__ Y, int planes,
                                                       const double* __restrict__ st, int* __restrict__ flag,
                                                       const int* __restrict__ live) {
  using T = typename P::T;
  const bool ended = all_ended(live);  // tested after the first row's loads, which need not wait for it
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Dd = static_cast<int>(S.Dd), Du = static_cast<int>(S.Du), nt = blockDim.x;
  const uint32_t line = static_cast<uint32_t>(Dd + 8) * 16u;
  T* xs = reinterpret_cast<T*>(smem_raw);
  typename P::Cf* tab = reinterpret_cast<typename P::Cf*>(smem_raw + kP * line);
  const int tid = threadIdx.x;
  const DevGauge G = S.dn_g;
  const RowCoefs<P, kXor> rc(G);
  const bool filter = !P::kScaled && *flag != 0;
  if (!kPhase)
    for (int i = tid; i < G.nt * 8; i += nt) tab[i] = P::coef(G.tab[i >> 3]);
  for (int i = tid; i < 8 * kP; i += nt) xs[(i >> 3) * (Dd + 8) + Dd + (i & 7)] = P::zero();  // padding entries' target
  const int items = Du * ((planes + kP - 1) / kP);
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int p0 = it / Du * kP, r = it - it / Du * Du;
    const int np = min(kP, planes - p0);
    const uint32_t u = S.umask[r];
    const int cuu = S.cnt_uu[r];
    const uint4 wp = S.wpl[r];
    const int64_t base = static_cast<int64_t>(p0) * S.dim + static_cast<int64_t>(r) * Dd;
    if (tid == 0 && it + static_cast<int>(gridDim.x) < items) {  // the next item's rows into L2 while this one is summed
      const int ni = it + gridDim.x, q0 = ni / Du * kP;
      for (int p = 0; p < kP && q0 + p < planes; ++p)
        prefetch_l2(W + static_cast<int64_t>(q0 + p) * S.dim + static_cast<int64_t>(ni % Du) * Dd, static_cast<uint32_t>(Dd) * 16u);
    }
    double sx[kP];
    bool saw = false;
#pragma unroll
    for (int p = 0; p < kP; ++p) sx[p] = P::kScaled && p < np ? (st ? st[kBtSin * 32 + p0 + p] : 1.0) : 1.0;
    for (int c = tid; c < Dd; c += nt) {
#pragma unroll
      for (int p = 0; p < kP; ++p)
        if (p < np) {
          T v = W[base + p * S.dim + c];
          if constexpr (P::kScaled) {
            v = P::times(sx[p], v);
            if (P::small(v)) {
              saw = true;
              v = P::zero();
            }
          } else if (filter) {
            v = P::filtered(v, 1.0);
          }
          xs[p * (Dd + 8) + c] = v;
        }
    }
    if (P::kScaled && saw) *flag = 1;
    __syncthreads();
    if (ended) return;
    for (int c = tid; c < Dd; c += nt) {
      const int d = gauge_string(G, c);  // table position c serves output string d
      const double dg = diag_value(S, u, S.dmask[d], cuu, S.cnt_dd[d], wp);
      RowSum<P, kP, kPhase, kXor> s;
      s.line = line;
      s.base = smem_raw;
#pragma unroll
      for (int p = 0; p < kP; ++p) s.acc[p] = P::times(dg, xs[p * (Dd + 8) + d]);
      s.walk(G, c, tab, rc);
#pragma unroll
      for (int p = 0; p < kP; ++p)
        if (p < np) Y[base + p * S.dim + d] = s.acc[p];
    }
    __syncthreads();
  }
}

// Row pass of sectors without the gauge table, or whose row does not fit shared memory: gathers from the row in L2,
// thread per state and plane.  Even and odd entries of a string's list in a sum each, added at the end.
template <class P>
__global__ void __launch_bounds__(kThreads) rows_gather_kernel(DevSector S, const typename P::T* __restrict__ W,
                                                               typename P::T* __restrict__ Y, int planes,
                                                               const int* __restrict__ flag,
                                                               const int* __restrict__ live) {
  static_assert(!P::kScaled, "complex128 chains without the gauge table run on the H v kernels of hv.cu");
  using T = typename P::T;
  if (all_ended(live)) return;
  const bool filter = *flag != 0;
  const int64_t total = S.dim * planes;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * kThreads) {
    const int64_t row = i / S.Dd;  // over all planes
    const int c = static_cast<int>(i - row * S.Dd), r = static_cast<int>(row % S.Du);
    const T* x = W + row * S.Dd;
    auto in = [&](uint32_t e) { return filter ? P::filtered(x[e], 1.0) : x[e]; };
    T a = P::times(diag_value(S, S.umask[r], S.dmask[c], S.cnt_uu[r], S.cnt_dd[c], S.wpl[r]), in(c)), b = P::zero();
    const int64_t e1 = S.dn_csr_ptr[c + 1];  // lists padded to a multiple of 8
    for (int64_t e = S.dn_csr_ptr[c]; e < e1; e += 4) {
      uint32_t q[4];
      T v[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) q[t] = S.dn_csr_ent[e + t];
#pragma unroll
      for (int t = 0; t < 4; ++t) v[t] = in(q[t] >> 9);
#pragma unroll
      for (int t = 0; t < 4; ++t) P::cmac((t & 1) ? b : a, P::dn_coef(S, q[t]), v[t]);
    }
    Y[i] = P::plus(a, b);
  }
}

// Column pass: y[r, c] += sum_j u_j x[src_j, c], and the two chains' <W, Y>.  Work item = (plane, chunk of 2 kT
// columns, output row), plane- then chunk-major over a persistent grid, so that the slab of the chunk (Du x 2 kT x 16
// bytes) stays in L2 while all rows read it; a thread has two columns, kT apart, and four sources of each in flight.
// The source list of the next item is fetched while this one is summed.  Bound by the gathers, which load both the L1
// pipe and L2 (4x4 (5,5) by items: 0.55 ms, 81 % of the wavefronts, 71 % of L2; complex64 0.53 ms, 82 and 75 %).
template <class P, bool kFilter>
__device__ __forceinline__ void cols_sum(const typename P::T* __restrict__ x0, const typename P::T* __restrict__ x1,
                                         const uint32_t* s_off, const typename P::Cf* s_cf, int deg, double sx,
                                         typename P::T& a0, typename P::T& a1) {
  using T = typename P::T;
  a0 = a1 = P::zero();
  int j = 0;
  for (; j + 4 <= deg; j += 4) {
    T v0[4], v1[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      v0[t] = x0[s_off[j + t]];
      v1[t] = x1[s_off[j + t]];
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const typename P::Cf c = s_cf[j + t];
      P::cmac(a0, c, kFilter ? P::filtered(v0[t], sx) : v0[t]);
      P::cmac(a1, c, kFilter ? P::filtered(v1[t], sx) : v1[t]);
    }
  }
  for (; j < deg; ++j) {
    const T v0 = x0[s_off[j]], v1 = x1[s_off[j]];
    const typename P::Cf c = s_cf[j];
    P::cmac(a0, c, kFilter ? P::filtered(v0, sx) : v0);
    P::cmac(a1, c, kFilter ? P::filtered(v1, sx) : v1);
  }
}

template <class P, int kT, bool kDot>
__global__ void __launch_bounds__(kT, P::kColThreads / kT) cols_kernel(DevSector S, const typename P::T* __restrict__ W,
                                                             typename P::T* __restrict__ Y, int planes,
                                                             const double* __restrict__ st, double* __restrict__ partial,
                                                             const int* __restrict__ flag, const int* __restrict__ live) {
  using T = typename P::T;
  constexpr int kPer = (kMaxDeg + kT - 1) / kT;  // list entries per thread
  __shared__ uint32_t s_off[2][kMaxDeg];
  __shared__ __align__(16) typename P::Cf s_cf[2][kMaxDeg];
  __shared__ double sh[2 * P::kC * kT / 32];
  const int t = threadIdx.x;
  const bool filter = *flag != 0, ended = all_ended(live);
  const uint32_t Dd = static_cast<uint32_t>(S.Dd), Du = static_cast<uint32_t>(S.Du);
  const uint32_t per = (Dd + 2 * kT - 1) / (2 * kT) * Du, total = per * static_cast<uint32_t>(planes);
  uint32_t off[kPer];
  typename P::Cf cf[kPer];
  auto fetch = [&](uint32_t it) {  // the source list of an item into registers; returns its length
    const uint32_t r = it % Du;    // per is a multiple of Du
    const int j0 = S.up_ptr[r], deg = S.up_ptr[r + 1] - j0;
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (t + q * kT < deg) {
        off[q] = static_cast<uint32_t>(S.up_src[j0 + t + q * kT]) * Dd;
        cf[q] = P::up_coef(S, j0 + t + q * kT);
      }
    return deg;
  };
  auto place = [&](int buf, int deg) {
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (t + q * kT < deg) {
        s_off[buf][t + q * kT] = off[q];
        s_cf[buf][t + q * kT] = cf[q];
      }
  };
  uint32_t it = blockIdx.x;
  int buf = 0, deg = 0;
  if (it < total) {
    deg = fetch(it);
    place(0, deg);
  }
  __syncthreads();
  if (ended) return;
  for (int p = 0; p < planes; ++p) {
    double d[2 * P::kC] = {};
    const uint32_t end = per * static_cast<uint32_t>(p + 1);
    const T* Wp = W + static_cast<int64_t>(p) * S.dim;
    T* Yp = Y + static_cast<int64_t>(p) * S.dim;
    const double sx = P::kScaled && st ? st[kBtSin * 32 + p] : 1.0;
    for (; it < end; it += gridDim.x) {
      const uint32_t next = it + gridDim.x;
      const int ndeg = next < total ? fetch(next) : 0;
      const uint32_t q = it - (end - per), chunk = q / Du, r = q - chunk * Du;
      const uint32_t c0 = chunk * (2 * kT) + t, c1 = c0 + kT;
      if (c0 < Dd) {
        const bool has1 = c1 < Dd;
        const uint32_t c1s = has1 ? c1 : c0;
        T a0, a1;
        if (filter)
          cols_sum<P, true>(Wp + c0, Wp + c1s, s_off[buf], s_cf[buf], deg, sx, a0, a1);
        else
          cols_sum<P, false>(Wp + c0, Wp + c1s, s_off[buf], s_cf[buf], deg, sx, a0, a1);
        const uint32_t o0 = r * Dd + c0, o1 = r * Dd + c1s;
        const T y0 = P::add_scaled(Yp[o0], a0, sx);
        if (kDot) P::dot(d, Wp[o0], y0, sx);
        Yp[o0] = y0;
        if (has1) {
          const T y1 = P::add_scaled(Yp[o1], a1, sx);
          if (kDot) P::dot(d, Wp[o1], y1, sx);
          Yp[o1] = y1;
        }
      }
      buf ^= 1;
      place(buf, ndeg);
      deg = ndeg;
      __syncthreads();
    }
    if (kDot) {
      block_totals<2 * P::kC, kT>(d, sh);
      if (t == 0) {
#pragma unroll
        for (int v = 0; v < 2 * P::kC; ++v) partial[(static_cast<int64_t>(blockIdx.x) * 32 + P::kC * p) * 2 + v] = d[v];
      }
    }
  }
}

// The same, one block per item and one partial per item (items [plane][item][2 kC]): the hardware hands the items out in
// order, so that all blocks stay within a chunk or two of each other and the slab stays in L2, where blocks of the
// persistent grid drift apart over the hundreds of items that a large plane gives each of them.
template <class P, int kT, bool kDot>
__global__ void __launch_bounds__(kT, P::kColThreads / kT) cols_items_kernel(DevSector S, const typename P::T* __restrict__ W,
                                                                             typename P::T* __restrict__ Y, uint32_t per,
                                                                             const double* __restrict__ st,
                                                                             double* __restrict__ items,
                                                                             const int* __restrict__ flag,
                                                                             const int* __restrict__ live) {
  using T = typename P::T;
  __shared__ uint32_t s_off[kMaxDeg];
  __shared__ __align__(16) typename P::Cf s_cf[kMaxDeg];
  __shared__ double sh[2 * P::kC * kT / 32];
  const int t = threadIdx.x;
  const bool filter = *flag != 0, ended = all_ended(live);  // tested late: the list loads need not wait for it
  const uint32_t Dd = static_cast<uint32_t>(S.Dd), Du = static_cast<uint32_t>(S.Du);
  const uint32_t p = blockIdx.x / per, it = blockIdx.x - p * per, chunk = it / Du, r = it - chunk * Du;
  const int j0 = S.up_ptr[r], deg = S.up_ptr[r + 1] - j0;
  for (int j = t; j < deg; j += kT) {
    s_off[j] = static_cast<uint32_t>(S.up_src[j0 + j]) * Dd;
    s_cf[j] = P::up_coef(S, j0 + j);
  }
  const T* Wp = W + static_cast<int64_t>(p) * S.dim;
  T* Yp = Y + static_cast<int64_t>(p) * S.dim;
  const double sx = P::kScaled && st ? st[kBtSin * 32 + p] : 1.0;
  const uint32_t c0 = chunk * (2 * kT) + t, c1 = c0 + kT;
  double d[2 * P::kC] = {};
  __syncthreads();
  if (c0 < Dd && !ended) {
    const bool has1 = c1 < Dd;
    const uint32_t c1s = has1 ? c1 : c0;
    T a0, a1;
    if (filter)
      cols_sum<P, true>(Wp + c0, Wp + c1s, s_off, s_cf, deg, sx, a0, a1);
    else
      cols_sum<P, false>(Wp + c0, Wp + c1s, s_off, s_cf, deg, sx, a0, a1);
    const uint32_t o0 = r * Dd + c0, o1 = r * Dd + c1s;
    const T y0 = P::add_scaled(Yp[o0], a0, sx);
    if (kDot) P::dot(d, Wp[o0], y0, sx);
    Yp[o0] = y0;
    if (has1) {
      const T y1 = P::add_scaled(Yp[o1], a1, sx);
      if (kDot) P::dot(d, Wp[o1], y1, sx);
      Yp[o1] = y1;
    }
  }
  if (kDot) {
    block_totals<2 * P::kC, kT>(d, sh);
    if (t == 0) {
#pragma unroll
      for (int v = 0; v < 2 * P::kC; ++v) items[static_cast<int64_t>(blockIdx.x) * (2 * P::kC) + v] = d[v];
    }
  }
}

// First level of the items' sums: block (plane, b) of nb adds its share of the plane's items into partial slot b.
template <int kC>
__global__ void __launch_bounds__(kThreads) fold_kernel(const double* __restrict__ items, uint32_t per, int nb,
                                                        double* __restrict__ partial) {
  __shared__ double sh[2 * kC * kThreads / 32];
  const int plane = blockIdx.x / nb, b = blockIdx.x - plane * nb;
  const uint32_t share = (per + nb - 1) / nb, i0 = b * share, i1 = min(per, i0 + share);
  const double* in = items + static_cast<int64_t>(plane) * per * (2 * kC);
  double d[2 * kC] = {};
  for (uint32_t i = i0 + threadIdx.x; i < i1; i += kThreads) {
#pragma unroll
    for (int v = 0; v < 2 * kC; ++v) d[v] += in[static_cast<int64_t>(i) * (2 * kC) + v];
  }
  block_totals<2 * kC, kThreads>(d, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int v = 0; v < 2 * kC; ++v) partial[(static_cast<int64_t>(b) * 32 + kC * plane) * 2 + v] = d[v];
  }
}

// W_{k+1} = s_in Y - c1 W_k - c2 W_{k-1} (in Y's buffer, FP64 then rounded), ||W_{k+1}||^2 partials per chain.  Streams
// three vectors in and one out.
template <class P>
__global__ void __launch_bounds__(kThreads, 4) update_kernel(typename P::T* __restrict__ Y,
                                                             const typename P::T* __restrict__ Wk,
                                                             const typename P::T* __restrict__ Wkm1, int64_t dim, int nb,
                                                             const double* __restrict__ st, int use_prev,
                                                             double* __restrict__ partial, int* __restrict__ flag,
                                                             const int* __restrict__ live) {
  using T = typename P::T;
  const bool ended = all_ended(live);
  __shared__ double sh[P::kC * kThreads / 32];
  const int plane = blockIdx.x / nb, b = blockIdx.x - plane * nb;
  double s_in[P::kC], c1r[P::kC], c1i[P::kC], c2[P::kC];
#pragma unroll
  for (int q = 0; q < P::kC; ++q) {
    const int ch = P::kC * plane + q;
    s_in[q] = P::kScaled ? 1.0 : st[kBtSin * 32 + ch];
    c1r[q] = st[kBtC1r * 32 + ch];
    c1i[q] = st[kBtC1i * 32 + ch];
    c2[q] = use_prev ? st[kBtC2 * 32 + ch] : 0.0;
  }
  if (ended) return;
  Neu acc[P::kC];
  const int64_t base = static_cast<int64_t>(plane) * dim, stride = static_cast<int64_t>(nb) * kThreads;
  for (int64_t i0 = static_cast<int64_t>(b) * kThreads + threadIdx.x; i0 < dim; i0 += 2 * stride) {
    T y[2], a[2], p[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int64_t o = base + (i0 + t * stride < dim ? i0 + t * stride : i0);
      y[t] = Y[o];
      a[t] = Wk[o];
      p[t] = use_prev ? Wkm1[o] : P::zero();
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (i0 + t * stride >= dim) continue;
      decltype(P::narrow(0.0, 0.0)) w[P::kC];
#pragma unroll
      for (int q = 0; q < P::kC; ++q) {
        const auto yy = P::get(y[t], q), aa = P::get(a[t], q), pp = P::get(p[t], q);
        double wr = s_in[q] * static_cast<double>(yy.x) - (c1r[q] * aa.x - c1i[q] * aa.y);
        double wi = s_in[q] * static_cast<double>(yy.y) - (c1r[q] * aa.y + c1i[q] * aa.x);
        wr -= c2[q] * pp.x;
        wi -= c2[q] * pp.y;
        w[q] = P::narrow(wr, wi);
        acc[q].add(static_cast<double>(w[q].x) * w[q].x + static_cast<double>(w[q].y) * w[q].y);
      }
      const T v = P::make(w);
      if (!P::kScaled && P::small(v)) *flag = 1;
      Y[base + i0 + t * stride] = v;
    }
  }
  double v[P::kC];
#pragma unroll
  for (int q = 0; q < P::kC; ++q) v[q] = acc[q].value();
  block_totals<P::kC, kThreads>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < P::kC; ++q) partial[b * 32 + P::kC * plane + q] = v[q];
  }
}

int sm_count() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

// Lines that the row pass can stage: 2, 1, or 0 (no gauge table, or a row does not fit).
template <class P>
int row_planes(const DevSector& S) {
  const size_t line = static_cast<size_t>(S.Dd + 8) * 16;
  const size_t tab = S.dn_g.phase ? 0 : static_cast<size_t>(S.dn_g.nt) * 8 * sizeof(typename P::Cf);
  return !S.dn_g.ent || line + tab > kMaxSmem ? 0 : 2 * line + tab <= kMaxSmem ? 2 : 1;
}

// Planes per item and threads of the row pass: two planes where two lines fit, so that the entries are read once for
// both; blocks no wider than a row, several on an SM, so that one block's staging overlaps another's hops (a single
// 1024-thread block leaves the SM idle while it stages, and most of its threads where a row is short).
template <class P, int kP, bool kPhase, bool kXor>
cudaError_t launch_rows_p(const DevSector& S, const typename P::T* W, typename P::T* Y, int planes, const double* st,
                          int* flag, const int* live, cudaStream_t s) {
  const auto k = rows_kernel<P, kP, kPhase, kXor>;
  const size_t sm = static_cast<size_t>(kP) * (S.Dd + 8) * 16 + (kPhase ? 0 : S.dn_g.nt * 8 * sizeof(typename P::Cf));
  const cudaError_t e = allow_shared(k, sm);
  if (e != cudaSuccess) return e;
  const int per_smem = std::max<int>(1, static_cast<int>((kMaxSmem + 1024) / (sm + 1024)));
  int threads = 1024;
  while (threads > 64 && (threads / 2 >= S.Dd || (threads > 256 && threads / 2 * per_smem >= 1024))) threads /= 2;
  const int per_sm = std::max(1, std::min(per_smem, 1024 / threads));
  const int64_t items = S.Du * ((planes + kP - 1) / kP);
  const int grid = static_cast<int>(std::min<int64_t>(items, static_cast<int64_t>(sm_count()) * per_sm));
  k<<<grid, threads, sm, s>>>(S, W, Y, planes, st, flag, live);
  return cudaGetLastError();
}

template <class P, int kP>
cudaError_t launch_rows_n(const DevSector& S, const typename P::T* W, typename P::T* Y, int planes, const double* st,
                          int* flag, const int* live, cudaStream_t s) {
  if (S.dn_g.phase)
    return S.dn_g.xor_real ? launch_rows_p<P, kP, true, true>(S, W, Y, planes, st, flag, live, s)
                           : launch_rows_p<P, kP, true, false>(S, W, Y, planes, st, flag, live, s);
  return S.dn_g.xor_real ? launch_rows_p<P, kP, false, true>(S, W, Y, planes, st, flag, live, s)
                         : launch_rows_p<P, kP, false, false>(S, W, Y, planes, st, flag, live, s);
}

template <class P>
cudaError_t launch_rows(const DevSector& S, const typename P::T* W, typename P::T* Y, int planes, const double* st,
                        int* flag, const int* live, cudaStream_t s) {
  const int rp = row_planes<P>(S);
  if (rp == 2 && planes > 1) return launch_rows_n<P, 2>(S, W, Y, planes, st, flag, live, s);
  if (rp > 0) return launch_rows_n<P, 1>(S, W, Y, planes, st, flag, live, s);
  if constexpr (P::kScaled) {
    return cudaErrorNotSupported;  // pl_fits
  } else {
    const int64_t blocks = std::min<int64_t>((S.dim * planes + kThreads - 1) / kThreads, static_cast<int64_t>(sm_count()) * 16);
    rows_gather_kernel<P><<<static_cast<unsigned>(blocks), kThreads, 0, s>>>(S, W, Y, planes, flag, live);
    return cudaGetLastError();
  }
}

template <class P, int kT>
int launch_cols_t(const DevSector& S, const typename P::T* W, typename P::T* Y, int planes, const double* st,
                  double* partial, double* items, const int* flag, const int* live, cudaStream_t s) {
  const int64_t per = (S.Dd + 2 * kT - 1) / (2 * kT) * S.Du;
  const int64_t grid = std::min<int64_t>({per * planes, static_cast<int64_t>(sm_count()) * (P::kColThreads / kT), kPlMaxBlocks});
  // From 8 items of a plane for each block of the persistent grid, one block per item: 4x4 (6,6) complex128 2.19 -> 1.86 ms,
  // 4x4 (5,6) complex64 1.09 -> 0.97 ms a plane; below, the persistent grid's prefetched lists: 4x3 (4,5) 40 us, 44 by items.
  if (per >= 8 * grid) {
    const unsigned n = static_cast<unsigned>(per * planes);
    if (!partial) {
      cols_items_kernel<P, kT, false><<<n, kT, 0, s>>>(S, W, Y, static_cast<uint32_t>(per), st, nullptr, flag, live);
      return 0;
    }
    cols_items_kernel<P, kT, true><<<n, kT, 0, s>>>(S, W, Y, static_cast<uint32_t>(per), st, items, flag, live);
    const int nb = std::max(1, kStreamBlocks / planes);
    fold_kernel<P::kC><<<nb * planes, kThreads, 0, s>>>(items, static_cast<uint32_t>(per), nb, partial);
    return nb;
  }
  if (partial)
    cols_kernel<P, kT, true><<<static_cast<unsigned>(grid), kT, 0, s>>>(S, W, Y, planes, st, partial, flag, live);
  else
    cols_kernel<P, kT, false><<<static_cast<unsigned>(grid), kT, 0, s>>>(S, W, Y, planes, st, partial, flag, live);
  return static_cast<int>(grid);
}

// Returns the grid: the number of partials per chain.
template <class P>
int launch_cols(const DevSector& S, const typename P::T* W, typename P::T* Y, int planes, const double* st,
                double* partial, double* items, const int* flag, const int* live, cudaStream_t s) {
  if (S.bt_cols == 1) return launch_cols_t<P, 64>(S, W, Y, planes, st, partial, items, flag, live, s);
  if (S.bt_cols == 2) return launch_cols_t<P, 256>(S, W, Y, planes, st, partial, items, flag, live, s);
  return launch_cols_t<P, 128>(S, W, Y, planes, st, partial, items, flag, live, s);
}

template <class P>
cudaError_t start(const DevSector& S, typename P::T* W, int planes, unsigned seed, bool given, const PlaneState& z,
                  cudaStream_t s) {
  const cudaError_t e = cudaMemsetAsync(z.flags, 0, kPlFlags * sizeof(int), s);
  if (e != cudaSuccess) return e;
  const int nb = std::max(1, kStreamBlocks / planes);
  start_kernel<P><<<nb * planes, kThreads, 0, s>>>(W, S.dim, seed, nb, z.partial, z.flags, S.umask, S.dmask, S.Dd, given);
  bt_scalars(z.partial, nb, 0, 0, P::kC * planes, P::kScaled, z.st, nullptr, nullptr, z.used, nullptr, z.flags + 2, s);
  return cudaGetLastError();
}

// The row and column passes number their work items in 32 bits.
bool items_fit(const DevSector& S, int planes) {
  const int64_t kT = S.bt_cols == 1 ? 64 : S.bt_cols == 2 ? 256 : 128;
  return (S.Dd + 2 * kT - 1) / (2 * kT) * S.Du <= (INT32_MAX - 65536) / std::max(1, planes);
}

template <class P>
cudaError_t step(const DevSector& S, const typename P::T* Wk, const typename P::T* Wkm1, typename P::T* Y, int planes,
                 int k, const PlaneState& z, cudaStream_t s) {
  // flags[2]: the live chains.  C64: flags[k % 2]: W_k has a tiny non-zero entry, written with W_k; flags[(k+1) % 2] is cleared for W_{k+1} by the
  // alpha scalars' kernel.  C128: flags[0], written by the row pass and cleared by that kernel.
  int* fin = z.flags + (P::kScaled ? 0 : (k & 1));
  int* fout = z.flags + (P::kScaled ? 0 : ((k + 1) & 1));
  if (!items_fit(S, planes)) return cudaErrorInvalidValue;
  // Below this a step is its launches, with work or without, and the reads of the count cost it 0.65 of 24 us (3x3 (4,4)).
  constexpr int64_t kCounted = int64_t(1) << 18;
  int* live = S.dim * planes >= kCounted ? z.flags + 2 : nullptr;
  const cudaError_t e = launch_rows<P>(S, Wk, Y, planes, z.st, fin, live, s);
  if (e != cudaSuccess) return e;
  const int nc = launch_cols<P>(S, Wk, Y, planes, z.st, z.partial, z.items, fin, live, s);
  bt_scalars(z.partial, nc, 1, k, P::kC * planes, P::kScaled, z.st, z.alpha, z.beta, z.used, fout, nullptr, s);
  const int nb = std::max(1, kStreamBlocks / planes);
  update_kernel<P><<<nb * planes, kThreads, 0, s>>>(Y, Wk, Wkm1, S.dim, nb, z.st, k > 0, z.partial, fout, live);
  bt_scalars(z.partial, nb, 2, k, P::kC * planes, P::kScaled, z.st, z.alpha, z.beta, z.used, nullptr, live, s);
  return cudaGetLastError();
}

template <class P>
cudaError_t apply(const DevSector& S, const typename P::T* X, typename P::T* Y, int planes, int* flag, cudaStream_t s) {
  if (!items_fit(S, planes)) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
  if (e == cudaSuccess) e = launch_rows<P>(S, X, Y, planes, nullptr, flag, nullptr, s);
  if (e != cudaSuccess) return e;
  launch_cols<P>(S, X, Y, planes, nullptr, nullptr, nullptr, flag, nullptr, s);
  return cudaGetLastError();
}

}  // namespace

int pl_group(const DevSector& S, bool c64, int planes) {
  constexpr int64_t kEnough = int64_t(256) << 20;
  const int64_t bytes = 16 * std::max<int64_t>(S.dim, 1);
  const int64_t least = (c64 ? row_planes<C64>(S) : row_planes<C128>(S));
  return static_cast<int>(std::min<int64_t>(planes, std::max<int64_t>(least, (kEnough + bytes - 1) / bytes)));
}

int64_t pl_items_doubles(const DevSector& S, bool c64, int planes) {
  const int kT = S.bt_cols == 1 ? 64 : S.bt_cols == 2 ? 256 : 128;
  const int64_t per = (S.Dd + 2 * kT - 1) / (2 * kT) * S.Du;
  return per * planes * (c64 ? 4 : 2);
}

bool pl_fits(const DevSector& S, int max_up_deg) { return row_planes<C128>(S) > 0 && max_up_deg <= kMaxDeg; }

cudaError_t pl_start(const DevSector& S, float4* W, int planes, unsigned seed, const PlaneState& z, cudaStream_t s) {
  return start<C64>(S, W, planes, seed, false, z, s);
}

cudaError_t pl_start(const DevSector& S, double2* W, int planes, unsigned seed, bool given, const PlaneState& z,
                     cudaStream_t s) {
  return start<C128>(S, W, planes, seed, given, z, s);
}

cudaError_t pl_step(const DevSector& S, const float4* Wk, const float4* Wkm1, float4* Y, int planes, int k,
                    const PlaneState& z, cudaStream_t s) {
  return step<C64>(S, Wk, Wkm1, Y, planes, k, z, s);
}

cudaError_t pl_step(const DevSector& S, const double2* Wk, const double2* Wkm1, double2* Y, int planes, int k,
                    const PlaneState& z, cudaStream_t s) {
  return step<C128>(S, Wk, Wkm1, Y, planes, k, z, s);
}

cudaError_t pl_apply(const DevSector& S, const float4* X, float4* Y, int planes, int* flag, cudaStream_t s) {
  return apply<C64>(S, X, Y, planes, flag, s);
}

cudaError_t pl_apply(const DevSector& S, const double2* X, double2* Y, int planes, int* flag, cudaStream_t s) {
  return apply<C128>(S, X, Y, planes, flag, s);
}

}  // namespace ftlm_b200
