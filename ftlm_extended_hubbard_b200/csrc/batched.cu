// Batched FTLM of a momentum block (complex64 vectors, FP64 scalars): its 32 Lanczos chains advance together.  Block
// vectors are V[representative][chain] (32 complex64 = 256 bytes), lane = chain, so that every gather of a
// representative is one coalesced 256-byte segment and the table lookups and signs of a source are shared by the 32
// chains.  The recurrence is that of planes.cu (unnormalised vectors, scalars on the device); a chain whose
// ||w||^2 < 1e-24 stops (reference breakdown rule, src/lanczos.cpp:187) and its later scale factors are 0.  Every
// kernel has a fixed grid (kBtBlocks) and fixed per-block work order: the FP64 reductions are bitwise repeatable.
#include <algorithm>

#include "batched.cuh"
#include "device.cuh"
#include "orbit.cuh"
#include "philox.cuh"

namespace ftlm_b200 {

namespace {

constexpr int kBtThreads = 256;  // 8 warps = 8 basis states per work item
constexpr int kBtWarps = kBtThreads / 32;

// Block-wide per-lane sum of NV doubles over the 8 warps; result valid in warp 0.
template <int NV>
__device__ __forceinline__ void lane_block_sum(double (&v)[NV], double* sh /* NV*kBtThreads */) {
  const int t = threadIdx.x;
#pragma unroll
  for (int i = 0; i < NV; ++i) sh[i * kBtThreads + t] = v[i];
  __syncthreads();
  if (t < 32) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double s = 0.0;
      for (int w = 0; w < kBtWarps; ++w) s += sh[i * kBtThreads + w * 32 + t];
      v[i] = s;
    }
  }
  __syncthreads();
}

// Start vectors: chain r uses Philox4x32-10 with key seed + r*100003 and counter = representative index, the same
// stream as the complex128 path's FTLM_START_PHILOX, rounded to complex64.
__global__ void __launch_bounds__(kBtThreads) bt_start_kernel(float2* __restrict__ W, int64_t dim, unsigned seed,
                                                              double* __restrict__ partial, int* __restrict__ flag) {
  __shared__ double sh[kBtThreads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned key = seed + static_cast<unsigned>(lane) * 100003u;
  Neu acc;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * kBtWarps + warp; i < dim; i += static_cast<int64_t>(gridDim.x) * kBtWarps) {
    const double2 g = philox_normal(i, key);
    const float2 z = make_float2(static_cast<float>(g.x), static_cast<float>(g.y));
    if (tinyf(z) && (z.x != 0.f || z.y != 0.f)) *flag = 1;
    W[i * 32 + lane] = z;
    acc.add(static_cast<double>(z.x) * z.x + static_cast<double>(z.y) * z.y);
  }
  double v[1] = {acc.value()};
  lane_block_sum<1>(v, sh);
  if (threadIdx.x < 32) partial[blockIdx.x * 32 + lane] = v[0];
}

__device__ __forceinline__ float2 filt(float2 v) { return tinyf(v) ? make_float2(0.f, 0.f) : v; }
__device__ __forceinline__ float4 filt4(float4 v) {
  const float2 a = filt(make_float2(v.x, v.y)), b = filt(make_float2(v.z, v.w));
  return make_float4(a.x, a.y, b.x, b.y);
}

// acc (two chains) += (-1)^neg c v with the sign applied to c's sign bits.
__device__ __forceinline__ void cmac4(float4& acc, float2 c, float4 v, uint32_t neg) {
  const uint32_t f = neg << 31;
  c.x = __uint_as_float(__float_as_uint(c.x) ^ f);
  c.y = __uint_as_float(__float_as_uint(c.y) ^ f);
  acc.x = fmaf(c.x, v.x, acc.x);
  acc.x = fmaf(-c.y, v.y, acc.x);
  acc.y = fmaf(c.x, v.y, acc.y);
  acc.y = fmaf(c.y, v.x, acc.y);
  acc.z = fmaf(c.x, v.z, acc.z);
  acc.z = fmaf(-c.y, v.w, acc.z);
  acc.w = fmaf(c.x, v.w, acc.w);
  acc.w = fmaf(c.y, v.z, acc.w);
}

__device__ __forceinline__ float4 fold_halves(float4 a) {
  a.x += __shfl_down_sync(0xffffffffu, a.x, 16);
  a.y += __shfl_down_sync(0xffffffffu, a.y, 16);
  a.z += __shfl_down_sync(0xffffffffu, a.z, 16);
  a.w += __shfl_down_sync(0xffffffffu, a.w, 16);
  return a;
}

// Gathers of the orbit pass: two half-warps take every other source of the warp's list.
template <bool kFilter>
__device__ __forceinline__ float4 bt_cols_sum(const float4* Wc, const uint32_t* s_off, const float2* s_cf, int deg8,
                                              int hv) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = hv; j0 < deg8; j0 += 8) {
    float4 v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = Wc[s_off[j0 + 2 * t]];
#pragma unroll
    for (int t = 0; t < 4; ++t) cmac4(acc, s_cf[j0 + 2 * t], kFilter ? filt4(v[t]) : v[t], 0u);
  }
  return fold_halves(acc);
}

// W_{k+1} = s_in Y - c1 W_k - c2 W_{k-1} (in Y's buffer, FP64 then rounded), ||W_{k+1}||^2 partials per chain.
__global__ void __launch_bounds__(kBtThreads, kBtBlocksPerSm) bt_update_kernel(float2* __restrict__ Y,
                                                                               const float2* __restrict__ Wk,
                                                                               const float2* __restrict__ Wkm1,
                                                                               int64_t dim, const double* __restrict__ st,
                                                                               int use_prev, double* __restrict__ partial,
                                                                               int* __restrict__ flag) {
  __shared__ double sh[kBtThreads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s_in = st[kBtSin * 32 + lane];
  const double c1r = st[kBtC1r * 32 + lane], c1i = st[kBtC1i * 32 + lane];
  const double c2 = use_prev ? st[kBtC2 * 32 + lane] : 0.0;
  Neu acc;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kBtWarps;
  for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * kBtWarps + warp; i0 < dim; i0 += 4 * stride) {
    float2 y[4], a[4], b[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int64_t i = i0 + t * stride;
      const int64_t o = (i < dim ? i : i0) * 32 + lane;
      y[t] = Y[o];
      a[t] = Wk[o];
      b[t] = use_prev ? Wkm1[o] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int64_t i = i0 + t * stride;
      if (i >= dim) continue;
      double wr = s_in * static_cast<double>(y[t].x) - (c1r * a[t].x - c1i * a[t].y);
      double wi = s_in * static_cast<double>(y[t].y) - (c1r * a[t].y + c1i * a[t].x);
      wr -= c2 * b[t].x;
      wi -= c2 * b[t].y;
      const float2 w = make_float2(static_cast<float>(wr), static_cast<float>(wi));
      if (tinyf(w) && (w.x != 0.f || w.y != 0.f)) *flag = 1;
      Y[i * 32 + lane] = w;
      acc.add(static_cast<double>(w.x) * w.x + static_cast<double>(w.y) * w.y);
    }
  }
  double v[1] = {acc.value()};
  lane_block_sum<1>(v, sh);
  if (threadIdx.x < 32) partial[blockIdx.x * 32 + lane] = v[0];
}

// A chain's total of the nblocks partial sums of a step, then its scalars of the recurrence; one block per chain.  The
// kernel is a serial chain of compensated additions, so its time is the number of them in series: with one warp for 32
// chains, all 740 partials in series, it took 88 us, a large part of every step below a million states (4x3 (6,6): 2 x 89
// of 1260 us); 256 threads per chain leave 3 to 10, then a fixed tree (bitwise repeatable): 4.5 us for 2368 partials of 32 chains.
// mode 0: start norms -> s_in = 1/||raw||, c2 = 0.
// mode 1: dot partials -> z = <q_k, H q_k> (s_in^2 <W_k, H W_k> unless scaled), alpha_k, c1 = z * s_in; clears a flag.
// mode 2: norm partials -> beta_k, next s_in = 1/beta_k, c2 = beta_k * s_in (old), breakdown bookkeeping.
constexpr int kScalarThreads = 256;

template <int kVals>
__device__ __forceinline__ void chain_totals(const double* __restrict__ partial, int nblocks, int chain,
                                             double (&tot)[kVals]) {
  __shared__ double sh[kVals][kScalarThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Neu acc[kVals];
#pragma unroll 4
  for (int b = threadIdx.x; b < nblocks; b += kScalarThreads) {
#pragma unroll
    for (int v = 0; v < kVals; ++v) acc[v].add(partial[(b * 32 + chain) * kVals + v]);
  }
#pragma unroll
  for (int v = 0; v < kVals; ++v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double os = __shfl_down_sync(0xffffffffu, acc[v].s, o), oc = __shfl_down_sync(0xffffffffu, acc[v].c, o);
      acc[v].add(os);
      acc[v].c += oc;
    }
    if (lane == 0) sh[v][warp] = acc[v].value();
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < kVals; ++v) {
    Neu t;
    for (int w = 0; w < kScalarThreads / 32; ++w) t.add(sh[v][w]);
    tot[v] = t.value();
  }
}

__global__ void __launch_bounds__(kScalarThreads) bt_scalar_kernel(const double* __restrict__ partial, int nblocks,
                                                                   int mode, int k, double* __restrict__ st,
                                                                   double* __restrict__ alpha, double* __restrict__ beta,
                                                                   int* __restrict__ used, int* __restrict__ clear,
                                                                   int* __restrict__ live, bool scaled) {
  const int chain = blockIdx.x;
  if (mode == 1) {
    double z[2];
    chain_totals<2>(partial, nblocks, chain, z);
    if (threadIdx.x != 0) return;
    if (chain == 0) *clear = 0;
    const double s_in = st[kBtSin * 32 + chain];
    const double f = scaled ? 1.0 : s_in * s_in;
    const double zr = z[0] * f, zi = z[1] * f;
    st[kBtC1r * 32 + chain] = zr * s_in;
    st[kBtC1i * 32 + chain] = zi * s_in;
    if (st[kBtActive * 32 + chain] != 0.0) alpha[k * 32 + chain] = zr;
    return;
  }
  double s[1];
  chain_totals<1>(partial, nblocks, chain, s);
  if (threadIdx.x != 0) return;
  const double n2 = s[0];
  if (mode == 0) {
    const double n0 = sqrt(n2);
    st[kBtSin * 32 + chain] = (n0 < 1e-18) ? 0.0 : 1.0 / n0;
    st[kBtC2 * 32 + chain] = 0.0;
    st[kBtActive * 32 + chain] = (n0 < 1e-18) ? 0.0 : 1.0;
    if (live && !(n0 < 1e-18)) atomicAdd(live, 1);
    used[chain] = 0;
    return;
  }
  const bool active = st[kBtActive * 32 + chain] != 0.0;
  const double s_in = st[kBtSin * 32 + chain];
  if (!active) {
    st[kBtSin * 32 + chain] = 0.0;
    st[kBtC2 * 32 + chain] = 0.0;
    return;
  }
  used[chain] = k + 1;
  if (n2 < 1e-24) {  // breakdown (src/lanczos.cpp:187): alpha_k kept, no beta_k
    st[kBtActive * 32 + chain] = 0.0;
    st[kBtSin * 32 + chain] = 0.0;
    st[kBtC2 * 32 + chain] = 0.0;
    if (live) atomicSub(live, 1);
    return;
  }
  const double b = sqrt(n2);
  beta[k * 32 + chain] = b;
  st[kBtC2 * 32 + chain] = b * s_in;
  st[kBtSin * 32 + chain] = 1.0 / b;
}

// Orbit momentum block, 32 chains: Y[a, :] = H_K W[a, :] (complex64 block vectors over the block's representatives) and
// the fused <W_k, Y> per chain.  Warp per representative: its sources come from the block's list (orbit.cuh), or, where it
// has none, from the sector's gather tables 32 at a time (a random 4-byte lookup per source), the surviving ones compacted
// by ballot; coefficients <rep a|H|s> eta conj(chi(R)) sqrt|A_b| / sqrt|A_a| in FP64, rounded to complex64.  Then the
// half-warps take every other source each and gather the 256-byte rows W[b, :].  Bound by the L1 pipe (71 % of its
// wavefronts) and instruction issue (64 %; 745 warp instructions a representative; rows of 24 instead of 32 chains take as
// long): 4x4 (4,4), 207,000 representatives, 258 us with the table lookups, 215 us with the lists.
constexpr int kOrbTerms = 256;

__device__ __forceinline__ void orb_push(bool ok, uint32_t off, float2 cf, int lane, int& cnt, uint32_t* s_off,
                                         float2* s_cf) {
  const uint32_t m = __ballot_sync(0xffffffffu, ok);
  if (ok) {
    const int pos = cnt + __popc(m & ((1u << lane) - 1u));
    s_off[pos] = off;
    s_cf[pos] = cf;
  }
  cnt += __popc(m);
}

__device__ __forceinline__ float2 orb_coef(const OrbitApplyDev& A, double2 c, uint32_t e, double inv_sa) {
  const double2 ch = A.chi_tab[(e >> 24) & 15u];
  const double f = (((e >> 28) & 1u) ? -1.0 : 1.0) * A.sqrtA[e & 0xFFFFFFu] * inv_sa;
  return make_float2(static_cast<float>(f * (c.x * ch.x + c.y * ch.y)), static_cast<float>(f * (c.y * ch.x - c.x * ch.y)));
}

__global__ void __launch_bounds__(kBtThreads, kBtBlocksPerSm) bt_orbit_kernel(OrbitApplyDev A, const float2* __restrict__ W,
                                                                              float2* __restrict__ Y,
                                                                              const double* __restrict__ st,
                                                                              double* __restrict__ partial,
                                                                              const int* __restrict__ flag) {
  __shared__ uint32_t s_off[kBtWarps][kOrbTerms];
  __shared__ float2 s_cf[kBtWarps][kOrbTerms];
  __shared__ double sh[4 * kBtThreads];
  __shared__ double2 s_dict[256];
  if (A.list) s_dict[threadIdx.x] = A.dict[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hv = lane >> 4, l = lane & 15;
  const bool filter = *flag != 0;
  const DevSector& S = A.S;
  const int64_t Dd = S.Dd;
  const float4* W4 = reinterpret_cast<const float4*>(W);
  float4* Y4 = reinterpret_cast<float4*>(Y);
  uint32_t* off = s_off[warp];
  float2* cfs = s_cf[warp];
  constexpr uint32_t kNone = 0xFFFFFFFFu;
  double d0r = 0.0, d0i = 0.0, d1r = 0.0, d1i = 0.0;
  for (int64_t a = static_cast<int64_t>(blockIdx.x) * kBtWarps + warp; a < A.dk;
       a += static_cast<int64_t>(gridDim.x) * kBtWarps) {
    const uint32_t pk = A.reps[a];
    const uint32_t u = pk >> 16, d = pk & 0xFFFFu;
    const int32_t ru = A.O.rank_u[u], rd = A.O.rank_d[d];
    const double inv_sa = 1.0 / A.sqrtA[a];
    int cnt = 0;
    __syncwarp();
    if (A.list) {
      cnt = A.cnt[a];
      const uint32_t* row = A.list + a * A.pitch;
      for (int j = lane; j < cnt; j += 32) {
        const uint32_t e = row[j];
        const double2 c = s_dict[e >> 24];
        off[j] = (e & 0xFFFFFFu) * 16u;
        cfs[j] = make_float2(static_cast<float>(c.x * inv_sa), static_cast<float>(c.y * inv_sa));
      }
    } else {
      const uint32_t q = prefix_parity_shifted(d);
      const int p1 = S.up_ptr[ru + 1];
      for (int p0 = S.up_ptr[ru]; p0 < p1; p0 += 32) {
        const int p = p0 + lane;
        bool ok = false;
        uint32_t o = 0;
        float2 cf = make_float2(0.f, 0.f);
        if (p < p1) {
          const uint32_t e = __ldg(A.table + static_cast<int64_t>(S.up_src[p]) * Dd + rd);
          if (e != kNone) {
            const uint32_t lh = S.up_lohi[p];
            double2 c = S.up_coef[p];
            if (((q >> (lh & 255u)) ^ (q >> (lh >> 8))) & 1u) c = make_double2(-c.x, -c.y);
            ok = true;
            o = (e & 0xFFFFFFu) * 16u;
            cf = orb_coef(A, c, e, inv_sa);
          }
        }
        orb_push(ok, o, cf, lane, cnt, off, cfs);
      }
      const int64_t rowbase = static_cast<int64_t>(ru) * Dd;
      const int64_t d1 = S.dn_csr_ptr[rd + 1];
      for (int64_t p0 = S.dn_csr_ptr[rd]; p0 < d1; p0 += 32) {
        const int64_t p = p0 + lane;
        bool ok = false;
        uint32_t o = 0;
        float2 cf = make_float2(0.f, 0.f);
        if (p < d1) {
          const uint32_t ent = S.dn_csr_ent[p];
          const int h = static_cast<int>((ent >> 1) & 255u);
          if (h != S.n_dn_hops) {
            const uint32_t e = __ldg(A.table + rowbase + (ent >> 9));
            if (e != kNone) {
              double2 c = S.dn_coef[h];
              if ((ent & 1u) ^ (static_cast<uint32_t>(__popc(u & S.dn_nmask[h])) & 1u)) c = make_double2(-c.x, -c.y);
              ok = true;
              o = (e & 0xFFFFFFu) * 16u;
              cf = orb_coef(A, c, e, inv_sa);
            }
          }
        }
        orb_push(ok, o, cf, lane, cnt, off, cfs);
      }
    }
    const int deg8 = (cnt + 7) & ~7;
    for (int j = cnt + lane; j < deg8; j += 32) {  // padding: a valid row, zero coefficient
      off[j] = static_cast<uint32_t>(a) * 16u;
      cfs[j] = make_float2(0.f, 0.f);
    }
    __syncwarp();
    const float4* Wc = W4 + l;
    const float4 acc = filter ? bt_cols_sum<true>(Wc, off, cfs, deg8, hv) : bt_cols_sum<false>(Wc, off, cfs, deg8, hv);
    if (hv == 0) {
      float4 w = W4[static_cast<uint32_t>(a) * 16u + l];
      const float4 wf = filter ? filt4(w) : w;
      const float dg = static_cast<float>(diag_value(S, u, d, S.cnt_uu[ru], S.cnt_dd[rd], S.wpl[ru]));
      float4 y;
      y.x = acc.x + dg * wf.x;
      y.y = acc.y + dg * wf.y;
      y.z = acc.z + dg * wf.z;
      y.w = acc.w + dg * wf.w;
      Y4[static_cast<uint32_t>(a) * 16u + l] = y;
      const double wx = w.x, wy = w.y, wz = w.z, ww = w.w;
      const double yx = y.x, yy = y.y, yz = y.z, yw = y.w;
      d0r = fma(wx, yx, fma(wy, yy, d0r));
      d0i = fma(wx, yy, fma(-wy, yx, d0i));
      d1r = fma(wz, yz, fma(ww, yw, d1r));
      d1i = fma(wz, yw, fma(-ww, yz, d1i));
    }
  }
  const int t = threadIdx.x;
  sh[0 * kBtThreads + t] = d0r;
  sh[1 * kBtThreads + t] = d0i;
  sh[2 * kBtThreads + t] = d1r;
  sh[3 * kBtThreads + t] = d1i;
  __syncthreads();
  if (t < 32) {
    const int ll = t & 15, which = t >> 4;
    double re = 0.0, im = 0.0;
    for (int w = 0; w < kBtWarps; ++w) {
      re += sh[(2 * which) * kBtThreads + w * 32 + ll];
      im += sh[(2 * which + 1) * kBtThreads + w * 32 + ll];
    }
    const int chain = 2 * ll + which;
    partial[(blockIdx.x * 32 + chain) * 2] = re;
    partial[(blockIdx.x * 32 + chain) * 2 + 1] = im;
  }
}

}  // namespace

void bt_scalars(const double* partial, int nblocks, int mode, int k, int lanes, bool scaled, double* st, double* alpha,
                double* beta, int* used, int* clear, int* live, cudaStream_t s) {
  bt_scalar_kernel<<<lanes, kScalarThreads, 0, s>>>(partial, nblocks, mode, k, st, alpha, beta, used, clear, live, scaled);
}

cudaError_t bt_start(float2* W, int64_t dim, unsigned seed, double* st, double* partial, int* used, int* flags,
                     cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(flags, 0, 2 * sizeof(int), s);
  if (e != cudaSuccess) return e;
  bt_start_kernel<<<kBtBlocks, kBtThreads, 0, s>>>(W, dim, seed, partial, flags);
  bt_scalars(partial, kBtBlocks, 0, 0, 32, false, st, nullptr, nullptr, used, nullptr, nullptr, s);
  return cudaGetLastError();
}

cudaError_t bt_orbit_step(const OrbitApplyDev& A, const float2* Wk, const float2* Wkm1, float2* Y, int k, double* st,
                          double* partial, double* alpha, double* beta, int* used, int* flags, cudaStream_t s) {
  // flags[k % 2]: W_k has a tiny non-zero entry; flags[(k+1) % 2] is cleared for W_{k+1} by the alpha scalars' kernel.
  int* fin = flags + (k & 1);
  int* fout = flags + ((k + 1) & 1);
  bt_orbit_kernel<<<kBtBlocks, kBtThreads, 0, s>>>(A, Wk, Y, st, partial, fin);
  bt_scalars(partial, kBtBlocks, 1, k, 32, false, st, alpha, beta, used, fout, nullptr, s);
  bt_update_kernel<<<kBtBlocks, kBtThreads, 0, s>>>(Y, Wk, Wkm1, A.dk, st, k > 0, partial, fout);
  bt_scalars(partial, kBtBlocks, 2, k, 32, false, st, alpha, beta, used, nullptr, nullptr, s);
  return cudaGetLastError();
}

}  // namespace ftlm_b200
