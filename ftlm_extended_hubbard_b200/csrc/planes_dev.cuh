// Element types and the row sum of the Lanczos chains in the spin-ordered basis, shared by planes.cu and chains.cu.
#pragma once

#include "batched.cuh"
#include "device.cuh"

namespace ftlm_b200 {

// The element types.  C64: two chains in FP32; Y = H W stays unscaled and 1/beta_{k-1} is applied in FP64 by the
// update; an entry with |W|^2 < 1e-28 is skipped as a source.  C128: one chain; the row pass stages s W (s =
// 1/beta_{k-1}), so Y = H q, and an entry with |s W|^2 < 1e-28 is skipped, as the reference does with q.
struct C64 {
  using T = float4;
  using Cf = float2;
  using Norm = Neu;  // a thread's share of a squared norm: compensated, as in every complex64 chain
  static constexpr int kC = 2;
  static constexpr bool kScaled = false;
  static constexpr int kColThreads = 1024;  // resident threads per SM of the column pass (registers)
  static __device__ __forceinline__ T zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
  static __device__ __forceinline__ bool small(T v) {  // a non-zero entry that is skipped as a source
    return (tinyf(make_float2(v.x, v.y)) && (v.x != 0.f || v.y != 0.f)) ||
           (tinyf(make_float2(v.z, v.w)) && (v.z != 0.f || v.w != 0.f));
  }
  static __device__ __forceinline__ T filtered(T v, double) {
    if (tinyf(make_float2(v.x, v.y))) v.x = v.y = 0.f;
    if (tinyf(make_float2(v.z, v.w))) v.z = v.w = 0.f;
    return v;
  }
  static __device__ __forceinline__ T times(double g, T v) {
    const float f = static_cast<float>(g);
    return make_float4(f * v.x, f * v.y, f * v.z, f * v.w);
  }
  static __device__ __forceinline__ T add_scaled(T y, T a, double) { return plus(y, a); }  // y + s a, s = 1
  static __device__ __forceinline__ T plus(T a, T b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
  static __device__ __forceinline__ Cf coef(double2 c) { return make_float2(__double2float_rn(c.x), __double2float_rn(c.y)); }
  static __device__ __forceinline__ Cf signed_coef(Cf c, uint32_t e) {
    const uint32_t f = e & 0x80000000u;
    return make_float2(__uint_as_float(__float_as_uint(c.x) ^ f), __uint_as_float(__float_as_uint(c.y) ^ f));
  }
  static __device__ __forceinline__ void cmac(T& acc, Cf c, T v) {
    acc.x = fmaf(c.x, v.x, acc.x);
    acc.x = fmaf(-c.y, v.y, acc.x);
    acc.y = fmaf(c.x, v.y, acc.y);
    acc.y = fmaf(c.y, v.x, acc.y);
    acc.z = fmaf(c.x, v.z, acc.z);
    acc.z = fmaf(-c.y, v.w, acc.z);
    acc.w = fmaf(c.x, v.w, acc.w);
    acc.w = fmaf(c.y, v.z, acc.w);
  }
  static __device__ __forceinline__ T shuffle(T v, int lane) {
    return make_float4(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane),
                       __shfl_sync(0xffffffffu, v.z, lane), __shfl_sync(0xffffffffu, v.w, lane));
  }
  // conj(w) y of the chains, (re, im) each
  static __device__ __forceinline__ void dot(double (&d)[4], T w, T y, double) {
    const double wx = w.x, wy = w.y, wz = w.z, ww = w.w;
    const double yx = y.x, yy = y.y, yz = y.z, yw = y.w;
    d[0] = fma(wx, yx, fma(wy, yy, d[0]));
    d[1] = fma(wx, yy, fma(-wy, yx, d[1]));
    d[2] = fma(wz, yz, fma(ww, yw, d[2]));
    d[3] = fma(wz, yw, fma(-ww, yz, d[3]));
  }
  static __device__ __forceinline__ Cf up_coef(const DevSector& S, int j) { return S.up_coef32[j]; }
  static __device__ __forceinline__ Cf dn_coef(const DevSector& S, uint32_t e) { return __ldg(S.dn_coef32s + (e & 511u)); }
  static __device__ __forceinline__ float2 get(T v, int q) { return q == 0 ? make_float2(v.x, v.y) : make_float2(v.z, v.w); }
  static __device__ __forceinline__ T make(const float2 (&z)[2]) { return make_float4(z[0].x, z[0].y, z[1].x, z[1].y); }
  static __device__ __forceinline__ float2 narrow(double re, double im) {
    return make_float2(static_cast<float>(re), static_cast<float>(im));
  }
};

struct Plain {
  double s = 0.0;
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ double value() const { return s; }
};

struct C128 {
  using T = double2;
  using Cf = double2;
  using Norm = Plain;
  static constexpr int kC = 1;
  static constexpr bool kScaled = true;
  static constexpr int kColThreads = 896;  // 4x4 (6,6): 2.19 ms, 2.33 with 1024
  static __device__ __forceinline__ T zero() { return make_double2(0.0, 0.0); }
  static __device__ __forceinline__ bool small(T v) { return tiny(v) && (v.x != 0.0 || v.y != 0.0); }
  static __device__ __forceinline__ T filtered(T v, double s) { return tiny(make_double2(s * v.x, s * v.y)) ? zero() : v; }
  static __device__ __forceinline__ T times(double g, T v) { return make_double2(g * v.x, g * v.y); }
  static __device__ __forceinline__ T add_scaled(T y, T a, double s) { return make_double2(fma(s, a.x, y.x), fma(s, a.y, y.y)); }
  static __device__ __forceinline__ Cf coef(double2 c) { return c; }
  static __device__ __forceinline__ Cf signed_coef(Cf c, uint32_t e) {
    const int f = static_cast<int>(e & 0x80000000u);
    return make_double2(__hiloint2double(__double2hiint(c.x) ^ f, __double2loint(c.x)),
                        __hiloint2double(__double2hiint(c.y) ^ f, __double2loint(c.y)));
  }
  static __device__ __forceinline__ void cmac(T& acc, Cf c, T v) {
    acc.x = fma(c.x, v.x, acc.x);
    acc.x = fma(-c.y, v.y, acc.x);
    acc.y = fma(c.x, v.y, acc.y);
    acc.y = fma(c.y, v.x, acc.y);
  }
  static __device__ __forceinline__ T shuffle(T v, int lane) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
  }
  static __device__ __forceinline__ void dot(double (&d)[2], T w, T y, double s) {  // conj(s w) y
    const double x = s * w.x, z = s * w.y;
    d[0] += x * y.x + z * y.y;
    d[1] += x * y.y - z * y.x;
  }
  static __device__ __forceinline__ Cf up_coef(const DevSector& S, int j) { return S.up_coef[j]; }
  static __device__ __forceinline__ Cf dn_coef(const DevSector& S, uint32_t e) {
    return signed_coef(S.dn_coef[(e >> 1) & 255u], e << 31);
  }
  static __device__ __forceinline__ double2 get(T v, int) { return v; }
  static __device__ __forceinline__ T make(const double2 (&z)[1]) { return z[0]; }
  static __device__ __forceinline__ double2 narrow(double re, double im) { return make_double2(re, im); }
};

// The two real coefficients of the gauge table as registers: an entry picks the second one where (entry & cls) is not
// zero and flips the sign by its bit 31.  In the XOR form the entry carries the bits by which the high words differ,
// so the second value is the first with the differing bits other than the sign flipped.
template <class P, bool kXor>
struct RowCoefs;
template <bool kXor>
struct RowCoefs<C64, kXor> {
  float a0, a1;
  float2 p0, p1;  // phase form: the two real values times (pc, ps)
  uint32_t cls;
  __device__ __forceinline__ explicit RowCoefs(const DevGauge& G) {
    a0 = __double2float_rn(G.real2[0]);
    p0 = make_float2(__double2float_rn(G.real2[0] * G.pc), __double2float_rn(G.real2[0] * G.ps));
    p1 = make_float2(__double2float_rn(G.real2[1] * G.pc), __double2float_rn(G.real2[1] * G.ps));
    if (kXor) {
      cls = 0x7FFC0000u;
      const int d = (__double2hiint(G.real2[0]) ^ __double2hiint(G.real2[1])) & 0x7FFC0000;
      a1 = __double2float_rn(__hiloint2double(__double2hiint(G.real2[0]) ^ d, __double2loint(G.real2[0])));
    } else {
      cls = 0x40000000u;
      a1 = __double2float_rn(G.real2[1]);
    }
  }
  static __device__ __forceinline__ float flip(float v, uint32_t bits) { return __uint_as_float(__float_as_uint(v) ^ bits); }
  __device__ __forceinline__ float pick(uint32_t e) const { return flip((e & cls) ? a1 : a0, e & 0x80000000u); }
  // Table-section entry in the phase form: real2[cls] (pc, +-ps), which is the table's value bit for bit.
  __device__ __forceinline__ float2 phase(uint32_t e) const {
    const float2 c = C64::signed_coef((e & 0x40000000u) ? p1 : p0, e);
    return make_float2(c.x, __uint_as_float(__float_as_uint(c.y) ^ ((e << 4) & 0x80000000u)));
  }
  static __device__ __forceinline__ void mac(float4& acc, float c, float4 v) {
    acc.x = fmaf(c, v.x, acc.x);
    acc.y = fmaf(c, v.y, acc.y);
    acc.z = fmaf(c, v.z, acc.z);
    acc.w = fmaf(c, v.w, acc.w);
  }
};

template <bool kXor>
struct RowCoefs<C128, kXor> {
  double a0, a1, pc, ps;
  __device__ __forceinline__ explicit RowCoefs(const DevGauge& G)
      : a0(G.real2[0]), a1(G.real2[1]), pc(G.pc), ps(G.ps) {}
  static __device__ __forceinline__ double flip(double v, uint32_t bits) {
    return __hiloint2double(__double2hiint(v) ^ static_cast<int>(bits), __double2loint(v));
  }
  __device__ __forceinline__ double pick(uint32_t e) const {
    if (kXor) return flip(a0, e & 0xFFFC0000u);
    return flip((e & 0x40000000u) ? a1 : a0, e & 0x80000000u);
  }
  // Table-section entry in the phase form: real2[cls] (pc, +-ps), bit for bit the table's value.
  __device__ __forceinline__ double2 phase(uint32_t e) const {
    const double c = flip((e & 0x40000000u) ? a1 : a0, e & 0x80000000u);
    return make_double2(c * pc, flip(c * ps, (e << 4) & 0x80000000u));
  }
  static __device__ __forceinline__ void mac(double2& acc, double c, double2 v) {
    acc.x = fma(c, v.x, acc.x);
    acc.y = fma(c, v.y, acc.y);
  }
};

// Sums of NV doubles over the block, in thread 0 (shuffles within a warp, then the warps in order).
template <int NV, int kT>
__device__ __forceinline__ void block_totals(double (&v)[NV], double* sh /* NV * kT / 32 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], o);
    if (lane == 0) sh[i * (kT / 32) + warp] = v[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double s = sh[i * (kT / 32)];
      for (int w = 1; w < kT / 32; ++w) s += sh[i * (kT / 32) + w];
      v[i] = s;
    }
  }
  __syncthreads();
}

// One output string of the row pass: the diagonal term and the down hops of kP staged lines (line p starts at base + p *
// line, Dd elements and 8 zeros for the table's padding entries), walked in the gauge table's order, so the sums do not
// depend on kP.
template <class P, int kP, bool kPhase, bool kXor>
struct RowSum {
  using Coefs = RowCoefs<P, kXor>;
  typename P::T acc[kP];
  uint32_t line;  // bytes per staged line
  const unsigned char* base;

  __device__ __forceinline__ const typename P::T& at(uint32_t e, int p) const {
    return *reinterpret_cast<const typename P::T*>(base + (e & 0x3FFF0u) + p * line);
  }
  __device__ __forceinline__ void real(uint32_t e, const Coefs& rc) {
    const auto c = rc.pick(e);
#pragma unroll
    for (int p = 0; p < kP; ++p) Coefs::mac(acc[p], c, at(e, p));
  }
  // Complex coefficient: from registers where the table has the phase form (kPhase), else from the block's copy of the
  // table (8 copies, copy i % 8: the 8 lanes of a quarter-warp read 8 different bank groups), with the entry's sign.
  __device__ __forceinline__ void cplx(uint32_t e, int i, const typename P::Cf* tab, const Coefs& rc) {
    typename P::Cf c;
    if constexpr (kPhase)
      c = rc.phase(e);
    else
      c = P::signed_coef(tab[((e >> 18) & 511u) * 8 + (i & 7)], e);
#pragma unroll
    for (int p = 0; p < kP; ++p) P::cmac(acc[p], c, at(e, p));
  }
  // The gauge-table walk of hv.cu's row pass for table position i (sections as whole 4-entry loads, the padding rounds
  // of each section's last load skipped, entry loads two ahead of use).
  __device__ __forceinline__ void walk(const DevGauge& G, int i, const typename P::Cf* tab, const Coefs& rc) {
    const int4 gp = G.grp[i >> 5];
    const int kr = gp.w & 0xFFFF, kt = gp.w >> 16;
    const uint4* ep = reinterpret_cast<const uint4*>(G.ent + gp.x) + (i & 31);
    uint4 cur = __ldg(ep);
    uint4 nxt = __ldg(ep + 32);
    int q = 0;
    auto next = [&]() {
      const uint4 e = cur;
      cur = nxt;
      nxt = __ldg(ep + (q + 2) * 32);
      ++q;
      return e;
    };
    for (int n = kr >> 2; n > 0; --n) {
      const uint4 e = next();
      real(e.x, rc);
      real(e.y, rc);
      real(e.z, rc);
      real(e.w, rc);
    }
    if (kr & 3) {
      const uint4 e = next();
      real(e.x, rc);
      if ((kr & 3) > 1) real(e.y, rc);
      if ((kr & 3) > 2) real(e.z, rc);
    }
    for (int n = kt >> 2; n > 0; --n) {
      const uint4 e = next();
      cplx(e.x, i, tab, rc);
      cplx(e.y, i, tab, rc);
      cplx(e.z, i, tab, rc);
      cplx(e.w, i, tab, rc);
    }
    if (kt & 3) {
      const uint4 e = next();
      cplx(e.x, i, tab, rc);
      if ((kt & 3) > 1) cplx(e.y, i, tab, rc);
      if ((kt & 3) > 2) cplx(e.z, i, tab, rc);
    }
  }
};

}  // namespace ftlm_b200
