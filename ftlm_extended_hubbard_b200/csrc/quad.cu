// Tridiagonal quadrature on the GPU, FP64 (reference src/ftlm_thermo.cpp:17-146, 150-256):
//   quad_jacobi   the reference's classical Jacobi (largest |off-diagonal| first, row-major
//                 first occurrence on ties), one warp per chain, the upper triangle in shared
//                 memory, only row 0 of the eigenvector matrix carried (rows of V never mix).
//                 Rotation arithmetic uses explicit round-to-nearest operations in the
//                 reference's evaluation order (no contraction), so results follow the
//                 reference's IEEE sequence up to the atan2/cos/sin implementations.
//   quad_eval     log sum_k w_k e^{-b lam_k} (+ the FTLM energy ratio) per chain and temperature.
//   quad_sector   ln(dim) + log mean_r e^{L_r} per temperature (src/ftlm_thermo.cpp:246-256).
//   gc_reduce     grand-canonical mu grid (benchmarks/bench_ftlm_nmu_rect.cpp:186-219).
//   ritz_bisect   exact Ritz values by Sturm-sequence bisection (lowest k).
#include <cfloat>
#include <math_constants.h>

#include "hv.cuh"
#include "launch.cuh"

namespace ftlm_b200 {

namespace {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// One warp per chain.  The strict upper triangle is packed (row i: A_ij, j > i, at tri_row(i) + j), the diagonal and
// row 0 of V apart.  The pivot comes from a maximum kept per row (lane k % 32 owns row k): a rotation (p, q) rewrites
// rows p and q, whose maxima are reduced as they are written, and the two entries (k, p), (k, q) of each row k above
// them.  Where the entry that was a row's maximum shrinks, the old value stays as an upper bound without a column,
// and the row is searched only when that bound is the largest of all (one rotation in three).  So the pivots, and
// with them every rotation, are those of a full search.
// The kernel is a serial chain of rotations (atan2, sincos, the row updates, the maxima), bound by its latency; the
// rows per lane are a template parameter so that nothing is spent on rows that are not there.  n = 60, 4 chains:
// 15.4 ms with a full search by 256 threads and four block barriers a rotation, 5.5 ms here (0.84 us a rotation, 0.37 of it
// the trigonometry); 1600 chains: 48 ms, here 8.1, since the packed triangle
// also lets 15 instead of 7 chains of n = 60 share an SM.
constexpr int kJacMaxRows = 5;       // rows per lane: n <= 160
constexpr unsigned kNoCol = 255u;    // the row's value is an upper bound, its column unknown

__device__ __forceinline__ int tri_row(int i, int n) { return i * n - (i * (i + 1)) / 2 - i - 1; }

// |v| as an ordered integer, 0 for NaN (which the strict > of a full search never takes either).
__device__ __forceinline__ unsigned long long jac_key(double v) {
  const unsigned long long k = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffull;
  return k > 0x7ff0000000000000ull ? 0ull : k;
}

// The lane that holds the warp's largest key, the smallest id among equals.  The upper halves decide unless two
// lanes share the largest one.
__device__ __forceinline__ int warp_top(unsigned long long key, unsigned id, unsigned mhi) {
  const unsigned hi = static_cast<unsigned>(key >> 32);
  unsigned m = __ballot_sync(0xffffffffu, hi == mhi);
  if (m & (m - 1u)) {
    const unsigned lo = static_cast<unsigned>(key);
    const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
    const bool top = hi == mhi && lo == mlo;
    const unsigned least = __reduce_min_sync(0xffffffffu, top ? id : 0xffffffffu);
    m = __ballot_sync(0xffffffffu, top && id == least);
  }
  return __ffs(static_cast<int>(m)) - 1;
}

template <int kRows>
__global__ void __launch_bounds__(32) jacobi_kernel(const double* __restrict__ alpha, const double* __restrict__ beta,
                                                    const int* __restrict__ nv, int ld, int max_rot_in, double tol,
                                                    double* __restrict__ lam, double* __restrict__ w0,
                                                    int* __restrict__ bad) {
  extern __shared__ double sm[];
  const int ch = blockIdx.x;
  int n = nv[ch];
  const int lane = threadIdx.x;
  // A chain length outside [0, ld] would overrun the shared triangle and the chain's rows of
  // alpha/beta/lam/w0: such a chain is skipped and reported through *bad (when given).
  if (n < 0 || n > ld) {
    if (lane == 0 && bad) atomicOr(bad, 1);
    n = 0;
  }
  const double* a = alpha + static_cast<int64_t>(ch) * ld;
  const double* b = beta + static_cast<int64_t>(ch) * ld;
  double* lo = lam + static_cast<int64_t>(ch) * ld;
  double* wo = w0 + static_cast<int64_t>(ch) * ld;
  if (n <= 0) return;
  if (n == 1) {
    if (lane == 0) {
      lo[0] = a[0];
      wo[0] = 1.0;
    }
    return;
  }
  double* D = sm;
  double* v0 = sm + n;
  double* A = sm + 2 * n;
  for (int i = lane; i < n * (n - 1) / 2; i += 32) A[i] = 0.0;
  __syncwarp();
  unsigned long long rk[kRows];  // per owned row k: key of its largest |A_kj|, j > k
  unsigned rc[kRows];            // and the first such column
  int ro[kRows];                 // tri_row of the row
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int k = lane + 32 * i;
    rk[i] = 0ull;
    rc[i] = static_cast<unsigned>(k + 1);
    ro[i] = tri_row(k, n);
    if (k < n) {
      D[k] = a[k];
      v0[k] = (k == 0) ? 1.0 : 0.0;
    }
    if (k + 1 < n) {
      A[ro[i] + k + 1] = b[k];
      rk[i] = jac_key(b[k]);
    }
  }
  __syncwarp();
  const int max_rot = max_rot_in > 0 ? max_rot_in : max(3000, 120 * n);
  for (int rot = 0; rot < max_rot; ++rot) {
    // Pivot: largest |A_ij| over i < j, first in row-major order (strict > as the reference).
    int p, q;
    unsigned long long big;
    for (;;) {
      unsigned long long v = rk[0];
      unsigned code = static_cast<unsigned>(lane) << 8 | rc[0];
#pragma unroll
      for (int i = 1; i < kRows; ++i)
        if (rk[i] > v) {
          v = rk[i];
          code = static_cast<unsigned>(lane + 32 * i) << 8 | rc[i];
        }
      const int src = warp_top(v, code, __reduce_max_sync(0xffffffffu, static_cast<unsigned>(v >> 32)));
      big = __shfl_sync(0xffffffffu, v, src);
      code = __shfl_sync(0xffffffffu, code, src);
      p = static_cast<int>(code >> 8);
      q = static_cast<int>(code & 255u);
      if (big == 0ull) {  // nothing off the diagonal: the reference's (0, 1)
        p = 0;
        q = 1;
        break;
      }
      if (q != static_cast<int>(kNoCol)) break;
      const double* row = A + tri_row(p, n);
      v = 0ull;
      code = 0u;
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int j = lane + 32 * i;
        const unsigned long long x = j > p && j < n ? jac_key(row[j]) : 0ull;
        if (x > v) {
          v = x;
          code = static_cast<unsigned>(j);
        }
      }
      const int at = warp_top(v, code, __reduce_max_sync(0xffffffffu, static_cast<unsigned>(v >> 32)));
      v = __shfl_sync(0xffffffffu, v, at);
      code = __shfl_sync(0xffffffffu, code, at);
#pragma unroll
      for (int i = 0; i < kRows; ++i)
        if (lane + 32 * i == p) {
          rk[i] = v;
          rc[i] = v ? code : static_cast<unsigned>(p + 1);
        }
    }
    if (!(__longlong_as_double(static_cast<long long>(big)) >= tol)) break;  // reference: break if max_abs < tol
    const int op = tri_row(p, n), oq = tri_row(q, n);
    const double app = D[p], aqq = D[q], apq = A[op + q];
    const double vip = v0[p], viq = v0[q];
    double apk[kRows], aqk[kRows];
    int ip[kRows], iq[kRows];
    bool in[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int k = lane + 32 * i;
      in[i] = k < n && k != p && k != q;
      ip[i] = k < p ? ro[i] + p : op + k;
      iq[i] = k < q ? ro[i] + q : oq + k;
      apk[i] = in[i] ? A[ip[i]] : 0.0;
      aqk[i] = in[i] ? A[iq[i]] : 0.0;
    }
    const double phi = mul(0.5, atan2(mul(2.0, apq), sub(aqq, app)));
    double c, s;
    sincos(phi, &s, &c);
    unsigned long long mp = 0ull, mq = 0ull;  // this lane's largest new entries of rows p and q
    unsigned cp = 0u, cq = 0u;
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int k = lane + 32 * i;
      const double rpk = sub(mul(c, apk[i]), mul(s, aqk[i]));
      const double rqk = add(mul(c, aqk[i]), mul(s, apk[i]));
      if (in[i]) {
        A[ip[i]] = rpk;
        A[iq[i]] = rqk;
      }
      const unsigned long long kp = in[i] ? jac_key(rpk) : 0ull, kq = in[i] ? jac_key(rqk) : 0ull;
      if (k > p && kp > mp) {
        mp = kp;
        cp = static_cast<unsigned>(k);
      }
      if (k > q && kq > mq) {
        mq = kq;
        cq = static_cast<unsigned>(k);
      }
      if (in[i] && k < q) {  // (k, q), and (k, p) where k < p, are entries of row k
        const bool both = k < p && kp >= kq;
        const unsigned long long x = both ? kp : kq;
        const unsigned xc = static_cast<unsigned>(both ? p : q);
        const bool was = rc[i] == static_cast<unsigned>(p) || rc[i] == static_cast<unsigned>(q);
        const bool up = x > rk[i];
        const bool tie = x == rk[i] && xc < rc[i] && rc[i] != kNoCol;
        rc[i] = up ? xc : was ? kNoCol : tie ? xc : rc[i];
        rk[i] = up ? x : rk[i];
      }
    }
    const unsigned hp = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(mp >> 32));
    const unsigned hq = __reduce_max_sync(0xffffffffu, static_cast<unsigned>(mq >> 32));
    const int lp = warp_top(mp, cp, hp), lq = warp_top(mq, cq, hq);
    mp = __shfl_sync(0xffffffffu, mp, lp);
    cp = __shfl_sync(0xffffffffu, cp, lp);
    mq = __shfl_sync(0xffffffffu, mq, lq);
    cq = __shfl_sync(0xffffffffu, cq, lq);
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int k = lane + 32 * i;
      if (k == p) {
        rk[i] = mp;
        rc[i] = mp ? cp : static_cast<unsigned>(k + 1);
      }
      if (k == q) {
        rk[i] = mq;
        rc[i] = mq ? cq : static_cast<unsigned>(k + 1);
      }
    }
    const double cc = mul(c, c), ss = mul(s, s), tsc = mul(mul(2.0, s), c);
    const double npp = add(sub(mul(cc, app), mul(tsc, apq)), mul(ss, aqq));
    const double nqq = add(add(mul(ss, app), mul(tsc, apq)), mul(cc, aqq));
    if (lane == 0) {
      D[p] = npp;
      D[q] = nqq;
      A[op + q] = 0.0;
      v0[p] = sub(mul(c, vip), mul(s, viq));
      v0[q] = add(mul(s, vip), mul(c, viq));
    }
    __syncwarp();
  }
  for (int k = lane; k < n; k += 32) {
    lo[k] = D[k];
    wo[k] = mul(v0[k], v0[k]);
  }
}

// src/ftlm_thermo.cpp:124-146 (log-sum-exp over Ritz pairs with w > 0) and the energy ratio.
__global__ void eval_kernel(const double* __restrict__ lam, const double* __restrict__ w0, const int* __restrict__ nv,
                            int nc, int ld, const double* __restrict__ bts, int nbt, double* __restrict__ logq,
                            double* __restrict__ energy, int* __restrict__ bad) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<int64_t>(nc) * nbt) return;
  const int ch = static_cast<int>(i / nbt), bi = static_cast<int>(i - static_cast<int64_t>(ch) * nbt);
  const int n = nv[ch];
  const double bT = bts[bi];
  const double* l = lam + static_cast<int64_t>(ch) * ld;
  const double* w = w0 + static_cast<int64_t>(ch) * ld;
  double out = -CUDART_INF, e = 0.0;
  if (n < 0 || n > ld) {  // invalid chain length (see jacobi_kernel): NaN outputs, reported
    if (bad) atomicOr(bad, 1);
    out = CUDART_NAN;
    e = CUDART_NAN;
  } else if (n == 1) {
    out = -bT * l[0];
    e = l[0];
  } else if (n > 1) {
    double mx = -CUDART_INF;
    for (int k = 0; k < n; ++k) {
      if (w[k] <= 0.0) continue;
      mx = fmax(mx, add(mul(-bT, l[k]), log(w[k])));
    }
    if (isfinite(mx)) {
      double s = 0.0, se = 0.0;
      for (int k = 0; k < n; ++k) {
        if (w[k] <= 0.0) continue;
        const double t = exp(sub(add(mul(-bT, l[k]), log(w[k])), mx));
        s = add(s, t);
        se = fma(l[k], t, se);
      }
      out = add(mx, log(s));
      e = se / s;
    }
  }
  logq[i] = out;
  energy[i] = e;
}

// src/ftlm_thermo.cpp:246-256: ln(dim) + max_l + log(sum_r e^{L_r - max_l} / count), chains
// with n <= 0 skipped.  Energy: e^{L_r}-weighted mean of the chain energies.
// One thread per sector and temperature; log_dims null: log_dim for all.
__global__ void sector_kernel(const double* __restrict__ logq_all, const double* __restrict__ eq_all,
                              const int* __restrict__ nv_all, int ns, int R, int nbt, double log_dim,
                              const double* __restrict__ log_dims, double* __restrict__ lnz_all,
                              double* __restrict__ energy_all) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ns * nbt) return;
  const int sec = i / nbt, bi = i - sec * nbt;
  const double* logq = logq_all + static_cast<int64_t>(sec) * R * nbt;
  const double* eq = eq_all + static_cast<int64_t>(sec) * R * nbt;
  const int* nv = nv_all + static_cast<int64_t>(sec) * R;
  double* lnz = lnz_all + static_cast<int64_t>(sec) * nbt;
  double* energy = energy_all + static_cast<int64_t>(sec) * nbt;
  if (log_dims) log_dim = log_dims[sec];
  double mx = -CUDART_INF;
  int cnt = 0;
  bool first = true;
  for (int r = 0; r < R; ++r) {
    if (nv[r] <= 0) continue;
    const double x = logq[r * nbt + bi];
    mx = first ? x : fmax(mx, x);
    first = false;
    ++cnt;
  }
  if (cnt == 0) {
    lnz[bi] = -CUDART_INF;
    energy[bi] = 0.0;
    return;
  }
  double s = 0.0, se = 0.0;
  for (int r = 0; r < R; ++r) {
    if (nv[r] <= 0) continue;
    const double t = exp(sub(logq[r * nbt + bi], mx));
    s = add(s, t);
    se = fma(t, eq[r * nbt + bi], se);
  }
  lnz[bi] = add(log_dim, add(mx, log(s / static_cast<double>(cnt))));
  energy[bi] = se / s;
}

__global__ void gc_kernel(const double* __restrict__ lnz_s, const double* __restrict__ e_s,
                          const int* __restrict__ N_s, int n_sec, const double* __restrict__ bts, int n_bt,
                          const double* __restrict__ mus, int n_mu, int n_sites, double* __restrict__ lnz_gc,
                          double* __restrict__ n_avg, double* __restrict__ e_avg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_bt * n_mu) return;
  const int b = i / n_mu, m = i - b * n_mu;
  const double bT = bts[b], mu = mus[m];
  const double bm = mul(bT, mu);
  double mx = -CUDART_INF;
  for (int s = 0; s < n_sec; ++s) {
    const double lz = lnz_s[static_cast<int64_t>(s) * n_bt + b];
    if (!isfinite(lz)) continue;
    mx = fmax(mx, add(lz, mul(bm, static_cast<double>(N_s[s]))));
  }
  if (!isfinite(mx)) {
    lnz_gc[i] = -CUDART_INF;
    n_avg[i] = 0.0;
    e_avg[i] = 0.0;
    return;
  }
  double sw = 0.0, snw = 0.0, sew = 0.0;
  for (int s = 0; s < n_sec; ++s) {
    const double lz = lnz_s[static_cast<int64_t>(s) * n_bt + b];
    if (!isfinite(lz)) continue;
    const double w = exp(sub(add(lz, mul(bm, static_cast<double>(N_s[s]))), mx));
    sw = add(sw, w);
    snw = add(snw, mul(static_cast<double>(N_s[s]), w));
    sew = fma(e_s[static_cast<int64_t>(s) * n_bt + b], w, sew);
  }
  lnz_gc[i] = add(mx, log(sw));
  n_avg[i] = (sw > 0.0) ? (snw / sw) / static_cast<double>(n_sites) : 0.0;
  e_avg[i] = (sw > 0.0) ? sew / sw : 0.0;
}

// Number of eigenvalues of the tridiagonal (a, b) strictly below x (Sturm sequence).
__device__ int sturm_count(const double* a, const double* b, int n, double x) {
  int cnt = 0;
  double d = 1.0;
  for (int i = 0; i < n; ++i) {
    const double bb = (i > 0) ? b[i - 1] * b[i - 1] : 0.0;
    d = (a[i] - x) - ((i > 0) ? bb / d : 0.0);
    if (d == 0.0) d = -DBL_MIN;  // pivot shift: treat an exact zero as a tiny negative
    if (d < 0.0) ++cnt;
  }
  return cnt;
}

__global__ void ritz_kernel(const double* __restrict__ a, const double* __restrict__ b, int n, int k,
                            double* __restrict__ ritz) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= k || j >= n) return;
  double lo = DBL_MAX, hi = -DBL_MAX;
  for (int i = 0; i < n; ++i) {
    const double r = ((i > 0) ? fabs(b[i - 1]) : 0.0) + ((i + 1 < n) ? fabs(b[i]) : 0.0);
    lo = fmin(lo, a[i] - r);
    hi = fmax(hi, a[i] + r);
  }
  const double span = hi - lo;
  lo -= 1e-12 * span + DBL_MIN;
  hi += 1e-12 * span + DBL_MIN;
  for (int it = 0; it < 200; ++it) {
    const double mid = 0.5 * (lo + hi);
    if (mid <= lo || mid >= hi) break;
    if (sturm_count(a, b, n, mid) > j)
      hi = mid;
    else
      lo = mid;
  }
  ritz[j] = 0.5 * (lo + hi);
}

}  // namespace

cudaError_t quad_jacobi(const double* alpha, const double* beta, const int* n, int nc, int ld, int max_rot,
                        double tol, double* lam, double* w0, cudaStream_t st, int* bad) {
  if (nc <= 0) return cudaSuccess;
  if (ld <= 0 || ld > 32 * kJacMaxRows) return cudaErrorInvalidValue;
  using K = void (*)(const double*, const double*, const int*, int, int, double, double*, double*, int*);
  static const K kernels[kJacMaxRows] = {jacobi_kernel<1>, jacobi_kernel<2>, jacobi_kernel<3>, jacobi_kernel<4>,
                                         jacobi_kernel<5>};
  const K k = kernels[(ld - 1) / 32];
  const size_t sm = (static_cast<size_t>(ld) * (ld - 1) / 2 + 2 * static_cast<size_t>(ld)) * sizeof(double);
  const cudaError_t e = allow_shared(k, sm);
  if (e != cudaSuccess) return e;
  k<<<nc, 32, sm, st>>>(alpha, beta, n, ld, max_rot, tol, lam, w0, bad);
  return cudaGetLastError();
}

cudaError_t quad_eval(const double* lam, const double* w0, const int* n, int nc, int ld, const double* bts, int nbt,
                      double* logq, double* energy, cudaStream_t st, int* bad) {
  const int64_t tot = static_cast<int64_t>(nc) * nbt;
  if (tot <= 0) return cudaSuccess;
  if ((tot + 127) / 128 > 0x7fffffffLL) return cudaErrorInvalidValue;
  eval_kernel<<<static_cast<unsigned>((tot + 127) / 128), 128, 0, st>>>(lam, w0, n, nc, ld, bts, nbt, logq, energy,
                                                                       bad);
  return cudaGetLastError();
}

cudaError_t quad_sector(const double* logq, const double* eq, const int* n, int R, int nbt, double log_dim,
                        double* lnz, double* energy, cudaStream_t st) {
  if (nbt <= 0) return cudaSuccess;
  sector_kernel<<<(nbt + 127) / 128, 128, 0, st>>>(logq, eq, n, 1, R, nbt, log_dim, nullptr, lnz, energy);
  return cudaGetLastError();
}

cudaError_t quad_sectors(const double* logq, const double* eq, const int* n, int ns, int R, int nbt,
                         const double* log_dims, double* lnz, double* energy, cudaStream_t st) {
  if (nbt <= 0 || ns <= 0) return cudaSuccess;
  sector_kernel<<<(ns * nbt + 63) / 64, 64, 0, st>>>(logq, eq, n, ns, R, nbt, 0.0, log_dims, lnz, energy);
  return cudaGetLastError();
}

cudaError_t gc_reduce_dev(const double* lnz_s, const double* e_s, const int* N_s, int n_sec, const double* bts,
                          int n_bt, const double* mus, int n_mu, int n_sites, double* lnz_gc, double* n_avg,
                          double* e_avg, cudaStream_t st) {
  const int tot = n_bt * n_mu;
  if (tot <= 0) return cudaSuccess;
  gc_kernel<<<(tot + 127) / 128, 128, 0, st>>>(lnz_s, e_s, N_s, n_sec, bts, n_bt, mus, n_mu, n_sites, lnz_gc, n_avg,
                                                e_avg);
  return cudaGetLastError();
}

cudaError_t ritz_bisect(const double* alpha, const double* beta, int n, int k, double* ritz, cudaStream_t st) {
  if (k <= 0 || n <= 0) return cudaSuccess;
  ritz_kernel<<<(k + 63) / 64, 64, 0, st>>>(alpha, beta, n, k, ritz);
  return cudaGetLastError();
}

}  // namespace ftlm_b200
