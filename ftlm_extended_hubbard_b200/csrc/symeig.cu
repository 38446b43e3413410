// Small dense symmetric eigen-problems on the GPU (FP64), one CTA per matrix:
//
//   symeig_kernel   parallel cyclic Jacobi (Brent-Luk round-robin ordering: m/2 disjoint rotations
//                   per round, m-1 rounds per sweep, sweeps until the off-diagonal Frobenius norm is
//                   below 1e-15 of the matrix norm), the matrix in shared memory (m <= 160, row
//                   stride m+1 so that column accesses of a warp fall in distinct bank pairs):
//                   eigenvalues of a dense matrix in ascending order.
//   tql_weights_kernel, tql_vectors_kernel
//                   implicit QL iteration of a tridiagonal matrix (Dubrulle, Martin and Wilkinson,
//                   Numer. Math. 12, 377 (1968)): eigenvalues in ascending order with the
//                   squared first row of the eigenvector matrix (the quadrature weights), or with all
//                   eigenvectors (row j of Vt = eigenvector j).
//   duhamel_kernel  the Duhamel weight matrix of one Lanczos chain from its eigen-decomposition:
//                   K = Z P Z^T, P_jk = Z_0j Z_0k (e^{-b l_j} - e^{-b l_k}) / (l_k - l_j) (the limit
//                   b e^{-b l_j} on the diagonal), with the same shift l_0 and the same expm1 form
//                   as the host restatement (tridiag.cpp), written in the moment kernel's layout.
//
// These replace host eigen-solves on the product paths: the converged quadrature of the
// differentiable forward, the gradient's Duhamel weights and the exact small-block ED of the
// k-resolved path (reference benchmarks/bench_ftlm_nmu_4x4_k.cpp:249-336 restated).
#include <cfloat>

#include "launch.cuh"
#include "symeig.cuh"

namespace ftlm_b200 {

namespace {

constexpr int kEigThreads = 256;
constexpr size_t kEigOwn = 2560;  // static shared memory of the kernels here, at most

// Pair k of round r of the circle method for m (even) players: player m-1 is fixed.
__device__ __forceinline__ void rr_pair(int r, int k, int m, int* p, int* q) {
  int a, b;
  if (k == 0) {
    a = r;
    b = m - 1;
  } else {
    a = (r + k) % (m - 1);
    b = (r - k + (m - 1)) % (m - 1);
  }
  *p = min(a, b);
  *q = max(a, b);
}

__global__ void __launch_bounds__(kEigThreads) symeig_kernel(const double* __restrict__ dense,
                                                             const int* __restrict__ nv, int ld,
                                                             double* __restrict__ lam, int* __restrict__ info) {
  extern __shared__ double sm[];
  __shared__ double rc[kMaxEig / 2], rs[kMaxEig / 2];
  __shared__ int rp[kMaxEig / 2], rq[kMaxEig / 2];
  __shared__ double red[kEigThreads / 32];
  __shared__ int s_done;
  const int ch = blockIdx.x;
  const int tid = threadIdx.x;
  int n = nv[ch];
  if (n < 0 || n > ld || ld > kMaxEig) {  // out of range: report, touch nothing
    if (tid == 0 && info) info[ch] = 2;
    return;
  }
  double* lo = lam + static_cast<int64_t>(ch) * ld;
  if (n == 0) {
    if (tid == 0 && info) info[ch] = 0;
    return;
  }
  const int m = n + (n & 1);  // even order; a padding index stays decoupled (zero row and column)
  const int S = m + 1;        // row stride in shared memory
  double* A = sm;
  for (int i = tid; i < m * S; i += kEigThreads) {
    const int r = i / S, c = i - r * S;
    double v = 0.0;
    if (r < n && c < n) v = dense[static_cast<int64_t>(ch) * ld * ld + static_cast<int64_t>(r) * ld + c];
    A[i] = v;
  }
  __syncthreads();
  // Frobenius norm for the stopping rule
  double fro = 0.0;
  for (int i = tid; i < m * S; i += kEigThreads) fro += A[i] * A[i];
  for (int off = 16; off > 0; off >>= 1) fro += __shfl_down_sync(0xffffffffu, fro, off);
  if ((tid & 31) == 0) red[tid >> 5] = fro;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < kEigThreads / 32; ++w) t += red[w];
    red[0] = t;
  }
  __syncthreads();
  const double stop = 1e-30 * red[0];  // off^2 <= (1e-15 ||A||_F)^2
  const int half = m / 2;
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    // off-diagonal norm
    double off2 = 0.0;
    for (int i = tid; i < m * S; i += kEigThreads) {
      const int r = i / S, c = i - r * S;
      if (c < m && r != c) off2 += A[i] * A[i];
    }
    for (int o = 16; o > 0; o >>= 1) off2 += __shfl_down_sync(0xffffffffu, off2, o);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = off2;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < kEigThreads / 32; ++w) t += red[w];
      s_done = !(t > stop);
    }
    __syncthreads();
    if (s_done) break;
    for (int r = 0; r < m - 1; ++r) {
      for (int k = tid; k < half; k += kEigThreads) {
        int p, q;
        rr_pair(r, k, m, &p, &q);
        const double apq = A[p * S + q];
        double c = 1.0, s = 0.0;
        if (apq != 0.0) {
          const double theta = (A[q * S + q] - A[p * S + p]) / (2.0 * apq);
          const double t = copysign(1.0, theta) / (fabs(theta) + sqrt(theta * theta + 1.0));
          c = 1.0 / sqrt(t * t + 1.0);
          s = t * c;
        }
        rc[k] = c;
        rs[k] = s;
        rp[k] = p;
        rq[k] = q;
      }
      __syncthreads();
      // rows: A <- J^T A
      for (int i = tid; i < half * m; i += kEigThreads) {
        const int k = i / m, j = i - k * m;
        const int p = rp[k], q = rq[k];
        const double c = rc[k], s = rs[k];
        const double x = A[p * S + j], y = A[q * S + j];
        A[p * S + j] = c * x - s * y;
        A[q * S + j] = s * x + c * y;
      }
      __syncthreads();
      // columns: A <- A J
      for (int i = tid; i < half * m; i += kEigThreads) {
        const int k = i / m, j = i - k * m;
        const int p = rp[k], q = rq[k];
        const double c = rc[k], s = rs[k];
        const double x = A[j * S + p], y = A[j * S + q];
        A[j * S + p] = c * x - s * y;
        A[j * S + q] = s * x + c * y;
      }
      __syncthreads();
      for (int k = tid; k < half; k += kEigThreads) {  // the rotation annihilates a_pq
        const int p = rp[k], q = rq[k];
        if (rs[k] != 0.0) {
          A[p * S + q] = 0.0;
          A[q * S + p] = 0.0;
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0 && info) info[ch] = s_done ? 0 : 1;
  // ascending order (ties by index): rank sort over the n real eigenvalues (the padding index, if
  // any, is index n and excluded)
  __syncthreads();
  for (int j = tid; j < n; j += kEigThreads) {
    const double lj = A[j * S + j];
    int rank = 0;
    for (int k = 0; k < n; ++k) {
      const double lk = A[k * S + k];
      rank += (lk < lj || (lk == lj && k < j)) ? 1 : 0;
    }
    lo[rank] = lj;
  }
}

// Implicit QL iteration of one symmetric tridiagonal of order n: d[i * st] the diagonal and e[i * st] the entry
// below it (e[n - 1] = 0), overwritten by the eigenvalues and zeros; every rotation is applied to columns i and
// i + 1 of one row of the eigenvector matrix, z[i * zst].  The rotations of a sweep are a serial chain (one rsqrt and
// about eight multiply-adds each), which bounds both kernels below; the loads of the next rotation are issued before
// the chain of this one.  Returns whether every eigenvalue converged within 60 sweeps.
__device__ __forceinline__ bool tql(double* d, double* e, int st, double* z, int zst, int n) {
  constexpr double kEps = 2.220446049250313e-16;
  for (int l = 0; l < n; ++l) {
    for (int it = 0;; ++it) {
      int m = l;
      double dm = d[l * st];
      for (; m < n - 1; ++m) {
        const double dn = d[(m + 1) * st];
        if (fabs(e[m * st]) <= kEps * (fabs(dm) + fabs(dn))) break;
        dm = dn;
      }
      if (m == l) break;
      if (it == 60) return false;
      const double el = e[l * st], dl = d[l * st];
      double g = (d[(l + 1) * st] - dl) / (2.0 * el);
      const double r0 = sqrt(fma(g, g, 1.0));
      g = dm - dl + el / (g + copysign(r0, g));
      double s = 1.0, c = 1.0, p = 0.0;
      double dnext = dm, ei = e[(m - 1) * st], di = d[(m - 1) * st], zi = z[(m - 1) * zst], zn = z[m * zst];
      int i = m - 1;
      for (; i >= l; --i) {
        const double f = s * ei, b = c * ei, dcur = di, zcur = zi;
        if (i > l) {
          ei = e[(i - 1) * st];
          di = d[(i - 1) * st];
          zi = z[(i - 1) * zst];
        }
        const double h = fma(f, f, g * g);
        if (h == 0.0) {  // the matrix splits at i + 1
          d[(i + 1) * st] = dnext - p;
          e[(i + 1) * st] = 0.0;
          e[m * st] = 0.0;
          z[(i + 1) * zst] = zn;
          break;
        }
        const double inv = rsqrt(h);
        e[(i + 1) * st] = h * inv;
        s = f * inv;
        c = g * inv;
        g = dnext - p;
        const double t = fma(dcur - g, s, 2.0 * c * b);
        p = s * t;
        d[(i + 1) * st] = g + p;
        g = fma(c, t, -b);
        dnext = dcur;
        z[(i + 1) * zst] = fma(s, zcur, c * zn);
        zn = fma(c, zcur, -s * zn);
      }
      if (i >= l) continue;
      d[l * st] = dnext - p;
      e[l * st] = g;
      e[m * st] = 0.0;
      z[l * zst] = zn;
    }
  }
  return true;
}

// Power of two that brings the largest |a_i|, |b_i| (n of the former, n - 1 of the latter) into [1, 2), so that the
// squares in tql neither overflow nor underflow; 0 for a zero matrix or entries that are not finite.
__device__ __forceinline__ double tql_scale(double big) {
  if (!(big > 0.0) || !(big <= DBL_MAX)) return 0.0;
  return scalbn(1.0, -ilogb(big));
}

// Chains per block: one lane each.  A chain is one lane's serial work, so few share a warp (the others wait for the
// longest); 32 chains of n = 80 are 8 blocks.
constexpr int kTqlChains = 4;

// Eigenvalues (ascending) and first-row weights.  Bound by the serial chain of about 0.85 n^2 rotations: 32 chains of
// n = 80 take 1.1 ms, against 2.3 ms for the parallel cyclic Jacobi on the dense matrix.
__global__ void __launch_bounds__(32) tql_weights_kernel(const double* __restrict__ alpha,
                                                         const double* __restrict__ beta, const int* __restrict__ nv,
                                                         int nm, int ld, double* __restrict__ lam,
                                                         double* __restrict__ w0, int* __restrict__ info) {
  extern __shared__ double sm[];
  const int lane = threadIdx.x;
  const int ch0 = blockIdx.x * kTqlChains;
  double* d = sm;
  double* e = d + ld * kTqlChains;
  double* z = e + ld * kTqlChains;
  for (int i = lane; i < ld * kTqlChains; i += 32) {
    const int ch = ch0 + i / ld, k = i % ld, at = k * kTqlChains + i / ld;
    const int n = ch < nm ? nv[ch] : 0;
    const bool in = k < n && n <= ld;
    d[at] = in ? alpha[static_cast<int64_t>(ch) * ld + k] : 0.0;
    e[at] = in && k + 1 < n ? beta[static_cast<int64_t>(ch) * ld + k] : 0.0;
    z[at] = k == 0 ? 1.0 : 0.0;
  }
  __syncwarp();
  double unscale = 1.0;
  if (lane < kTqlChains && ch0 + lane < nm) {
    const int n = nv[ch0 + lane];
    if (n < 0 || n > ld) {  // out of range: report, write nothing
      if (info) info[ch0 + lane] = 2;
    } else {
      double big = 0.0;
      bool finite = true;
      for (int k = 0; k < n; ++k) {
        const double a = fabs(d[k * kTqlChains + lane]), b = fabs(e[k * kTqlChains + lane]);
        finite = finite && a <= DBL_MAX && b <= DBL_MAX;
        big = fmax(big, fmax(a, b));
      }
      const double sc = finite ? tql_scale(big) : 0.0;
      bool ok = true;
      if (sc != 0.0) {
        for (int k = 0; k < n; ++k) {
          d[k * kTqlChains + lane] *= sc;
          e[k * kTqlChains + lane] *= sc;
        }
        ok = tql(d + lane, e + lane, kTqlChains, z + lane, kTqlChains, n);
        unscale = 1.0 / sc;
      }
      if (info) info[ch0 + lane] = ok ? 0 : 1;
    }
  }
  __syncwarp();
  for (int c = 0; c < kTqlChains && ch0 + c < nm; ++c) {
    const int n = nv[ch0 + c];
    if (n < 0 || n > ld) continue;
    const double us = __shfl_sync(0xffffffffu, unscale, c);
    for (int j = lane; j < n; j += 32) {
      const double lj = d[j * kTqlChains + c];
      int rank = 0;
      for (int k = 0; k < n; ++k) {
        const double lk = d[k * kTqlChains + c];
        rank += (lk < lj || (lk == lj && k < j)) ? 1 : 0;
      }
      const double zj = z[j * kTqlChains + c];
      lam[static_cast<int64_t>(ch0 + c) * ld + rank] = lj * us;
      w0[static_cast<int64_t>(ch0 + c) * ld + rank] = zj * zj;
    }
  }
}

// Eigenvalues (ascending) and all eigenvectors, one block per matrix: thread k owns row k of the eigenvector matrix
// (Z[i][k] in shared memory, conflict-free), and every warp runs the scalar recurrence on its own copy of the
// tridiagonal, identically, so no barrier is needed until the end.
__global__ void __launch_bounds__(kMaxEig) tql_vectors_kernel(const double* __restrict__ alpha,
                                                              const double* __restrict__ beta,
                                                              const int* __restrict__ nv, int ld,
                                                              double* __restrict__ lam, double* __restrict__ vt,
                                                              int* __restrict__ info) {
  extern __shared__ double sm[];
  const int ch = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n = nv[ch];
  if (n < 0 || n > ld) {
    if (tid == 0 && info) info[ch] = 2;
    return;
  }
  double* d = sm + 2 * ld * warp;
  double* e = d + ld;
  double* z = sm + 2 * ld * (blockDim.x >> 5) + tid;
  const int zst = blockDim.x;
  double big = 0.0;
  bool finite = true;
  for (int i = lane; i < n; i += 32) {
    d[i] = alpha[static_cast<int64_t>(ch) * ld + i];
    e[i] = i + 1 < n ? beta[static_cast<int64_t>(ch) * ld + i] : 0.0;
    finite = finite && fabs(d[i]) <= DBL_MAX && fabs(e[i]) <= DBL_MAX;
    big = fmax(big, fmax(fabs(d[i]), fabs(e[i])));
  }
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  finite = __all_sync(0xffffffffu, finite);
  for (int i = 0; i < n; ++i) z[i * zst] = i == tid ? 1.0 : 0.0;
  const double sc = finite ? tql_scale(big) : 0.0;
  bool ok = true;
  if (sc != 0.0) {
    for (int i = lane; i < n; i += 32) {
      d[i] *= sc;
      e[i] *= sc;
    }
    __syncwarp();
    ok = tql(d, e, 1, z, zst, n);
  }
  __syncwarp();
  if (tid == 0 && info) info[ch] = ok ? 0 : 1;
  const double us = sc != 0.0 ? 1.0 / sc : 1.0;
  for (int j = 0; j < n; ++j) {
    const double lj = d[j];
    int rank = 0;
    for (int k = lane; k < n; k += 32) rank += (d[k] < lj || (d[k] == lj && k < j)) ? 1 : 0;
    rank = __reduce_add_sync(0xffffffffu, rank);
    if (tid == 0) lam[static_cast<int64_t>(ch) * ld + rank] = lj * us;
    if (tid < n) vt[(static_cast<int64_t>(ch) * ld + rank) * ld + tid] = z[j * zst];
  }
}

// K = Z P Z^T in the moment kernel's layout Kp[(c*ld + i)*ld + l] / (sc_i sc_l), 0 outside the chain's n rows, with
// Z[i][j] = Vt[j][i] (ascending l_j); g = sum_j Z_0j^2 e^{-b (l_j - l_0)}, lmin = l_0.
// P is formed once in shared memory (one expm1 and one division an entry); both products then read it and V.
constexpr int kDuhThreads = 512;

__global__ void __launch_bounds__(kDuhThreads) duhamel_kernel(const double* __restrict__ lam,
                                                              const double* __restrict__ vt,
                                                              const int* __restrict__ nv, int ld, double bT,
                                                              const double* __restrict__ scale,
                                                              double* __restrict__ Y, double* __restrict__ Kp,
                                                              double* __restrict__ g_out,
                                                              double* __restrict__ lmin_out) {
  extern __shared__ double P[];  // [n][n]
  const int ch = blockIdx.x;
  const int tid = threadIdx.x;
  const int n = nv[ch];
  double* Kc = Kp + static_cast<int64_t>(ch) * ld * ld;
  if (n <= 0 || n > ld) {
    for (int e = tid; e < ld * ld; e += kDuhThreads) Kc[e] = 0.0;
    if (tid == 0) g_out[ch] = lmin_out[ch] = 0.0;
    return;
  }
  const double* l = lam + static_cast<int64_t>(ch) * ld;
  const double* V = vt + static_cast<int64_t>(ch) * ld * ld;  // V[j*ld + i] = Z[i][j]
  double* y = Y + static_cast<int64_t>(ch) * ld * ld;
  const double* sc = scale + static_cast<int64_t>(ch) * ld;
  const double shift = l[0];
  __shared__ double ew[kMaxEig], z0[kMaxEig];
  for (int j = tid; j < n; j += kDuhThreads) {
    ew[j] = exp(-bT * (l[j] - shift));
    z0[j] = V[static_cast<int64_t>(j) * ld];
  }
  __syncthreads();
  for (int e = tid; e < n * n; e += kDuhThreads) {
    const int j = e / n, k = e - j * n;
    const int a = min(j, k), b = max(j, k);
    const double ea = ew[a];
    const double delta = l[b] - l[a];
    P[e] = z0[j] * ((a == b || delta == 0.0) ? bT * ea : ea * (-expm1(-bT * delta)) / delta);
  }
  __syncthreads();
  // Y[i][k] = sum_j Z_ij Z_0j D_jk, then K_il = sum_k Y_ik Z_0k Z_lk
  for (int e = tid; e < n * n; e += kDuhThreads) {
    const int k = e / n, i = e - k * n;
    double acc = 0.0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) acc = fma(V[static_cast<int64_t>(j) * ld + i], P[j * n + k], acc);
    y[static_cast<int64_t>(k) * ld + i] = acc * z0[k];
  }
  __syncthreads();
  for (int e = tid; e < ld * ld; e += kDuhThreads) {
    const int i = e / ld, lq = e - i * ld;
    double acc = 0.0;
    if (i < n && lq < n) {
#pragma unroll 4
      for (int k = 0; k < n; ++k)
        acc = fma(y[static_cast<int64_t>(k) * ld + i], V[static_cast<int64_t>(k) * ld + lq], acc);
      acc /= sc[i] * sc[lq];
    }
    Kc[e] = acc;
  }
  if (tid == 0) {
    double gs = 0.0;
    for (int j = 0; j < n; ++j) gs += z0[j] * z0[j] * ew[j];
    g_out[ch] = gs;
    lmin_out[ch] = shift;
  }
}

// R = [[Re H, -Im H], [Im H, Re H]] (2dk x 2dk, row-major) from the columns of H (column j at
// cols + j*dk): the real symmetric embedding of a Hermitian matrix (each eigenvalue twice).
__global__ void embed_kernel(const double2* __restrict__ cols, int dk, double* __restrict__ R) {
  const int m = 2 * dk;
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= static_cast<int64_t>(dk) * dk) return;
  const int j = static_cast<int>(e / dk), i = static_cast<int>(e - static_cast<int64_t>(j) * dk);
  const double2 h = cols[static_cast<int64_t>(j) * dk + i];  // H[i][j]
  R[static_cast<int64_t>(i) * m + j] = h.x;
  R[static_cast<int64_t>(i) * m + j + dk] = -h.y;
  R[static_cast<int64_t>(i + dk) * m + j] = h.y;
  R[static_cast<int64_t>(i + dk) * m + j + dk] = h.x;
}

}  // namespace

cudaError_t embed_hermitian(const double2* cols, int dk, double* R, cudaStream_t st) {
  const int64_t tot = static_cast<int64_t>(dk) * dk;
  if (tot <= 0) return cudaSuccess;
  embed_kernel<<<static_cast<unsigned>((tot + 255) / 256), 256, 0, st>>>(cols, dk, R);
  return cudaGetLastError();
}

cudaError_t symeig_tridiag(const double* alpha, const double* beta, const int* n, int nm, int ld, double* lam,
                           double* v0, double* vt, int* info, cudaStream_t st) {
  if (nm <= 0) return cudaSuccess;
  if (ld > kMaxEig || ld <= 0 || (!v0 && !vt)) return cudaErrorInvalidValue;
  if (vt) {
    const int threads = (ld + 31) / 32 * 32;
    const size_t sm = (static_cast<size_t>(2) * ld * (threads / 32) + static_cast<size_t>(ld) * threads) * sizeof(double);
    const cudaError_t e = allow_shared(tql_vectors_kernel, sm);
    if (e != cudaSuccess) return e;
    tql_vectors_kernel<<<nm, threads, sm, st>>>(alpha, beta, n, ld, lam, vt, info);
  } else {
    const size_t sm = static_cast<size_t>(3) * ld * kTqlChains * sizeof(double);
    tql_weights_kernel<<<(nm + kTqlChains - 1) / kTqlChains, 32, sm, st>>>(alpha, beta, n, nm, ld, lam, v0, info);
  }
  return cudaGetLastError();
}

cudaError_t symeig_dense(const double* A, const int* n, int nm, int ld, double* lam, int* info, cudaStream_t st) {
  if (nm <= 0) return cudaSuccess;
  if (ld > kMaxEig || ld <= 0) return cudaErrorInvalidValue;
  const int m = ld + (ld & 1);
  const size_t sm = (static_cast<size_t>(m) * (m + 1) + m) * sizeof(double);
  const cudaError_t e = allow_shared(symeig_kernel, sm, kEigOwn);
  if (e != cudaSuccess) return e;
  symeig_kernel<<<nm, kEigThreads, sm, st>>>(A, n, ld, lam, info);
  return cudaGetLastError();
}

cudaError_t duhamel_weights_dev(const double* lam, const double* vt, const int* n, int nc, int ld, double bT,
                                const double* scale, double* Y, double* Kp, double* g, double* lmin, cudaStream_t st) {
  if (nc <= 0) return cudaSuccess;
  const size_t sm = static_cast<size_t>(ld) * ld * sizeof(double);
  const cudaError_t e = allow_shared(duhamel_kernel, sm, kEigOwn);
  if (e != cudaSuccess) return e;
  duhamel_kernel<<<nc, kDuhThreads, sm, st>>>(lam, vt, n, ld, bT, scale, Y, Kp, g, lmin);
  return cudaGetLastError();
}

}  // namespace ftlm_b200
