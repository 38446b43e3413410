// Krylov moments for the FTLM parameter gradient; contract in grad.cuh.
//
// Block = kE consecutive states of one plane (of the planes' one or two chains).  A thread keeps its own state's
// entry of every W_l in shared memory (only it reads them: conflict-free, no barrier), then for rows i, kIB at a time,
// the block stages K'[i][*] of the plane's chains and forms
//   X_i = sum_l K'_il W_l   (FP64),
// accumulating Re(conj W_i X_i) (times the diagonal operators) and Re(conj(A W_i) X_i).  Bound by the FP64 rate for
// long chains (4 n^2 operations per chain and state); kIB rows share each conversion of W_l to FP64 and each load.
// Fixed grid and fixed per-block order: the sums are bitwise repeatable.
#include <algorithm>

#include "grad.cuh"
#include "launch.cuh"

namespace ftlm_b200 {

namespace {

constexpr int kIB = 4;  // rows of K' staged per pass

template <typename T>
struct Elem;
template <>
struct Elem<float4> {  // two complex64 chains
  static constexpr int kC = 2;
  static __device__ __forceinline__ void get(const float4& v, double (&re)[2], double (&im)[2]) {
    re[0] = v.x;
    im[0] = v.y;
    re[1] = v.z;
    im[1] = v.w;
  }
};
template <>
struct Elem<double2> {  // one complex128 chain
  static constexpr int kC = 1;
  static __device__ __forceinline__ void get(const double2& v, double (&re)[1], double (&im)[1]) {
    re[0] = v.x;
    im[0] = v.y;
  }
};

template <typename T>
__global__ void __launch_bounds__(256) moments_kernel(DevSector S, const T* __restrict__ W, const T* __restrict__ AW,
                                                      int64_t vstride, int64_t pstride, const double* __restrict__ Kp,
                                                      const int* __restrict__ used, int chains, int ld, int nb,
                                                      double* __restrict__ partial) {
  constexpr int kC = Elem<T>::kC;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int E = blockDim.x;
  const int t = threadIdx.x;
  const int plane = blockIdx.x / nb, b = blockIdx.x - plane * nb;
  int n = 0;  // the plane's longest chain
#pragma unroll
  for (int q = 0; q < kC; ++q)
    if (plane * kC + q < chains) n = max(n, min(used[plane * kC + q], ld));
  T* Ws = reinterpret_cast<T*>(smraw);                                                    // [n][E]
  double* Ks = reinterpret_cast<double*>(smraw + static_cast<size_t>(n) * E * sizeof(T));  // [n][kIB][kC]
  const T* Wp = W + plane * pstride;
  const T* Ap = AW + plane * pstride;
  const double* Kc = Kp + static_cast<int64_t>(plane) * kC * ld * ld;
  double accD[kC] = {}, accP[kC] = {}, accA[kC] = {};
  const int64_t nch = (S.dim + E - 1) / E;
  for (int64_t ch = b; ch < nch; ch += nb) {
    const int64_t e = ch * E + t;
    const bool valid = e < S.dim;
    double aD = 0.0, aP = 0.0;
    if (valid) {
      for (int l = 0; l < n; ++l) Ws[l * E + t] = Wp[static_cast<int64_t>(l) * vstride + e];
      const int64_t ru = e / S.Dd, rd = e - ru * S.Dd;
      const uint32_t u = S.umask[ru], d = S.dmask[rd];
      const uint4 w = S.wpl[ru];
      aD = static_cast<double>(__popc(u & d));
      aP = static_cast<double>(S.cnt_uu[ru] + S.cnt_dd[rd] + __popc(d & w.x) + 2 * __popc(d & w.y) +
                               4 * __popc(d & w.z) + 8 * __popc(d & w.w));
    }
    double sW[kC] = {}, sA[kC] = {};
    for (int i0 = 0; i0 < n; i0 += kIB) {
      __syncthreads();
      for (int idx = t; idx < kIB * n * kC; idx += E) {
        const int l = idx % n, q = idx / n % kC, ib = idx / (n * kC);
        Ks[(l * kIB + ib) * kC + q] =
            (i0 + ib < n && plane * kC + q < chains) ? Kc[(static_cast<int64_t>(q) * ld + i0 + ib) * ld + l] : 0.0;
      }
      __syncthreads();
      if (!valid) continue;
      double xr[kIB][kC] = {}, xi[kIB][kC] = {};
      for (int l = 0; l < n; ++l) {
        double re[kC], im[kC];
        Elem<T>::get(Ws[l * E + t], re, im);
#pragma unroll
        for (int ib = 0; ib < kIB; ++ib) {
#pragma unroll
          for (int q = 0; q < kC; ++q) {
            const double k = Ks[(l * kIB + ib) * kC + q];
            xr[ib][q] = fma(k, re[q], xr[ib][q]);
            xi[ib][q] = fma(k, im[q], xi[ib][q]);
          }
        }
      }
#pragma unroll
      for (int ib = 0; ib < kIB; ++ib) {
        const int i = i0 + ib;
        if (i >= n) break;
        double re[kC], im[kC];
        Elem<T>::get(Ws[i * E + t], re, im);
#pragma unroll
        for (int q = 0; q < kC; ++q) sW[q] = fma(re[q], xr[ib][q], fma(im[q], xi[ib][q], sW[q]));
        Elem<T>::get(Ap[static_cast<int64_t>(i) * vstride + e], re, im);
#pragma unroll
        for (int q = 0; q < kC; ++q) sA[q] = fma(re[q], xr[ib][q], fma(im[q], xi[ib][q], sA[q]));
      }
    }
#pragma unroll
    for (int q = 0; q < kC; ++q) {
      accD[q] = fma(aD, sW[q], accD[q]);
      accP[q] = fma(aP, sW[q], accP[q]);
      accA[q] += sA[q];
    }
  }
  // block sums per chain
  __syncthreads();
  double* red = reinterpret_cast<double*>(smraw);  // [3 * kC][E]
#pragma unroll
  for (int q = 0; q < kC; ++q) {
    red[(3 * q) * E + t] = accD[q];
    red[(3 * q + 1) * E + t] = accP[q];
    red[(3 * q + 2) * E + t] = accA[q];
  }
  __syncthreads();
  const int warp = t >> 5, lane = t & 31;
  for (int v = warp; v < 3 * kC; v += E >> 5) {
    double sum = 0.0;
    for (int j = lane; j < E; j += 32) sum += red[v * E + j];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0 && plane * kC + v / 3 < chains) partial[(static_cast<int64_t>(b) * chains + plane * kC + v / 3) * 3 + v % 3] = sum;
  }
}

// out[v] = sum over the blocks of partial[block][v], in order.
__global__ void sum_blocks_kernel(const double* __restrict__ partial, int blocks, int nv, double* __restrict__ out) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  double s = 0.0;
  for (int b = 0; b < blocks; ++b) s += partial[static_cast<int64_t>(b) * nv + v];
  out[v] = s;
}

template <typename T>
cudaError_t launch(const DevSector& S, const T* W, const T* AW, int64_t vstride, int64_t pstride, int chains,
                   const double* Kp, const int* used, int ld, double* partial, double* out, cudaStream_t st) {
  constexpr int kC = Elem<T>::kC;
  const int planes = (chains + kC - 1) / kC, n = ld;
  int dev = 0, sms = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  // widest block whose slice of the n vectors fits in shared memory, not wider than the sector
  int E = 256;
  auto bytes = [&](int e) {
    return std::max(static_cast<size_t>(n) * e * sizeof(T) + static_cast<size_t>(kIB) * n * kC * sizeof(double),
                    static_cast<size_t>(3 * kC) * e * sizeof(double));
  };
  while (E > 32 && (bytes(E) > static_cast<size_t>(optin) || E / 2 >= S.dim)) E /= 2;
  const size_t smem = bytes(E);
  if (n <= 0 || smem > static_cast<size_t>(optin)) return cudaErrorInvalidValue;
  const cudaError_t e = allow_shared(moments_kernel<T>, smem);
  if (e != cudaSuccess) return e;
  const int64_t nch = (S.dim + E - 1) / E;
  const int per_sm = std::max(1, std::min(static_cast<int>(static_cast<size_t>(optin) / smem), 2048 / E));
  const int64_t cap = std::max<int64_t>(1, (static_cast<int64_t>(sms) * per_sm + planes - 1) / planes);
  const int nb = static_cast<int>(std::min<int64_t>({nch, cap, kGradMaxBlocks}));
  moments_kernel<T><<<nb * planes, E, smem, st>>>(S, W, AW, vstride, pstride, Kp, used, chains, ld, nb, partial);
  sum_blocks_kernel<<<(3 * chains + 63) / 64, 64, 0, st>>>(partial, nb, 3 * chains, out);
  return cudaGetLastError();
}

}  // namespace

cudaError_t grad_moments(const DevSector& S, const float4* W, const float4* AW, int64_t vstride, int64_t pstride,
                         int chains, const double* Kp, const int* used, int ld, double* partial, double* out,
                         cudaStream_t st) {
  return launch(S, W, AW, vstride, pstride, chains, Kp, used, ld, partial, out, st);
}

cudaError_t grad_moments(const DevSector& S, const double2* W, const double2* AW, int64_t vstride, int64_t pstride,
                         int chains, const double* Kp, const int* used, int ld, double* partial, double* out,
                         cudaStream_t st) {
  return launch(S, W, AW, vstride, pstride, chains, Kp, used, ld, partial, out, st);
}

}  // namespace ftlm_b200
