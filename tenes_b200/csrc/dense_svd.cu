// Dense SVD of matrices whose shared-memory image fits one SM: a Householder QR
// of the matrix with its columns sorted by norm, then the one-sided Jacobi of
// R^H (jacobi.cu) -- the preconditioning of Drmac & Veselic, SIAM J. Matrix
// Anal. Appl. 29 (2008) 1322.  On the graded projector matrices of a CTMRG move
// the Jacobi of R^H needs 8 sweeps, that of the matrix itself 19 (40 x 40,
// D = 2, chi = 10).  cuSOLVER's gesvd, which these matrices took before, is a
// chain of about 900 launches there (3 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"
#include "scaling.cuh"

namespace tg {
namespace {

constexpr int kQrThreads = 512;
constexpr size_t kSmemMax = 227 * 1024;
// a column of a smaller norm (squared) is lifted before its reflector is made:
// its squares lose digits, and the reflector would not be unitary
constexpr double kTinyNorm2 = 1e-240;
constexpr double kLift = 3.273390607896142e150, kUnlift = 3.054936363499605e-151;  // 2^500, 2^-500

__device__ __forceinline__ double conj_of(double x) { return x; }
__device__ __forceinline__ cplx conj_of(cplx x) { return make_double2(x.x, -x.y); }
__device__ __forceinline__ double abs2(double x) { return x * x; }
__device__ __forceinline__ double abs2(cplx x) { return fma(x.x, x.x, x.y * x.y); }
__device__ __forceinline__ double real_of(double x) { return x; }
__device__ __forceinline__ double real_of(cplx x) { return x.x; }
__device__ __forceinline__ double imag_of(double) { return 0.0; }
__device__ __forceinline__ double imag_of(cplx x) { return x.y; }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ double times(double a, double b) { return a * b; }
__device__ __forceinline__ cplx times(cplx a, double b) { return make_double2(a.x * b, a.y * b); }
__device__ __forceinline__ cplx mul(cplx a, cplx b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double sub(double a, double b) { return a - b; }
__device__ __forceinline__ cplx sub(cplx a, cplx b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double fma_conj(double a, double b, double c) { return fma(a, b, c); }  // conj(a) b + c
__device__ __forceinline__ cplx fma_conj(cplx a, cplx b, cplx c) {
  return make_double2(fma(a.y, b.y, fma(a.x, b.x, c.x)), fma(-a.y, b.x, fma(a.x, b.y, c.y)));
}
template <typename T>
__device__ __forceinline__ T make(double re, double im) {
  if constexpr (is_cplx<T>::value) return make_double2(re, im);
  else return re;
}
__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ cplx warp_sum(cplx v) { return make_double2(warp_sum(v.x), warp_sum(v.y)); }

// A (m x k, m >= k; element (r, c) = M[r * sr + c * sc], conjugated when
// `conj`) = Q R P^T, the columns taken in the order of descending norm:
// reflectors H_j = 1 - tau_j v_j v_j^H with v_j(j) = 1 to V (row j = v_j, zeros
// before j) and tau, Q = H_0 H_1 ...; R^H (k x k, row-major) to L; perm[c] = the
// column of A at place c.  One CTA, the matrix in shared memory; every warp
// holds the reflector of a step in registers (computed by each warp for itself,
// so a step has one barrier) and applies it to its share of the columns.
// *info is set to 1 when the matrix holds a value that is not finite.  A matrix
// far from unit scale is factored times a power of two, which L takes out again.
template <typename T, int RPL>
__global__ void __launch_bounds__(kQrThreads)
    sorted_qr_kernel(const T* __restrict__ M, int64_t sr, int64_t sc, bool conj, int m, int k, T* __restrict__ V,
                     T* __restrict__ tau, T* __restrict__ L, int* __restrict__ perm, int* info) {
  extern __shared__ __align__(16) unsigned char qsm[];
  const int ld = m | 1;
  T* a = reinterpret_cast<T*>(qsm);                          // column-major, pitch ld
  double* nrm = reinterpret_cast<double*>(a + static_cast<size_t>(ld) * k);
  int* at = reinterpret_cast<int*>(nrm + k);                 // place c holds column at[c]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  int* warp_top = reinterpret_cast<int*>(nrm);  // (static shared memory would not fit beside the largest matrices)
  int top = 0;
  for (int idx = tid; idx < m * k; idx += blockDim.x) {
    const int r = sc == 1 ? idx / k : idx % m, c = sc == 1 ? idx % k : idx / m;
    const T v = M[r * sr + c * sc];
    top = max(top, magnitude(v));
    a[c * ld + r] = conj ? conj_of(v) : v;
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) warp_top[warp] = top;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, lane < nw ? warp_top[lane] : 0);
  double unscale;
  const double range = range_scale(top, unscale);
  if (range != 1.0)  // the same in every thread
    for (int idx = tid; idx < ld * k; idx += blockDim.x)
      if (idx % ld < m) a[idx] = times(a[idx], range);
  __syncthreads();  // also before warp_top's place takes the norms
  if (tid == 0 && top >= 0x7ff00000 && info) atomicExch(info, 1);
  for (int c = warp; c < k; c += nw) {
    double s = 0.0;
    for (int r = lane; r < m; r += 32) s += abs2(a[c * ld + r]);
    s = warp_sum(s);
    if (lane == 0) {
      nrm[c] = s;
      at[c] = c;
    }
  }
  __syncthreads();
  for (int c = tid; c < k; c += blockDim.x) {
    const double v = nrm[c];
    int pos = 0;
    for (int o = 0; o < k; ++o) pos += nrm[o] > v || (!(nrm[o] < v) && o < c);
    at[min(pos, k - 1)] = c;
  }
  __syncthreads();
  for (int c = tid; c < k; c += blockDim.x) perm[c] = at[c];
  for (int j = 0; j < k; ++j) {
    const T* x = a + at[j] * ld;
    T v[RPL];
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int r = lane + 32 * i;
      v[i] = r > j && r < m ? x[r] : make<T>(0.0, 0.0);
      s += abs2(v[i]);
    }
    s = warp_sum(s);
    T alpha = x[j];
    double unlift = unscale;
    if (fma(real_of(alpha), real_of(alpha), fma(imag_of(alpha), imag_of(alpha), s)) < kTinyNorm2) {
      bool some = imag_of(alpha) != 0.0;
#pragma unroll
      for (int i = 0; i < RPL; ++i) some = some || magnitude(v[i]) != 0;
      if (__any_sync(0xffffffffu, some)) {  // not for the zero columns of a padded matrix
        s = 0.0;
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
          v[i] = times(v[i], kLift);
          s += abs2(v[i]);
        }
        s = warp_sum(s);
        alpha = times(alpha, kLift);
        unlift *= kUnlift;
        if (fma(real_of(alpha), real_of(alpha), fma(imag_of(alpha), imag_of(alpha), s)) < kTinyNorm2) {
          // nothing against the matrix, 1e-240 of it: no reflector
          s = 0.0;
          alpha = make<T>(real_of(alpha), 0.0);
        }
      }
    }
    const double ar = real_of(alpha), ai = imag_of(alpha);
    double beta = ar;
    T t = make<T>(0.0, 0.0);
    if (s > 0.0 || ai != 0.0) {
      beta = -copysign(sqrt(fma(ar, ar, fma(ai, ai, s))), ar);
      t = make<T>((beta - ar) / beta, -ai / beta);
      // 1 / (alpha - beta)
      const double dr = ar - beta, inv = 1.0 / fma(dr, dr, ai * ai);
      const T scale = make<T>(dr * inv, -ai * inv);
#pragma unroll
      for (int i = 0; i < RPL; ++i) v[i] = mul(scale, v[i]);
    }
#pragma unroll
    for (int i = 0; i < RPL; ++i)
      if (lane + 32 * i == j) v[i] = make<T>(1.0, 0.0);
    if (warp == 0) {
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        const int r = lane + 32 * i;
        if (r < m) V[static_cast<int64_t>(j) * m + r] = v[i];
      }
      if (lane == 0) tau[j] = t;
    }
    // L = R^H: row c, column j <= c holds conj(R(j, c))
    if (tid < j) L[static_cast<int64_t>(tid) * k + j] = make<T>(0.0, 0.0);
    if (tid == j) L[static_cast<int64_t>(j) * k + j] = make<T>(beta * unlift, 0.0);
    const T tc = conj_of(t);
    for (int c = j + 1 + warp; c < k; c += nw) {
      T* y = a + at[c] * ld;
      T z[RPL], d = make<T>(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        const int r = lane + 32 * i;
        z[i] = r >= j && r < m ? y[r] : make<T>(0.0, 0.0);
        d = fma_conj(v[i], z[i], d);
      }
      d = mul(tc, warp_sum(d));
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        const int r = lane + 32 * i;
        if (r >= j && r < m) {
          const T u = sub(z[i], mul(v[i], d));
          y[r] = u;
          if (r == j) L[static_cast<int64_t>(c) * k + j] = times(conj_of(u), unscale);
        }
      }
    }
    __syncthreads();
  }
}

// Singular vectors of A from the Jacobi of L = R^H, L W = U S: column i of Q W
// (left, m long) to left[r * lsr + i * lsi], and column i of P U (right, k long)
// to right[c * rsc + i * rsi], each conjugated where asked.  A warp a column;
// reflectors are applied from the last to the first.
template <typename T, int RPL>
__global__ void __launch_bounds__(128)
    apply_q_kernel(const T* __restrict__ V, const T* __restrict__ tau, const int* __restrict__ perm,
                   const T* __restrict__ W, const T* __restrict__ U, int m, int k, T* __restrict__ left, int64_t lsr,
                   int64_t lsi, bool conj_left, T* __restrict__ right, int64_t rsc, int64_t rsi, bool conj_right) {
  const int lane = threadIdx.x & 31, i = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (i >= k) return;
  T x[RPL], next[RPL];
#pragma unroll
  for (int q = 0; q < RPL; ++q) {
    const int r = lane + 32 * q;
    x[q] = r < k ? W[static_cast<int64_t>(r) * k + i] : make<T>(0.0, 0.0);
    next[q] = r < m ? V[static_cast<int64_t>(k - 1) * m + r] : make<T>(0.0, 0.0);
  }
  for (int j = k - 1; j >= 0; --j) {
    T v[RPL], d = make<T>(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < RPL; ++q) {
      v[q] = next[q];
      const int r = lane + 32 * q;
      if (j > 0 && r < m) next[q] = V[static_cast<int64_t>(j - 1) * m + r];
      d = fma_conj(v[q], x[q], d);
    }
    d = mul(tau[j], warp_sum(d));
#pragma unroll
    for (int q = 0; q < RPL; ++q) x[q] = sub(x[q], mul(v[q], d));
  }
#pragma unroll
  for (int q = 0; q < RPL; ++q) {
    const int r = lane + 32 * q;
    if (r < m) left[r * lsr + i * lsi] = conj_left ? conj_of(x[q]) : x[q];
  }
  for (int c = lane; c < k; c += 32) {
    const T u = U[static_cast<int64_t>(c) * k + i];
    right[perm[c] * rsc + i * rsi] = conj_right ? conj_of(u) : u;
  }
}

template <typename T>
size_t qr_smem(int64_t m, int64_t k) {
  // the norms' place also holds a value of every warp
  return sizeof(T) * static_cast<size_t>((m | 1) * k) +
         std::max((sizeof(double) + sizeof(int)) * static_cast<size_t>(k), sizeof(int) * (kQrThreads / 32));
}

}  // namespace

template <typename T>
bool dense_svd_supported(int64_t nrow, int64_t ncol) {
  const int64_t m = std::max(nrow, ncol), k = std::min(nrow, ncol);
  return k >= 1 && k <= jacobi_svd_max_k<T>() && m <= 256 && qr_smem<T>(m, k) <= kSmemMax;
}

template <typename T>
void dense_svd(const T* M, int64_t nrow, int64_t ncol, T* U, double* S, T* VT, int* info, cudaStream_t st) {
  if (!dense_svd_supported<T>(nrow, ncol)) fail(TG_E_INPUT, "dense_svd: unsupported shape");
  const bool tall = nrow >= ncol;  // A = M, else A = M^H
  const int m = static_cast<int>(std::max(nrow, ncol)), k = static_cast<int>(std::min(nrow, ncol));
  const int64_t kk = static_cast<int64_t>(k) * k;
  void* buf = nullptr;
  TG_CUDA(cudaMallocAsync(&buf, sizeof(T) * static_cast<size_t>(static_cast<int64_t>(k) * m + k + 3 * kk) + sizeof(int) * k, st));
  T* V = static_cast<T*>(buf);
  T* tau = V + static_cast<int64_t>(k) * m;
  T* L = tau + k;
  T* Uj = L + kk;
  T* Wj = Uj + kk;
  int* perm = reinterpret_cast<int*>(Wj + kk);
  const size_t smem = qr_smem<T>(m, k);
  auto go = [&](auto qr, auto apply) {
    {
      ProfScope ps(PK_SOLVER, st, (is_cplx<T>::value ? 4.0 : 1.0) * 2.0 * m * k * k, 0.0);
      ensure_dynamic_smem(reinterpret_cast<const void*>(qr), smem);
      qr<<<1, kQrThreads, smem, st>>>(M, tall ? ncol : 1, tall ? 1 : ncol, !tall, m, k, V, tau, L, perm, info);
      TG_CHECK_LAUNCH();
    }
    jacobi_svd<T>(L, k, Uj, S, Wj, false, st);
    // tall: M = (Q W) S (P U)^H; else M = (P U) S (Q W)^H.  U (nrow x k), VT (k x ncol), row-major.
    apply<<<(k + 3) / 4, 128, 0, st>>>(V, tau, perm, Wj, Uj, m, k, tall ? U : VT, tall ? k : 1, tall ? 1 : ncol, !tall,
                                       tall ? VT : U, tall ? 1 : k, tall ? ncol : 1, tall);
    TG_CHECK_LAUNCH();
    count_launch(2);
  };
  if (m <= 32) go(sorted_qr_kernel<T, 1>, apply_q_kernel<T, 1>);
  else if (m <= 64) go(sorted_qr_kernel<T, 2>, apply_q_kernel<T, 2>);
  else if (m <= 128) go(sorted_qr_kernel<T, 4>, apply_q_kernel<T, 4>);
  else go(sorted_qr_kernel<T, 8>, apply_q_kernel<T, 8>);
  TG_CUDA(cudaFreeAsync(buf, st));
}

#define TG_INST(T)                                       \
  template bool dense_svd_supported<T>(int64_t, int64_t); \
  template void dense_svd<T>(const T*, int64_t, int64_t, T*, double*, T*, int*, cudaStream_t);
TG_INST(double)
TG_INST(cplx)
#undef TG_INST

}  // namespace tg
