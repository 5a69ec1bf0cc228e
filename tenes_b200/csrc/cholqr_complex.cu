// Orthonormalisation of a tall complex FP64 panel by shifted CholeskyQR, every
// pass in one launch of one thread-block cluster: the phases of cholqr.cu
// (Gram partials, a fixed-order sum over the cluster, the Cholesky factor on
// CTA 0, a blocked triangular solve of each CTA's rows) with real and imaginary
// planes in shared memory and four real DMMAs a complex product.
//
// The form it replaces in the exact truncated SVD (a Gram product, a sum, a
// one-CTA factor with its inverse, a product back) takes about 60 us a pass at
// 243 x 43, 47 of them in the one CTA; here the factor's multiply-adds run on
// DMMA and the solve needs no inverse: 70 us a call of two to four passes (26 us
// a pass), and a 2 x 2, D = 3, chi = 27 complex environment went from 119 to 75
// ms.  What is left is the chain of pivots on CTA 0 and four cluster barriers a
// pass.  The randomised projectors keep the other form: their results carry its
// roundings.  A warp's Gram blocks are sized for k <= 48 and k <= 88 apart (75
// -> 71 us), and the sum over the cluster reads four CTAs at a time (all
// sixteen in flight: 87 us).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "counter_rng.cuh"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace tg {
namespace {

constexpr int ZQ_THREADS = 256;
constexpr int ZQ_WARPS = ZQ_THREADS / 32;
constexpr int ZQ_KPMAX = 88;  // k rounded up to 8: two kp x ld and two kp x LDY planes fill 215 of the 227 KB
constexpr int ZQ_RB = 48;     // rows of Y staged per chunk
constexpr int ZQ_LDY = ZQ_RB + 4;  // 4 (mod 16): conflict-free fragment loads
// upper 8 x 8 blocks a warp holds for k <= 48 and for k <= 88
constexpr int ZQ_SLOTS48 = (6 * 7 / 2 + ZQ_WARPS - 1) / ZQ_WARPS;
constexpr int ZQ_SLOTS88 = (11 * 12 / 2 + ZQ_WARPS - 1) / ZQ_WARPS;

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
// accumulator fragment of an 8 x 8 block -> the A fragments of its k-steps 0, 1
__device__ __forceinline__ void acc_to_a(const double (&c)[2], int lane, double& f0, double& f1) {
  const int src = (lane & ~3) + ((lane & 3) >> 1);
  const double v0 = __shfl_sync(0xffffffffu, c[0], src), v1 = __shfl_sync(0xffffffffu, c[1], src);
  const double w0 = __shfl_sync(0xffffffffu, c[0], src + 2), w1 = __shfl_sync(0xffffffffu, c[1], src + 2);
  f0 = (lane & 1) ? v1 : v0;
  f1 = (lane & 1) ? w1 : w0;
}
__host__ __device__ inline int row_pitch(int kp) { return kp + ((20 - (kp & 15)) & 15); }  // 4 (mod 16)

// Upper Cholesky factor of the kp x kp Hermitian matrix (Ar, Ai) in place (upper
// triangle), as cholesky_blocked in cholqr.cu: A = R^H R, the diagonal blocks
// replaced by their inverses at the end.
__device__ void cholesky(double* Ar, double* Ai, int kp, int ld, double* dinv, const int* btab, int* flag) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = kp / 8, nblk = nb * (nb + 1) / 2;
  const int g = lane >> 2, t = lane & 3;
  for (int J = 0; J < nb; ++J) {
    const int j0 = 8 * J, ncol = kp - j0 - 8;
    double ar[8][8], ai[8][8];
    if (warp == 0 || warp * 32 < ncol) {
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = r; c < 8; ++c) {
          ar[r][c] = Ar[(j0 + r) * ld + j0 + c];
          ai[r][c] = c > r ? Ai[(j0 + r) * ld + j0 + c] : 0.0;
        }
      const int col = j0 + 8 + warp * 32 + lane;
      const bool has = warp * 32 + lane < ncol;
      double pr[8], pi[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        pr[r] = has ? Ar[(j0 + r) * ld + col] : 0.0;
        pi[r] = has ? Ai[(j0 + r) * ld + col] : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        double piv = ar[j][j];
        if (!(piv > 0.0)) {
          if (tid == 0 && flag) atomicExch(flag, 1);
          piv = 1.0;
        }
        const double inv = rsqrt(piv);
        if (tid == 0) dinv[j0 + j] = inv;
        ar[j][j] = piv * inv;
#pragma unroll
        for (int c = j + 1; c < 8; ++c) {
          ar[j][c] *= inv;
          ai[j][c] *= inv;
        }
        pr[j] *= inv;
        pi[j] *= inv;
#pragma unroll
        for (int r = j + 1; r < 8; ++r) {  // row r -= conj(R(j, r)) row j
#pragma unroll
          for (int c = r; c < 8; ++c) {
            ar[r][c] -= ar[j][r] * ar[j][c] + ai[j][r] * ai[j][c];
            if (c > r) ai[r][c] -= ar[j][r] * ai[j][c] - ai[j][r] * ar[j][c];
          }
          pr[r] -= ar[j][r] * pr[j] + ai[j][r] * pi[j];
          pi[r] -= ar[j][r] * pi[j] - ai[j][r] * pr[j];
        }
      }
      if (has) {  // each block-row column is read and written by its owner lane only
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          Ar[(j0 + r) * ld + col] = pr[r];
          Ai[(j0 + r) * ld + col] = pi[r];
        }
      }
    }
    __syncthreads();  // every warp has loaded the diagonal block
    if (warp == 0 && lane < 8) {  // lane c writes column c of R_JJ (no trailing block touches it)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c == lane) {
#pragma unroll
          for (int r = 0; r <= c; ++r) {
            Ar[(j0 + r) * ld + j0 + c] = ar[r][c];
            Ai[(j0 + r) * ld + j0 + c] = ai[r][c];
          }
        }
    }
    // trailing blocks (K, L), J < K <= L: A_KL -= R_JK^H R_JL
    for (int b = (J + 1) * nb - J * (J + 1) / 2 + warp; b < nblk; b += ZQ_WARPS) {
      const int bb = btab[b], K = bb >> 8, L = bb & 255;
      const int at = (8 * K + g) * ld + 8 * L + 2 * t;
      double cr[2] = {Ar[at], Ar[at + 1]}, ci[2] = {Ai[at], Ai[at + 1]};
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const int row = (j0 + 4 * ks + t) * ld + g;
        const double kr = Ar[row + 8 * K], ki = Ai[row + 8 * K], lr = Ar[row + 8 * L], li = Ai[row + 8 * L];
        dmma(cr, -kr, lr);
        dmma(ci, -kr, li);
        dmma(cr, -ki, li);
        dmma(ci, ki, lr);
      }
      Ar[at] = cr[0];
      Ar[at + 1] = cr[1];
      Ai[at] = ci[0];
      Ai[at + 1] = ci[1];
    }
    __syncthreads();
  }
  // diagonal blocks -> their inverses: warp J, lane c solves R_JJ x = e_c
  for (int J = warp; J < nb; J += ZQ_WARPS) {
    const int j0 = 8 * J, c = lane & 7;
    double xr[8], xi[8];
#pragma unroll
    for (int r = 7; r >= 0; --r) {
      double sr = (r == c) ? 1.0 : 0.0, si = 0.0;
#pragma unroll
      for (int m = r + 1; m < 8; ++m)
        if (m <= c) {
          const double br = Ar[(j0 + r) * ld + j0 + m], bi = Ai[(j0 + r) * ld + j0 + m];
          sr -= br * xr[m] - bi * xi[m];
          si -= br * xi[m] + bi * xr[m];
        }
      xr[r] = (r <= c) ? sr * dinv[j0 + r] : 0.0;
      xi[r] = (r <= c) ? si * dinv[j0 + r] : 0.0;
    }
    __syncwarp();
    if (lane < 8) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        Ar[(j0 + r) * ld + j0 + c] = xr[r];
        Ai[(j0 + r) * ld + j0 + c] = xi[r];
      }
    }
  }
  __syncthreads();
}

template <int ZQ_SLOTS>
__global__ void __launch_bounds__(ZQ_THREADS, 1)
    cholqr_complex_kernel(cplx* Y, double* scratch, int n, int k, int passes, int shifted, double shift,
                          double noise_scale, unsigned long long key_re, unsigned long long key_im, int* flag) {
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank()), cs = static_cast<int>(cluster.num_blocks());
  extern __shared__ __align__(16) double zq_smem[];
  const int kp = (k + 7) & ~7, nb = kp >> 3, ld = row_pitch(kp), plane = kp * ld;
  double* Ur = zq_smem;  // rows of Y / X, column by column
  double* Ui = Ur + kp * ZQ_LDY;
  double* Rr = Ui + kp * ZQ_LDY;  // Gram partial, reduced slice, then R with inverted diagonal blocks
  double* Ri = Rr + plane;
  double* ds = Ri + plane;  // equilibration D
  double* dinv = ds + kp;   // 1 / R_ii
  int* btab = reinterpret_cast<int*>(dinv + kp);  // (bi << 8) | bj of the upper 8 x 8 blocks
  const int nblk = nb * (nb + 1) / 2, total = nblk * 64;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    int q = 0;
    for (int bi = 0; bi < nb; ++bi)
      for (int bj = bi; bj < nb; ++bj) btab[q++] = (bi << 8) | bj;
  }
  auto entry = [&](int e) {  // element e of the upper blocks -> offset in a plane
    const int b = btab[e >> 6], w = e & 63;
    return ((b >> 8) * 8 + (w >> 3)) * ld + (b & 255) * 8 + (w & 7);
  };
  // a lane's two entries of block b
  auto pair_at = [&](int b) {
    const int bb = btab[b];
    return ((bb >> 8) * 8 + g) * ld + (bb & 255) * 8 + 2 * t;
  };
  const int rows_per = ((n + cs - 1) / cs + 7) & ~7;
  const int r0 = min(n, rank * rows_per), r1 = min(n, r0 + rows_per);
  const int nch = (r1 - r0 + ZQ_RB - 1) / ZQ_RB;
  const bool resident = nch <= 1;  // the rows stay in shared memory across passes
  const int per = (total + cs - 1) / cs;
  auto stage = [&](int rc, int nr) {  // rows [rc, rc + nr), zero-padded to 8 rows and kp columns
    const int nr8 = (nr + 7) & ~7;
#pragma unroll 4
    for (int idx = tid; idx < kp * nr8; idx += ZQ_THREADS) {
      const int c = idx / nr8, r = idx - c * nr8;
      const cplx v = (r < nr && c < k) ? Y[static_cast<size_t>(c) * n + rc + r] : make_double2(0.0, 0.0);
      Ur[c * ZQ_LDY + r] = v.x;
      Ui[c * ZQ_LDY + r] = v.y;
    }
    __syncthreads();
  };
  auto unstage = [&](int rc, int nr) {
    for (int idx = tid; idx < k * nr; idx += ZQ_THREADS) {
      const int c = idx / nr, r = idx - c * nr;
      Y[static_cast<size_t>(c) * n + rc + r] = make_double2(Ur[c * ZQ_LDY + r], Ui[c * ZQ_LDY + r]);
    }
  };
  __syncthreads();
  if (nch == 1) stage(r0, r1 - r0);

  for (int pass = 0; pass < passes; ++pass) {
    // ---- 1. Gram partial Y^H Y of rows [r0, r1)
    double cr[ZQ_SLOTS][2], ci[ZQ_SLOTS][2];
#pragma unroll
    for (int s = 0; s < ZQ_SLOTS; ++s) cr[s][0] = cr[s][1] = ci[s][0] = ci[s][1] = 0.0;
    for (int ch = 0; ch < nch; ++ch) {
      const int rc = r0 + ch * ZQ_RB, nr = min(ZQ_RB, r1 - rc), nr8 = (nr + 7) & ~7;
      if (!resident) stage(rc, nr);
      for (int r = 0; r < nr8; r += 4) {
#pragma unroll
        for (int s = 0; s < ZQ_SLOTS; ++s) {
          const int b = warp + s * ZQ_WARPS;
          if (b < nblk) {
            const int bb = btab[b];
            const int oa = ((bb >> 8) * 8 + g) * ZQ_LDY + t + r, ob = ((bb & 255) * 8 + g) * ZQ_LDY + t + r;
            const double xr = Ur[oa], xi = Ui[oa], yr = Ur[ob], yi = Ui[ob];
            dmma(cr[s], xr, yr);
            dmma(ci[s], xr, yi);
            dmma(cr[s], xi, yi);
            dmma(ci[s], -xi, yr);
          }
        }
      }
      if (!resident) __syncthreads();  // before the next chunk is staged
    }
    // the previous pass's factor is read by the others until here
    if (pass > 0) cluster.sync();
#pragma unroll
    for (int s = 0; s < ZQ_SLOTS; ++s) {
      const int b = warp + s * ZQ_WARPS;
      if (b < nblk) {
        const int at = pair_at(b);
        Rr[at] = cr[s][0];
        Rr[at + 1] = cr[s][1];
        Ri[at] = ci[s][0];
        Ri[at + 1] = ci[s][1];
      }
    }
    cluster.sync();
    // ---- 2. sum this CTA's slice of the entries over the cluster, in rank order
    for (int e = rank * per + tid; e < min(total, (rank + 1) * per); e += ZQ_THREADS) {
      const int off = entry(e);
      double vr = 0.0, vi = 0.0;
#pragma unroll 4
      for (int q = 0; q < 16; ++q)
        if (q < cs) {
          vr += cluster.map_shared_rank(Rr, q)[off];
          vi += cluster.map_shared_rank(Ri, q)[off];
        }
      Rr[off] = vr;
      Ri[off] = vi;
    }
    cluster.sync();
    // ---- 3. CTA 0: gather, equilibrate, shift, factor
    if (rank == 0) {
      for (int e = tid; e < total; e += ZQ_THREADS) {
        const int owner = e / per;
        if (owner != 0) {
          const int off = entry(e);
          Rr[off] = cluster.map_shared_rank(Rr, owner)[off];
          Ri[off] = cluster.map_shared_rank(Ri, owner)[off];
        }
      }
      __syncthreads();
      for (int i = tid; i < kp; i += ZQ_THREADS) {
        if (i >= k) Rr[i * ld + i] = 1.0;  // padding columns: identity
        const double d = Rr[i * ld + i];
        ds[i] = (i < k && d > 0.0) ? 1.0 / sqrt(d) : 1.0;
      }
      __syncthreads();
      for (int b = warp; b < nblk; b += ZQ_WARPS) {
        const int bb = btab[b], at = pair_at(b), r = (bb >> 8) * 8 + g;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = (bb & 255) * 8 + 2 * t + h;
          if (r < k && c < k) {
            const double w = ds[r] * ds[c];
            Rr[at + h] = Rr[at + h] * w + ((r == c && pass < shifted) ? shift : 0.0);
            Ri[at + h] *= w;
          }
        }
      }
      __syncthreads();
      cholesky(Rr, Ri, kp, ld, dinv, btab, flag);
      // R and D to the global scratch, read from L2 by the other CTAs
      for (int b = warp; b < nblk; b += ZQ_WARPS) {
        const int at = pair_at(b);
        *reinterpret_cast<double2*>(scratch + at) = *reinterpret_cast<const double2*>(Rr + at);
        *reinterpret_cast<double2*>(scratch + plane + at) = *reinterpret_cast<const double2*>(Ri + at);
      }
      for (int i = tid; i < kp; i += ZQ_THREADS) scratch[2 * plane + i] = ds[i];
      __threadfence();
    }
    cluster.sync();
    // ---- 4. R and D from the scratch (L2 only: the lines change every pass)
    if (rank != 0) {
#pragma unroll 3
      for (int b = warp; b < nblk; b += ZQ_WARPS) {
        const int at = pair_at(b);
        *reinterpret_cast<double2*>(Rr + at) = __ldcg(reinterpret_cast<const double2*>(scratch + at));
        *reinterpret_cast<double2*>(Ri + at) = __ldcg(reinterpret_cast<const double2*>(scratch + plane + at));
      }
      for (int i = tid; i < kp; i += ZQ_THREADS) ds[i] = __ldcg(scratch + 2 * plane + i);
      __syncthreads();
    }
    // ---- 5. X R = Y D on 8-row blocks, X written over the rows in U
    const bool noisy = pass == 0 && noise_scale != 0.0;
    for (int ch = 0; ch < nch; ++ch) {
      const int rc = r0 + ch * ZQ_RB, nr = min(ZQ_RB, r1 - rc), nr8 = (nr + 7) & ~7;
      if (!resident) stage(rc, nr);
      for (int rb = warp; rb < nr8 / 8; rb += ZQ_WARPS) {
        const int row = rb * 8 + g;
#pragma unroll 1
        for (int J = 0; J < nb; ++J) {
          const int c0 = 8 * J + 2 * t;
          double ar[2] = {Ur[c0 * ZQ_LDY + row] * ds[c0], Ur[(c0 + 1) * ZQ_LDY + row] * ds[c0 + 1]};
          double ai[2] = {Ui[c0 * ZQ_LDY + row] * ds[c0], Ui[(c0 + 1) * ZQ_LDY + row] * ds[c0 + 1]};
          double br[2] = {0.0, 0.0}, bi[2] = {0.0, 0.0};  // the second products: two shorter chains
#pragma unroll 2
          for (int I = 0; I < 2 * J; ++I) {  // 4 columns of X a step
            const int kc = 4 * I + t, at = kc * ld + 8 * J + g;
            const double xr = Ur[kc * ZQ_LDY + row], xi = Ui[kc * ZQ_LDY + row], rr = Rr[at], ri = Ri[at];
            dmma(ar, -xr, rr);
            dmma(ai, -xr, ri);
            dmma(br, xi, ri);
            dmma(bi, -xi, rr);
          }
          ar[0] += br[0];
          ar[1] += br[1];
          ai[0] += bi[0];
          ai[1] += bi[1];
          double fr0, fr1, fi0, fi1;
          acc_to_a(ar, lane, fr0, fr1);
          acc_to_a(ai, lane, fi0, fi1);
          const int at0 = (8 * J + t) * ld + 8 * J + g, at1 = (8 * J + 4 + t) * ld + 8 * J + g;
          const double dr0 = Rr[at0], di0 = Ri[at0], dr1 = Rr[at1], di1 = Ri[at1];
          double xr[2] = {0.0, 0.0}, xi[2] = {0.0, 0.0};
          dmma(xr, fr0, dr0);
          dmma(xi, fr0, di0);
          dmma(xr, -fi0, di0);
          dmma(xi, fi0, dr0);
          dmma(xr, fr1, dr1);
          dmma(xi, fr1, di1);
          dmma(xr, -fi1, di1);
          dmma(xi, fi1, dr1);
          Ur[c0 * ZQ_LDY + row] = xr[0];
          Ur[(c0 + 1) * ZQ_LDY + row] = xr[1];
          Ui[c0 * ZQ_LDY + row] = xi[0];
          Ui[(c0 + 1) * ZQ_LDY + row] = xi[1];
          __syncwarp();  // X_J visible to the warp's later fragment loads
        }
      }
      if (noisy) {  // after the solve, which needs the unperturbed X
        __syncthreads();
        for (int idx = tid; idx < k * nr; idx += ZQ_THREADS) {
          const int c = idx / nr, r = idx - c * nr;
          const uint64_t at = static_cast<uint64_t>(c) * n + rc + r;
          Ur[c * ZQ_LDY + r] += noise_scale * counter_unit_uniform(at, key_re);
          Ui[c * ZQ_LDY + r] += noise_scale * counter_unit_uniform(at, key_im);
        }
      }
      __syncthreads();
      if (!resident || pass == passes - 1) {
        unstage(rc, nr);
        if (!resident) __syncthreads();
      }
    }
  }
  cluster.sync();  // no CTA leaves while its shared memory may be read
}

size_t smem_bytes(int kp) {
  const int nb = kp / 8;
  return sizeof(double) * (2 * (static_cast<size_t>(kp) * ZQ_LDY + static_cast<size_t>(kp) * row_pitch(kp)) + 2 * kp) +
         sizeof(int) * static_cast<size_t>(nb * (nb + 1) / 2);
}

using Kernel = decltype(&cholqr_complex_kernel<ZQ_SLOTS88>);

cudaLaunchConfig_t config(int cs, size_t smem, cudaStream_t st, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(cs));
  cfg.blockDim = dim3(ZQ_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = static_cast<unsigned>(cs);
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// cluster size the current device runs the kernel with (16, else 8, else 0), kept per device
int cluster_size() {
  static std::mutex mu;
  static int size[kMaxDevices];
  static bool probed[kMaxDevices] = {};
  const int dev = current_device();
  std::lock_guard<std::mutex> guard(mu);
  if (!probed[dev]) {
    probed[dev] = true;
    size[dev] = 0;
    const size_t smem = smem_bytes(ZQ_KPMAX);
    const Kernel kernels[2] = {cholqr_complex_kernel<ZQ_SLOTS48>, cholqr_complex_kernel<ZQ_SLOTS88>};
    bool ok = true;
    for (Kernel f : kernels) {
      ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) ==
                     cudaSuccess;
      cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    }
    for (int c : {16, 8}) {
      cudaLaunchAttribute at;
      const cudaLaunchConfig_t cfg = config(c, smem, nullptr, &at);
      int n0 = 0, n1 = 0;
      if (ok && cudaOccupancyMaxActiveClusters(&n0, kernels[0], &cfg) == cudaSuccess && n0 > 0 &&
          cudaOccupancyMaxActiveClusters(&n1, kernels[1], &cfg) == cudaSuccess && n1 > 0) {
        size[dev] = c;
        break;
      }
    }
    cudaGetLastError();
  }
  return size[dev];
}

}  // namespace

bool cholqr_complex_supported(int64_t n, int64_t k) {
  return k >= 1 && k <= ZQ_KPMAX && n >= 1 && n * k < (int64_t(1) << 31) && cluster_size() > 0;
}

int64_t cholqr_complex_scratch_doubles(int64_t k) {
  const int kp = static_cast<int>((k + 7) / 8 * 8);
  return 2 * static_cast<int64_t>(kp) * row_pitch(kp) + kp;
}

void cholqr_complex(cplx* Y, int64_t n, int64_t k, int passes, int shifted_passes, uint64_t noise_stream,
                    double noise_scale, double* scratch, int* flag, cudaStream_t st) {
  if (!cholqr_complex_supported(n, k)) fail(TG_E_INPUT, "cholqr_complex: unsupported panel shape");
  // shifted CholeskyQR (Fukaya et al., SIAM J. Sci. Comput. 42 (2020) A477):
  // s = 11 (m n + n (n+1)) u ||X||_2^2 with ||X||_2^2 <= k for unit columns
  const double u = 1.1102230246251565e-16;
  const double s = 11.0 * (static_cast<double>(n) * k + static_cast<double>(k) * (k + 1)) * u * k;
  ProfScope ps(PK_SOLVER, st, 4.0 * passes * (2.0 * static_cast<double>(n) * k * k + k * k * k / 3.0), 0.0);
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t cfg = config(cluster_size(), smem_bytes(static_cast<int>((k + 7) / 8 * 8)), st, &at);
  TG_CUDA(cudaLaunchKernelEx(&cfg, k <= 48 ? cholqr_complex_kernel<ZQ_SLOTS48> : cholqr_complex_kernel<ZQ_SLOTS88>, Y, scratch, static_cast<int>(n), static_cast<int>(k), passes,
                             shifted_passes, s, noise_scale, static_cast<unsigned long long>(noise_key_re(noise_stream)),
                             static_cast<unsigned long long>(noise_key_im(noise_stream)), flag));
  count_launch();
}

}  // namespace tg
