// FP64 products whose 64 x 64 output tiles cannot fill the GPU, on small tiles.
//
// The products of a CTMRG move at D <= 5 are of this kind (243 x 37 x 243,
// 512 x 42 x 512, 40 x 40 x 40): on the 64 x 64 tiles of gemm_kernel such a
// product runs on a handful of SMs, and the FP64 pipe of those few SMs (64
// multiply-adds a cycle) bounds it -- a complex 64 x 64 x 243 tile alone takes
// 33 us.  Tiles of 16 to 32 rows and columns spread the same work over the 148
// SMs.  K is cut where gemm() cuts it for the 64 x 64 tiles and every element
// is summed in the same order (k ascending in steps of 4, then the parts in
// turn), so the choice of the tile changes no bit of a result: the randomised
// projectors carry a difference of one rounding to the eighth digit of an
// environment.  Measured, product alone, gemm_kernel -> here: 40 x 40 x 40 8.2
// -> 4.4 us, 512 x 42 x 512 18.5 -> 9.8 us, 82 x 82 x 2592 26.6 -> 16.4 us;
// complex, inside a D = 3, chi = 27 sweep: 21.6 -> 3.9 us on average.  The
// parts of a split product are summed in distributed shared
// memory by a cluster of up to 8 CTAs, in place of a second launch.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "kernels.cuh"

namespace tg {
namespace {

namespace cg = cooperative_groups;

constexpr int TK = 32;      // K of a stage
constexpr int TSTAGES = 3;  // cp.async ring
constexpr int kSMs = 148;

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src, int bytes) {  // the rest is zero-filled
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void add_to(double& a, double b) { a += b; }
__device__ __forceinline__ void add_to(cplx& a, cplx b) {
  a.x += b.x;
  a.y += b.y;
}

template <typename T>
struct TileParams {
  const T* A;
  const T* B;
  T* C;
  GemmDesc d;
  int64_t kchunk;  // K of one part (a multiple of 16)
  int split;       // parts, the cluster's size where `parts` is null
  T* parts;        // split products (split x M x N, row-major) instead of C
  bool pairs_a, pairs_b;
};

// An operand stage keeps the operand's own order, so that its copies are
// contiguous on both sides: k-contiguous operands as [row][KP], the others as
// [k][R + pad].  Both pitches make the fragment reads (8 rows x 4 k) free of
// bank conflicts: KP = 36 (4 mod 16 doubles, 4 mod 8 complex values), rows
// padded to 4 mod 16 doubles or 2 mod 8 complex values.
constexpr int KP = TK + 4;
template <typename T, int R>
struct Stage {
  static constexpr int LD = R + (is_cplx<T>::value ? 2 : (20 - R % 16) % 16);
  static constexpr int size = R * KP > TK * LD ? R * KP : TK * LD;
};

// Copies rows r0 .. r0 + R - 1 and K columns k0 .. k0 + TK - 1 of the operand
// X(r, k) = X[r sr + k sk] into a stage, zeros outside rows x K.  `kc`: sk is
// 1 (else sr is).  `pairs` (real values): two neighbours a copy; the host sets
// it where every pair starts on a 16-byte boundary.
template <typename T, int R>
__device__ __forceinline__ void load_stage(T* dst, const T* X, int64_t sr, int64_t sk, bool kc, bool pairs, int64_t r0,
                                           int64_t rows, int64_t k0, int64_t K) {
  const int tid = threadIdx.x;
  if (sizeof(T) == 8 && pairs) {
#pragma unroll
    for (int i = 0; i < R * TK / 256; ++i) {
      const int idx = tid + i * 128;
      const int r = kc ? idx / (TK / 2) : idx % (R / 2) * 2, k = kc ? idx % (TK / 2) * 2 : idx / (R / 2);
      const int64_t gr = r0 + r, gk = k0 + k;
      const int64_t left = kc ? K - gk : rows - gr;
      const bool ok = gr < rows && gk < K;
      copy_async<16>(dst + (kc ? r * KP + k : k * Stage<T, R>::LD + r), ok ? X + gr * sr + gk * sk : X,
                     ok ? (left > 1 ? 16 : 8) : 0);
    }
  } else {
#pragma unroll
    for (int i = 0; i < R * TK / 128; ++i) {
      const int idx = tid + i * 128;
      const int r = kc ? idx / TK : idx % R, k = kc ? idx % TK : idx / R;
      const int64_t gr = r0 + r, gk = k0 + k;
      const bool ok = gr < rows && gk < K;
      copy_async<sizeof(T)>(dst + (kc ? r * KP + k : k * Stage<T, R>::LD + r), ok ? X + gr * sr + gk * sk : X,
                            ok ? static_cast<int>(sizeof(T)) : 0);
    }
  }
}

template <typename T, int FM, int FN>
struct TileShape {
  static constexpr int BM = 16 * FM, BN = 16 * FN;  // 2 x 2 warps of FM x FN fragments
  static constexpr int SA = Stage<T, BM>::size, STAGE = SA + Stage<T, BN>::size;
  // the output tile takes the stages' place after the last one
  static constexpr size_t bytes = sizeof(T) * static_cast<size_t>(TSTAGES * STAGE);
  static_assert(TSTAGES * STAGE >= BM * BN, "the output tile fits the stages");
};

template <typename T, int FM, int FN>
__global__ void __launch_bounds__(128) tile_gemm_kernel(const __grid_constant__ TileParams<T> p) {
  using S = TileShape<T, FM, FN>;
  constexpr bool CPLX = is_cplx<T>::value;
  constexpr int BM = S::BM, BN = S::BN;
  extern __shared__ __align__(16) unsigned char tile_smem[];
  T* sm = reinterpret_cast<T*>(tile_smem);
  const GemmDesc& d = p.d;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp & 1) * (8 * FM), wn = (warp >> 1) * (8 * FN);
  const int part = blockIdx.z % p.split;
  const int64_t bz = blockIdx.z / p.split;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * BM, n0 = static_cast<int64_t>(blockIdx.x) * BN;
  const int64_t kb = part * p.kchunk;
  const int64_t K = min(d.K - kb, p.kchunk);
  const T* A = p.A + bz * d.bA + kb * d.sAk;
  const T* B = p.B + bz * d.bB + kb * d.sBk;
  const bool a_kc = d.sAk == 1, b_kc = d.sBn != 1;
  const int nk = static_cast<int>((K + TK - 1) / TK);
  // fragment strides of the stages (rows, k)
  const int arow = a_kc ? KP : 1, ak = a_kc ? 1 : Stage<T, BM>::LD;
  const int brow = b_kc ? KP : 1, bk = b_kc ? 1 : Stage<T, BN>::LD;

  auto issue = [&](int kt) {
    if (kt < nk) {
      T* as = sm + (kt % TSTAGES) * S::STAGE;
      load_stage<T, BM>(as, A, d.sAm, d.sAk, a_kc, p.pairs_a, m0, d.M, static_cast<int64_t>(kt) * TK, K);
      load_stage<T, BN>(as + S::SA, B, d.sBn, d.sBk, b_kc, p.pairs_b, n0, d.N, static_cast<int64_t>(kt) * TK, K);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");  // an empty group keeps the count uniform
  };

  double acc_r[FM][FN][2], acc_i[CPLX ? FM : 1][CPLX ? FN : 1][2];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j) {
      acc_r[i][j][0] = acc_r[i][j][1] = 0.0;
      if constexpr (CPLX) acc_i[i][j][0] = acc_i[i][j][1] = 0.0;
    }

#pragma unroll
  for (int s = 0; s < TSTAGES - 1; ++s) issue(s);
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(TSTAGES - 2) : "memory");
    __syncthreads();
    issue(kt + TSTAGES - 1);
    const T* as = sm + (kt % TSTAGES) * S::STAGE;
    const T* bs = as + S::SA;
#pragma unroll
    for (int k4 = 0; k4 < TK; k4 += 4) {
      const int kr = k4 + (lane & 3);
      const T* af = as + (wm + (lane >> 2)) * arow + kr * ak;
      const T* bf = bs + (wn + (lane >> 2)) * brow + kr * bk;
      if constexpr (CPLX) {
        double ar[FM], ai[FM], br[FN], bi[FN];
#pragma unroll
        for (int i = 0; i < FM; ++i) {
          const cplx v = af[i * 8 * arow];
          ar[i] = v.x;
          ai[i] = d.conjA ? -v.y : v.y;
        }
#pragma unroll
        for (int j = 0; j < FN; ++j) {
          const cplx v = bf[j * 8 * brow];
          br[j] = v.x;
          bi[j] = d.conjB ? -v.y : v.y;
        }
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) {
            dmma(acc_r[i][j][0], acc_r[i][j][1], ar[i], br[j]);
            dmma(acc_i[i][j][0], acc_i[i][j][1], ar[i], bi[j]);
          }
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) {
            dmma(acc_r[i][j][0], acc_r[i][j][1], -ai[i], bi[j]);
            dmma(acc_i[i][j][0], acc_i[i][j][1], ai[i], br[j]);
          }
      } else {
        double a[FM], b[FN];
#pragma unroll
        for (int i = 0; i < FM; ++i) a[i] = af[i * 8 * arow];
#pragma unroll
        for (int j = 0; j < FN; ++j) b[j] = bf[j * 8 * brow];
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) dmma(acc_r[i][j][0], acc_r[i][j][1], a[i], b[j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();  // the stages are free

#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = (wm + i * 8 + (lane >> 2)) * BN + wn + j * 8 + 2 * (lane & 3) + h;
        if constexpr (CPLX) sm[e] = make_double2(acc_r[i][j][h], acc_i[i][j][h]);
        else sm[e] = acc_r[i][j][h];
      }
  const bool to_parts = p.parts != nullptr;
  T* C = to_parts ? p.parts + part * d.M * d.N : p.C + bz * d.bC;
  const int64_t sCm = to_parts ? d.N : d.sCm, sCn = to_parts ? 1 : d.sCn;
  const bool cluster = p.split > 1 && !to_parts;
  cg::cluster_group cl = cg::this_cluster();
  if (cluster) cl.sync();
  else __syncthreads();
  const int step = cluster ? 128 * p.split : 128;
  for (int idx = (cluster ? part * 128 : 0) + tid; idx < BM * BN; idx += step) {
    // neighbouring threads write neighbouring elements of C
    const int mm = sCn == 1 ? idx / BN : idx % BM, nn = sCn == 1 ? idx % BN : idx / BM;
    const int64_t gm = m0 + mm, gn = n0 + nn;
    if (gm >= d.M || gn >= d.N) continue;
    T v = sm[mm * BN + nn];
    if (cluster) {
      v = *cl.map_shared_rank(sm + mm * BN + nn, 0);
      for (int r = 1; r < p.split; ++r) add_to(v, *cl.map_shared_rank(sm + mm * BN + nn, r));
    }
    T* c = C + gm * sCm + gn * sCn;
    if (d.accumulate && !to_parts) add_to(v, *c);
    *c = v;
  }
  if (cluster) cl.sync();  // no CTA leaves while its tile is being read
}

template <typename T, int FM, int FN>
void launch_tile(const TileParams<T>& p, cudaStream_t st) {
  using S = TileShape<T, FM, FN>;
  const GemmDesc& d = p.d;
  ensure_dynamic_smem(reinterpret_cast<const void*>(tile_gemm_kernel<T, FM, FN>), S::bytes);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((d.N + S::BN - 1) / S::BN), static_cast<unsigned>((d.M + S::BM - 1) / S::BM),
                     static_cast<unsigned>(d.batch * p.split));
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = S::bytes;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 1;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = p.parts ? 1u : static_cast<unsigned>(p.split);
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  TG_CUDA(cudaLaunchKernelEx(&cfg, tile_gemm_kernel<T, FM, FN>, p));
}

}  // namespace

// Expected cycles of the product on bm x bn tiles: the tiles of one SM in
// turn, each bounded by the FP64 pipe (64 multiply-adds a cycle at best, 4 for
// a complex one; 0.8 of it measured) or by its operands' way from L2 (17 bytes
// a cycle and SM, from 2592 x 2592 x 2592 on 32 x 32 tiles: 2086 us, against
// 1239 us on gemm_kernel's 64 x 64).
double gemm_tile_cycles(const GemmDesc& d, int64_t bm, int64_t bn, int64_t nparts, int64_t kchunk, bool cplx_) {
  const int64_t tiles = (d.M + bm - 1) / bm * ((d.N + bn - 1) / bn) * d.batch * nparts;
  const double kc = static_cast<double>((std::min(kchunk, d.K) + 15) / 16 * 16);
  const double fp = static_cast<double>(bm * bn) * kc * (cplx_ ? 4 : 1) / (0.8 * 64.0);
  const double ld = static_cast<double>(bm + bn) * kc * (cplx_ ? 16 : 8) / 17.0;
  return static_cast<double>((tiles + kSMs - 1) / kSMs) * std::max(fp, ld);
}

template <typename T>
bool gemm_tiles(const T* A, const T* B, T* C, const GemmDesc& d, int64_t nparts, int64_t kchunk, double other_cycles,
                T* parts, cudaStream_t st) {
  static const int shapes[][2] = {{2, 2}, {2, 1}, {1, 2}, {1, 1}};
  int fm = 0, fn = 0;
  double best = other_cycles;
  for (const auto& s : shapes) {
    if ((d.M + 16 * s[0] - 1) / (16 * s[0]) > 65535 || d.batch * nparts > 65535) continue;
    const double c = gemm_tile_cycles(d, 16 * s[0], 16 * s[1], nparts, kchunk, is_cplx<T>::value);
    if (c < best) {
      fm = s[0];
      fn = s[1];
      best = c;
    }
  }
  if (fm == 0) return false;
  TileParams<T> p{A, B, C, d, kchunk, static_cast<int>(nparts), parts, false, false};
  // a unit stride, and every pair of neighbours along it on a 16-byte boundary
  auto pairs = [&](const T* x, int64_t unit, int64_t lead, int64_t batch) {
    return sizeof(T) == 8 && unit == 1 && lead % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
           (d.batch == 1 || batch % 2 == 0);
  };
  p.pairs_a = d.sAk == 1 ? pairs(A, 1, d.sAm, d.bA) : pairs(A, d.sAm, d.sAk, d.bA);
  p.pairs_b = d.sBn == 1 ? pairs(B, 1, d.sBk, d.bB) : pairs(B, d.sBk, d.sBn, d.bB);
  if (fm == 2 && fn == 2) launch_tile<T, 2, 2>(p, st);
  else if (fm == 2) launch_tile<T, 2, 1>(p, st);
  else if (fn == 2) launch_tile<T, 1, 2>(p, st);
  else launch_tile<T, 1, 1>(p, st);
  TG_CHECK_LAUNCH();
  count_launch();
  return true;
}

template bool gemm_tiles<double>(const double*, const double*, double*, const GemmDesc&, int64_t, int64_t, double,
                                 double*, cudaStream_t);
template bool gemm_tiles<cplx>(const cplx*, const cplx*, cplx*, const GemmDesc&, int64_t, int64_t, double, cplx*,
                               cudaStream_t);

}  // namespace tg
