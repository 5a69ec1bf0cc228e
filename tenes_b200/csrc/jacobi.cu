// One-sided Jacobi for matrices that fit one SM's shared memory: the SVD of
// the rSVD / Rayleigh-Ritz cores and the corner spectra.
//
// What bounds it is the chain of a rotation round -- dot product, sum over the
// lanes, rotation angle, update, barrier -- times the rounds of all sweeps, and
// behind it the shared-memory traffic of the columns.  So
// * the matrix kernel keeps the columns of A only.  The right vectors W need
//   the same rotations but none of the dot products, and their rows do not
//   depend on each other: the rotations go to a log in global memory, which
//   jacobi_w_kernel applies to the rows of the identity, four rows a CTA, after
//   the matrix kernel.  (With W beside A a round moved twice the columns.)
// * most rounds pair the columns of two halves, (a_i, b_(i+r) mod h): column
//   a_i stays in its lanes' registers for the whole stage and only b moves
//   (halves, then the halves of the halves; a circle tournament inside the
//   remaining quarters).
// * the angle is computed from single-precision t = tan: the rotation is
//   orthogonal to double precision for any t (c = 1 / sqrt(1 + t^2), s = c t),
//   and an error of 1e-7 in t leaves 1e-7 of the off-diagonal element, below
//   the square of it that the sweep leaves anyway.
// The randomised projectors and what runs beside them take the circle
// tournament over all columns and the double-precision angle instead (kCircle):
// their environments carry a difference of one rounding to the eighth digit,
// so the order of the rotations is part of the result there.  (Complex ones
// stay with jacobi_svd_kernel, which keeps W beside A.)
// Measured, against A and W in one CTA: 96 x 96 real 954 -> 540 us and 174 us
// for W, 82 x 82 in circle order 830 -> 594 and 170 us, 37 x 37 complex 287 ->
// 186 and 62 us; 16 spectra of 72 x 72 corners 3.34 -> 0.48 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>
#include <type_traits>

#include "kernels.cuh"
#include "rotation.cuh"
#include "scaling.cuh"

namespace tg {
namespace {

constexpr int kJacobiSweeps = 60;

// ---- the rotation schedule: every pair of n columns once per sweep
//
// Stage 0: halves [0, h) and [h, n), h rounds.  Stage 1: the halves of each
// half, q0 rounds.  Stage 2: a circle tournament inside each quarter.  pair()
// gives group g's columns in round r of a stage; p is the resident one in the
// first two stages.
struct Schedule {
  int n, h, q0, q1;           // half of n; quarters of the halves
  int m0, m1, m2, m3;         // sizes of the quarters
  int rounds0, rounds1, rounds2, groups;
  __host__ __device__ Schedule(int n_, bool circle_only) : n(n_) {
    if (circle_only) {  // one "quarter" of all columns
      h = q0 = m0 = n;
      q1 = m1 = m2 = m3 = 0;
      rounds0 = rounds1 = 0;
      rounds2 = n > 1 ? n + (n & 1) - 1 : 0;
      groups = (n + 1) / 2;
      return;
    }
    h = (n + 1) / 2;
    q0 = (h + 1) / 2;
    q1 = (n - h + 1) / 2;
    m0 = q0;
    m1 = h - q0;
    m2 = q1;
    m3 = n - h - q1;
    rounds0 = n - h > 0 ? h : 0;
    rounds1 = m1 > 0 ? q0 : 0;
    rounds2 = m0 > 1 ? m0 + (m0 & 1) - 1 : 0;  // m0 is the largest quarter
    const int circle = (m0 + 1) / 2 + (m1 + 1) / 2 + (m2 + 1) / 2 + (m3 + 1) / 2;
    groups = h > q0 + q1 ? h : q0 + q1;
    if (circle > groups) groups = circle;
  }
  __host__ __device__ int rounds() const { return rounds0 + rounds1 + rounds2; }
  __device__ int resident(int stage, int g) const {  // -1: none
    if (stage == 0) return g < h ? g : -1;
    return g < q0 ? g : (g - q0 < q1 ? h + g - q0 : -1);
  }
  // round r < size of stage 0 or 1 pairs group g's resident column with
  // base + (j + r) mod size, where that is below base + count
  __device__ void partners(int stage, int g, int& base, int& size, int& count, int& j) const {
    j = g;
    size = h;
    base = h;
    count = n - h;
    if (stage == 1) {
      if (g < q0) {
        size = q0;
        base = q0;
        count = m1;
      } else {
        j = g - q0;
        size = q1;
        base = h + q1;
        count = m3;
      }
    }
  }
  __device__ bool circle(int g, int r, int& p, int& q) const {
    int base = 0, m = m0, k = g;
    if (k >= (m + 1) / 2) {
      k -= (m + 1) / 2;
      base += m;
      m = m1;
      if (k >= (m + 1) / 2) {
        k -= (m + 1) / 2;
        base += m;
        m = m2;
        if (k >= (m + 1) / 2) {
          k -= (m + 1) / 2;
          base += m;
          m = m3;
          if (k >= (m + 1) / 2) return false;
        }
      }
    }
    const int np = m + (m & 1);  // position 0 fixed, the others rotating
    if (r >= np - 1) return false;
    auto player = [&](int kk) {
      if (kk == 0) return 0;
      const int x = kk - 1 + r;
      return (x >= np - 1 ? x - (np - 1) : x) + 1;
    };
    int a = player(k), b = player(np - 1 - k);
    if (a > b) {
      const int t = a;
      a = b;
      b = t;
    }
    p = base + a;
    q = base + b;
    return b < m;
  }
  // columns of slot g in round r of the whole sweep, false: none
  __device__ bool pair(int g, int r, int& p, int& q) const {
    if (r < rounds0 + rounds1) {
      const int stage = r < rounds0 ? 0 : 1, rr = stage == 0 ? r : r - rounds0;
      int base, size, count, j;
      partners(stage, g, base, size, count, j);
      p = resident(stage, g);
      if (p < 0 || rr >= size) return false;
      j = j + rr >= size ? j + rr - size : j + rr;
      q = base + j;
      return j < count;
    }
    return circle(g, r - rounds0 - rounds1, p, q);
  }
};

template <bool CPLX>
struct Rot;  // a logged rotation: p' = c p - s (ph q), q' = s p + c (ph q)
template <>
struct __align__(16) Rot<false> {
  double c, s;  // s carries no phase; the sign of ph is the sign of c
};
template <>
struct __align__(32) Rot<true> {
  double c, s, phr, phi;
};

__device__ __forceinline__ double re_of(double x) { return x; }
__device__ __forceinline__ double re_of(cplx x) { return x.x; }
__device__ __forceinline__ double im_of(cplx x) { return x.y; }

// rotation_angle in double precision
__device__ __forceinline__ void angle_double(double al, double be, double g, double& t, double& c, double& s) {
  const double tau = be - al;
  const double w = fma(tau, tau, 4.0 * g * g);
  const double den = fabs(tau) + w * rsqrt(w);
  const double rd = rsqrt(den);
  t = copysign(2.0 * g, tau) * (rd * rd);
  c = rsqrt(fma(t, t, 1.0));
  s = c * t;
}
// (p, q) -> (c p - s b, s p + c b) with b = ph q
__device__ __forceinline__ void rotate_pair(double c, double s, double phr, double phi, double& pr, double& pi,
                                            double& qr, double& qi) {
  const double br = qr * phr - qi * phi, bi = qr * phi + qi * phr;
  const double ar = pr, ai = pi;
  pr = c * ar - s * br;
  pi = c * ai - s * bi;
  qr = s * ar + c * br;
  qi = s * ai + c * bi;
}

// sum of |x|^2 over a shared-memory array, whole CTA
__device__ double block_sum(double a) {
  __shared__ double wsum[32];
  __shared__ double total;
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x < 32) {
    double b = (threadIdx.x < (blockDim.x >> 5)) ? wsum[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) b += __shfl_xor_sync(0xffffffffu, b, o);
    if (threadIdx.x == 0) total = b;
  }
  __syncthreads();
  return total;
}

// Rotates the columns of A (n x n, row-major in global memory) to
// orthogonality; LANES lanes hold a column, lane l its rows l + LANES i.
// kSvd, kCircle: column norms descending to S, the normalised columns in that
// order to U, the rotations to `log` (round-major) and {sweeps, position of
// every column} to `info`.  kSpectrum: the norms, divided by their 2-norm,
// descending to S, one matrix a CTA (mats[blockIdx.x]).  Both of kSvd and
// kSpectrum scale a matrix far from 1 by a power of two first: the rotation
// test squares the columns' inner products, the fourth power of the entries.
// WIDE: more columns than the CTA's lanes can hold; a group takes several pairs
// of a circle tournament in turn.
enum JacobiMode { kSpectrum, kSvd, kCircle };
template <bool CPLX, int LANES, int RPL, int MODE, int THREADS, bool WIDE>
__global__ void __launch_bounds__(THREADS)
    jacobi_kernel(const void* A0, const void* const* mats, int n, void* U0, double* S, Rot<CPLX>* log, int* info) {
  using T = typename std::conditional<CPLX, cplx, double>::type;
  constexpr bool VEC = MODE != kSpectrum;
  // columns padded with zeros to the lanes' rows, so that no access needs a
  // guard; the odd pitch keeps the transposing copy from A free of conflicts
  constexpr int LD = LANES * RPL + 1;
  extern __shared__ double jsm[];
  const int nn = n * n;
  double* ar = jsm;
  double* ai = jsm + n * LD;                  // complex only
  double* nrm = jsm + (CPLX ? 2 : 1) * n * LD;  // squared norms
  __shared__ int rotated;
  const T* A = static_cast<const T*>(VEC ? A0 : mats[blockIdx.x]);
  S += VEC ? 0 : static_cast<int64_t>(blockIdx.x) * n;
  const Schedule sch(n, MODE == kCircle || WIDE);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int g = tid / LANES, gl = tid % LANES;

  double total = 0.0;
  int top = 0;
  for (int idx = tid; idx < nn; idx += blockDim.x) {
    const int r = idx / n, c = idx % n;
    const T v = A[idx];
    if constexpr (MODE != kCircle) top = max(top, magnitude(v));
    ar[c * LD + r] = re_of(v);
    total = fma(re_of(v), re_of(v), total);
    if constexpr (CPLX) {
      ai[c * LD + r] = im_of(v);
      total = fma(im_of(v), im_of(v), total);
    }
  }
  for (int idx = tid; idx < n * (LD - n); idx += blockDim.x) {
    const int c = idx / (LD - n), r = n + idx % (LD - n);
    ar[c * LD + r] = 0.0;
    if constexpr (CPLX) ai[c * LD + r] = 0.0;
  }
  __shared__ int warp_top[32];
  if constexpr (MODE != kCircle) {
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0) warp_top[warp] = top;
  }
  total = block_sum(total);  // its barriers also order the stores above
  double unscale = 1.0;
  if constexpr (MODE != kCircle) {
    const double scale = range_scale(__reduce_max_sync(0xffffffffu, lane < nw ? warp_top[lane] : 0), unscale);
    if (scale != 1.0) {  // the same in every thread
      total = 0.0;
      for (int idx = tid; idx < (CPLX ? 2 : 1) * n * LD; idx += blockDim.x) {  // both planes
        ar[idx] *= scale;
        total = fma(ar[idx], ar[idx], total);
      }
      total = block_sum(total);
    }
  }
  const double tol = static_cast<double>(n) * 2.220446049250313e-16, tol2 = tol * tol;
  const double small2 = tol2 * total;  // columns of rounding noise

  auto load = [&](int at, double (&x)[RPL], double (&y)[CPLX ? RPL : 1]) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      x[i] = ar[at + i * LANES];
      if constexpr (CPLX) y[i] = ai[at + i * LANES];
    }
  };
  auto store = [&](int at, const double (&x)[RPL], const double (&y)[CPLX ? RPL : 1]) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      ar[at + i * LANES] = x[i];
      if constexpr (CPLX) ai[at + i * LANES] = y[i];
    }
  };
  // rotates the columns in registers, their squared norms al and be with
  // them; every lane of the warp takes part in the sums
  auto rotate = [&](bool valid, double (&xp)[RPL], double (&yp)[CPLX ? RPL : 1], double (&xq)[RPL],
                    double (&yq)[CPLX ? RPL : 1], double& al, double& be, Rot<CPLX>* out) {
    double gr = 0, gi = 0, gr2 = 0, gi2 = 0;  // two accumulators: shorter FP64 chains
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      double& a = (i & 1) ? gr2 : gr;
      a = fma(xp[i], xq[i], a);
      if constexpr (CPLX) {
        double& b = (i & 1) ? gi2 : gi;
        a = fma(yp[i], yq[i], a);
        b = fma(xp[i], yq[i], b);
        b = fma(-yp[i], xq[i], b);
      }
    }
    gr += gr2;
    gi += gi2;
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      gr += __shfl_xor_sync(0xffffffffu, gr, o, LANES);
      if constexpr (CPLX) gi += __shfl_xor_sync(0xffffffffu, gi, o, LANES);
    }
    bool turn;
    double gabs = 0.0, phr = 1.0, phi = 0.0;
    if constexpr (MODE == kCircle) {
      gabs = fabs(gr);
      turn = valid && !(gabs == 0.0 || al <= small2 || be <= small2 || gabs * gabs <= tol2 * al * be);
    } else {
      gabs = CPLX ? fma(gr, gr, gi * gi) : gr * gr;  // its square here
      turn = valid && gabs > 0.0 && al > small2 && be > small2 && gabs > tol2 * al * be;
    }
    if (turn) {
      if constexpr (!CPLX) {
        gabs = fabs(gr);
        phr = gr >= 0 ? 1.0 : -1.0;
      } else {
        const double inv = rsqrt(gabs);
        gabs *= inv;
        phr = gr * inv;
        phi = -gi * inv;
      }
      double t, c, s;
      if constexpr (MODE == kCircle) angle_double(al, be, gabs, t, c, s);
      else rotation_angle(al, be, gabs, t, c, s);
      al = al - t * gabs;
      be = be + t * gabs;
      const double sph = s * phr, cph = c * phr;  // real: phr = +-1
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        if constexpr (CPLX) {
          rotate_pair(c, s, phr, phi, xp[i], yp[i], xq[i], yq[i]);
        } else {
          const double p = xp[i], q = xq[i];
          xp[i] = c * p - sph * q;
          xq[i] = s * p + cph * q;
        }
      }
      if (gl == 0) {
        rotated = 1;
        if constexpr (VEC) {
          if constexpr (CPLX) *out = Rot<CPLX>{c, s, phr, phi};
          else *out = Rot<CPLX>{phr * c, s};
        }
      }
    } else if (VEC && gl == 0 && valid) {
      if constexpr (CPLX) *out = Rot<CPLX>{1.0, 0.0, 1.0, 0.0};
      else *out = Rot<CPLX>{1.0, 0.0};
    }
    return turn;
  };

  double xp[RPL], xq[RPL], yp[CPLX ? RPL : 1], yq[CPLX ? RPL : 1];
  int sweep = 0;
  for (; sweep < kJacobiSweeps; ++sweep) {
    __syncthreads();
    for (int c = warp; c < n; c += nw) {  // exact norms, updated with each rotation below
      double a = 0;
      for (int r = lane; r < n; r += 32) {
        a = fma(ar[c * LD + r], ar[c * LD + r], a);
        if constexpr (CPLX) a = fma(ai[c * LD + r], ai[c * LD + r], a);
      }
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if (lane == 0) nrm[c] = a;
    }
    if (tid == 0) rotated = 0;
    __syncthreads();
    Rot<CPLX>* out = VEC ? log + static_cast<int64_t>(sweep) * sch.rounds() * sch.groups + g : nullptr;
    if constexpr (MODE != kCircle && !WIDE) {
      for (int stage = 0; stage < 2; ++stage) {
        const int rounds = stage == 0 ? sch.rounds0 : sch.rounds1;
        const int p = sch.resident(stage, g);
        int base, size, count, j;  // round r pairs p with base + (j + r) mod size, if that is below count
        sch.partners(stage, g, base, size, count, j);
        const int at_p = max(p, 0) * LD + gl;
        load(at_p, xp, yp);
        double al = nrm[max(p, 0)];
        int left = p >= 0 ? size : 0;  // a smaller quarter runs out of rounds first
        for (int r = 0; r < rounds; ++r) {
          const bool valid = left > 0 && j < count;
          const int q = valid ? base + j : 0;
          load(q * LD + gl, xq, yq);
          double be = nrm[q];
          if (rotate(valid, xp, yp, xq, yq, al, be, out)) {
            store(q * LD + gl, xq, yq);
            if (gl == 0) nrm[q] = be;
          }
          if (++j == size) j = 0;
          --left;
          if (VEC) out += sch.groups;
          __syncthreads();
        }
        if (p >= 0) {
          store(at_p, xp, yp);
          if (gl == 0) nrm[p] = al;
        }
        __syncthreads();
      }
    }
    for (int r = 0; r < sch.rounds2; ++r) {
      // whole warps stay together in the sums: `first` is the same for all
      for (int first = 0; first < (WIDE ? sch.groups : 1); first += THREADS / LANES) {
        int p = 0, q = 0;
        const bool valid = sch.circle(g + first, r, p, q);
        if (!valid) p = q = 0;
        load(p * LD + gl, xp, yp);
        load(q * LD + gl, xq, yq);
        double al = nrm[p], be = nrm[q];
        if (rotate(valid, xp, yp, xq, yq, al, be, VEC ? out + first : nullptr)) {
          store(p * LD + gl, xp, yp);
          store(q * LD + gl, xq, yq);
          if (gl == 0) {
            nrm[p] = al;
            nrm[q] = be;
          }
        }
      }
      if (VEC) out += sch.groups;
      __syncthreads();
    }
    if (!rotated) break;
  }
  __syncthreads();
  for (int c = warp; c < n; c += nw) {
    double a = 0;
    for (int r = lane; r < n; r += 32) {
      a = fma(ar[c * LD + r], ar[c * LD + r], a);
      if constexpr (CPLX) a = fma(ai[c * LD + r], ai[c * LD + r], a);
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) nrm[c] = sqrt(a);
  }
  __syncthreads();
  double unit = 1.0;
  if constexpr (!VEC) {
    const double v = tid < n ? nrm[tid] : 0.0;
    const double tot = block_sum(v * v);
    unit = tot > 0.0 ? sqrt(tot) : 0.0;
  }
  if (VEC && tid == 0) info[0] = min(sweep, kJacobiSweeps - 1) + 1;  // sweeps in the log
  for (int c = tid; c < n; c += blockDim.x) {
    const double v = nrm[c];
    int pos = 0;
    for (int o = 0; o < n; ++o) {
      const double w = nrm[o];
      pos += (w > v) || (w == v && o < c);
    }
    S[pos] = VEC ? v * unscale : (unit > 0.0 ? v / unit : 0.0);
    if (VEC) info[1 + c] = pos;
  }
  if constexpr (VEC) {
    __syncthreads();  // info is read back by the whole CTA
    T* U = static_cast<T*>(U0);
    for (int idx = tid; idx < nn; idx += blockDim.x) {
      const int r = idx / n, c = idx % n;  // column c -> output column info[1 + c]
      const double inv = nrm[c] > 0.0 ? 1.0 / nrm[c] : 0.0;
      const int64_t o = static_cast<int64_t>(r) * n + info[1 + c];
      if constexpr (CPLX) U[o] = make_double2(ar[c * LD + r] * inv, ai[c * LD + r] * inv);
      else U[o] = ar[c * LD + r] * inv;
    }
  }
}

// W = the product of the logged rotations: a warp carries one row of the
// identity through them, lane l the pairs l, l + 32, ... of a round.  Rotations
// are loaded AHEAD rounds before they are applied, over the latency of L2; the
// schedule is laid out in shared memory first.
constexpr int kWRows = 4;  // rows (warps) a CTA
template <bool CPLX, int SLOTS, int AHEAD>
__global__ void __launch_bounds__(32 * kWRows)
    jacobi_w_kernel(const Rot<CPLX>* __restrict__ log, const int* __restrict__ info, int n, bool circle, void* W0) {
  using T = typename std::conditional<CPLX, cplx, double>::type;
  extern __shared__ __align__(16) unsigned char wsm[];
  T* rows = reinterpret_cast<T*>(wsm);
  unsigned short* pairs = reinterpret_cast<unsigned short*>(rows + kWRows * n);  // p | q << 8, 0: none
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Schedule sch(n, circle);
  const int rounds = sch.rounds(), groups = sch.groups;
  for (int idx = threadIdx.x; idx < rounds * groups; idx += 32 * kWRows) {
    const int r = idx / groups;
    int p, q;
    pairs[idx] = sch.pair(idx - r * groups, r, p, q) ? static_cast<unsigned short>(p | q << 8) : 0;
  }
  const int row = blockIdx.x * kWRows + warp;
  T* w = rows + warp * n;
  for (int c = lane; c < n; c += 32) {
    if constexpr (CPLX) w[c] = make_double2(c == row ? 1.0 : 0.0, 0.0);
    else w[c] = c == row ? 1.0 : 0.0;
  }
  __syncthreads();
  if (row >= n) return;
  const int total = info[0] * rounds;
  Rot<CPLX> ring[AHEAD][SLOTS];
  unsigned pq[AHEAD][SLOTS];
  const Rot<CPLX>* next = log + lane;
  int at = lane, left = rounds;  // where the round to be fetched next starts in `pairs`
  auto fetch = [&](bool more, Rot<CPLX> (&rot)[SLOTS], unsigned (&c)[SLOTS]) {
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      c[k] = 0;
      if (more && lane + 32 * k < groups) {  // an entry without a pair is loaded too (and skipped): no load waits for another
        rot[k] = next[32 * k];
        c[k] = pairs[at + 32 * k];
      }
    }
    next += groups;
    at += groups;
    if (--left == 0) {
      left = rounds;
      at = lane;
    }
  };
  auto apply = [&](const Rot<CPLX> (&rot)[SLOTS], const unsigned (&c)[SLOTS]) {
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) {
      if (c[k] == 0) continue;
      const int p = c[k] & 255, q = c[k] >> 8;
      const double s = rot[k].s;
      if constexpr (CPLX) {
        if (s == 0.0 && rot[k].phr == 1.0) continue;  // not rotated
        T a = w[p], b = w[q];
        rotate_pair(rot[k].c, s, rot[k].phr, rot[k].phi, a.x, a.y, b.x, b.y);
        w[p] = a;
        w[q] = b;
      } else {
        if (s == 0.0 && rot[k].c == 1.0) continue;
        const T a = w[p], b = w[q];
        const double cc = fabs(rot[k].c), sph = copysign(1.0, rot[k].c) * s, cph = rot[k].c;
        w[p] = cc * a - sph * b;
        w[q] = s * a + cph * b;
      }
    }
    __syncwarp();
  };
#pragma unroll
  for (int a = 0; a < AHEAD; ++a) fetch(a < total, ring[a], pq[a]);
  for (int t = 0; t < total; t += AHEAD) {
#pragma unroll
    for (int a = 0; a < AHEAD; ++a) {
      apply(ring[a], pq[a]);
      fetch(t + a + AHEAD < total, ring[a], pq[a]);
    }
  }
  T* W = static_cast<T*>(W0) + static_cast<int64_t>(row) * n;
  for (int c = lane; c < n; c += 32) W[info[1 + c]] = w[c];
}

template <bool CPLX>
void launch_w(const Rot<CPLX>* log, const int* info, int n, bool circle, void* W, cudaStream_t st) {
  const Schedule sch(n, circle);
  const size_t smem = (CPLX ? 16 : 8) * static_cast<size_t>(kWRows * n) +
                      sizeof(unsigned short) * static_cast<size_t>(sch.rounds() * sch.groups);
  auto go = [&](auto kernel) {
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    kernel<<<(n + kWRows - 1) / kWRows, 32 * kWRows, smem, st>>>(log, info, n, circle, W);
  };
  // slots: the groups of a round (at most 60) over the lanes
  if (sch.groups <= 32) go(jacobi_w_kernel<CPLX, 1, 8>);
  else go(jacobi_w_kernel<CPLX, 2, CPLX ? 4 : 6>);
  TG_CHECK_LAUNCH();
  count_launch();
}

// LANES x RPL covers the rows; 16 lanes a column and a group a pair up to 96
// columns (with 8 lanes and 16-byte accesses 48 columns took 145 us against
// 135, 96 columns 556 against 541).  Above, 8 lanes hold a column in 512
// (complex 256) threads, which take the pairs of a round in two or three turns:
// the one form that reaches the 160 columns of a spectrum without spilling.  119
// columns take 2.52 ms so (and spectra of 109 columns 2.42 ms, against 7.29 ms a
// warp a pair); a whole round at once on 16 lanes of 8 rows, up to 119 columns,
// was measured at 1.42 and 1.15 ms and is not built.
constexpr int kMaxResident = 96;
template <bool CPLX, int MODE>
void launch_jacobi(const void* A, const void* const* mats, int count, int n, void* U, double* S, Rot<CPLX>* log,
                   int* info, cudaStream_t st) {
  auto go = [&](auto kernel, int lanes, int rows, int threads) {
    const size_t smem = sizeof(double) * static_cast<size_t>((CPLX ? 2 : 1) * n * (lanes * rows + 1) + n);
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    const int need = (Schedule(n, MODE == kCircle).groups * lanes + 31) / 32 * 32;
    kernel<<<count, threads > 0 ? threads : need, smem, st>>>(A, mats, n, U, S, log, info);
  };
  if (n <= 16) go(jacobi_kernel<CPLX, 16, 1, MODE, 192, false>, 16, 1, 0);
  else if (n <= 32) go(jacobi_kernel<CPLX, 16, 2, MODE, 320, false>, 16, 2, 0);
  else if (n <= 48) go(jacobi_kernel<CPLX, 16, 3, MODE, 448, false>, 16, 3, 0);
  else if (n <= 64) go(jacobi_kernel<CPLX, 16, 4, MODE, 576, false>, 16, 4, 0);
  else if (n <= kMaxResident) go(jacobi_kernel<CPLX, 16, 6, MODE, 800, false>, 16, 6, 0);
  else if constexpr (!CPLX) go(jacobi_kernel<CPLX, 8, 21, MODE, 512, true>, 8, 21, 512);
  else if constexpr (MODE == kSpectrum) go(jacobi_kernel<CPLX, 8, 15, MODE, 256, true>, 8, 15, 256);
  else fail(TG_E_INPUT, "jacobi: n out of range");  // complex SVDs stop at jacobi_svd_max_k
  TG_CHECK_LAUNCH();
  count_launch();
}

}  // namespace

template <typename T>
int jacobi_svd_max_k() {
  return is_cplx<T>::value ? 84 : 119;
}

template <typename T>
void jacobi_svd(const T* A, int64_t k, T* U, double* S, T* W, bool circle, cudaStream_t st) {
  constexpr bool CPLX = is_cplx<T>::value;
  if (k < 1 || k > jacobi_svd_max_k<T>()) fail(TG_E_INPUT, "jacobi_svd: k out of range");
  ProfScope ps(PK_SOLVER, st, (CPLX ? 4.0 : 1.0) * 10.0 * static_cast<double>(k) * k * k, 0.0);
  if constexpr (CPLX) {
    if (circle) {
      jacobi_svd_complex(A, k, U, S, W, st);
      return;
    }
  }
  const int n = static_cast<int>(k);
  const bool tournament = circle || n > kMaxResident;  // as the kernel's
  const Schedule sch(n, tournament);
  const size_t log_bytes = sizeof(Rot<CPLX>) * kJacobiSweeps * static_cast<size_t>(std::max(sch.rounds(), 1) * sch.groups);
  void* buf = nullptr;
  TG_CUDA(cudaMallocAsync(&buf, log_bytes + sizeof(int) * static_cast<size_t>(n + 1), st));
  auto* log = static_cast<Rot<CPLX>*>(buf);
  int* info = reinterpret_cast<int*>(static_cast<unsigned char*>(buf) + log_bytes);
  if constexpr (!CPLX) {
    if (circle) launch_jacobi<CPLX, kCircle>(A, nullptr, 1, n, U, S, log, info, st);
  }
  if (!circle) launch_jacobi<CPLX, kSvd>(A, nullptr, 1, n, U, S, log, info, st);
  launch_w<CPLX>(log, info, n, tournament, W, st);
  TG_CUDA(cudaFreeAsync(buf, st));
}

template <typename T>
void batched_spectrum(const T* const* mats, int count, int n, double* out, cudaStream_t st) {
  if (count <= 0) return;
  constexpr bool CPLX = is_cplx<T>::value;
  // the matrix lives in shared memory: n <= 160 (real), 112 (complex)
  const int nmax = CPLX ? 112 : 160;
  if (n > nmax || n < 1)
    fail(TG_E_INPUT, "batched_spectrum: 1 <= chi <= " + std::to_string(nmax) + " required");
  ProfScope ps(PK_SPECTRUM, st, 0.0, sizeof(T) * static_cast<double>(count) * n * n);
  launch_jacobi<CPLX, kSpectrum>(nullptr, reinterpret_cast<const void* const*>(mats), count, n, nullptr, out, nullptr,
                             nullptr, st);
}

#define TG_INST(T)                                                                       \
  template int jacobi_svd_max_k<T>();                                                    \
  template void jacobi_svd<T>(const T*, int64_t, T*, double*, T*, bool, cudaStream_t);         \
  template void batched_spectrum<T>(const T* const*, int, int, double*, cudaStream_t);
TG_INST(double)
TG_INST(cplx)
#undef TG_INST

}  // namespace tg
