// ggem_pair.cu -- Kernel B: the local regularized-Stokeslet pair sums.
//
// u_i = sum_j G(r_ij) f_j + self term, with G the local regularized Green's
// tensor of GGEMStokes::green_tensor_local_regularized (ggem_stokes.C:304-357)
// summed as GGEMStokes::local_solution_bead (ggem_stokes.C:427-503) and the
// self term of PMSystemStokes::compute_point_velocity (pm_system_stokes.C:446-455).
//
// Two arithmetic paths:
//  * FP64: groups of lanes walk the target's row of the pair list, minimum
//    image and tensor (piecewise quintics in r^2) in FP64; without a list one
//    thread per target slot sweeps the neighbour cells of the stencil.
//  * FP32: groups of kGroup lanes share one target and walk its cached CSR
//    pair list (consecutive entries, so the gathered sources of a group sit
//    in the same cells).  The displacement is formed from cell-relative
//    coordinates plus the stencil shift (exact cell offsets);
//    G = A(s) I + B(s) x x^T with A, B = e^{-alpha^2 s} times a polynomial
//    in s (or a cubic table when that fit is not accurate enough); each lane
//    keeps Kahan-compensated FP32 sums; the group reduces them as float-float
//    values in FP32 and forms one FP64 add per output component.
// Algorithmic work per in-cutoff ordered pair: 28 + 19*nrhs flops (FMA = 2,
// rsqrt/exp/erf = 1 each), bound by the FP32 pipe.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "ggem_ff.cuh"
#include "ggem_internal.cuh"

namespace ggem {
namespace {

__device__ __forceinline__ int wrap_i(int k, int n) {
  k %= n;
  return k < 0 ? k + n : k;
}

__device__ __forceinline__ void min_image(const Grid &g, double d[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (g.periodic[k]) {
      const double xs = g.L[k];
      if (d[k] <= -xs / 2.0) d[k] += xs;
      if (d[k] > xs / 2.0) d[k] -= xs;
    }
  }
}

__device__ __forceinline__ void self_term(const DevConsts &K, int self_mode, const double f[3],
                                          double u[3]) {
  if (self_mode == GGEM_SELF_BEAD) {
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = (u[a] - K.coeff_1 * f[a]) + f[a];
  } else if (self_mode == GGEM_SELF_LAGRANGIAN) {
#pragma unroll
    for (int a = 0; a < 3; ++a) u[a] = u[a] + K.coeff_2 * f[a];
  }
}

// Minimum image (pm_periodic_boundary.C:350-374: d <= -L/2 adds L, d > L/2
// subtracts it) with the comparisons on the bit patterns: an FP64 comparison
// costs as much of the FP64 pipe as an addition, an integer one nothing of
// it.  half: the bits of L/2, or of infinity on an open axis; wrapped
// positions keep |d| < L, so one shift suffices.
struct MinImage {
  long long half[3], L[3];
};

__device__ __forceinline__ bool past_half(double d, long long half) {
  const long long b = __double_as_longlong(d);
  return (b & 0x7fffffffffffffffll) + (b < 0 ? 1 : 0) > half;
}

// +L for a negative d, -L for a positive one
__device__ __forceinline__ double shift_image(double d, long long L) {
  const long long sign = __double_as_longlong(d) & (long long)0x8000000000000000ull;
  return d + __longlong_as_double(L | (sign ^ (long long)0x8000000000000000ull));
}

// The three axes of a pair.  The additions are behind a branch of the warp's
// active lanes: away from the box faces (81% of the targets at N = 200k, phi
// = 0.1) no lane takes them, which is 3 of a pair's 33 FP64 instructions.
__device__ __forceinline__ void min_image3(const MinImage &mi, double &x, double &y, double &z) {
  const bool ox = past_half(x, mi.half[0]), oy = past_half(y, mi.half[1]),
             oz = past_half(z, mi.half[2]);
  if (__any_sync(__activemask(), ox || oy || oz)) {
    if (ox) x = shift_image(x, mi.L[0]);
    if (oy) y = shift_image(y, mi.L[1]);
    if (oz) z = shift_image(z, mi.L[2]);
  }
}

// one 256-bit read-only load of what an earlier kernel wrote: volatile and
// with a memory clobber, so that it stays behind wait_prior_grid
__device__ __forceinline__ double4_32a ld_f64x4(const double4_32a *p) {
  double4_32a v;
  asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// the same of the tensor's pieces, written once before any product: the
// compiler may move it anywhere
__device__ __forceinline__ double4_32a ld_piece(const double4_32a *p) {
  double4_32a v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
      : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
      : "l"(p));
  return v;
}

// The FP64 tensor of a pair (Tensor64): ten fused multiply-adds and one
// subtraction on the FP64 pipe, against ~230 instructions for a square root,
// two divisions, two erf and two exp.  eps2: the bits of r_eps^2, below
// which the tensor is coeff_2 I (ggem_stokes.C:304-357).
__device__ __forceinline__ void tensor64(const Tensor64 &T, double s, long long eps2,
                                         double coeff_2, double &A, double &B) {
  const int hi = __double2hiint(s);
  const int idx = min(max((hi >> (20 - kTab64Sub)) - T.base, 0), T.last);
  const double4_32a *r = T.rec + 3 * idx;
  const double4_32a r2 = ld_piece(r + 2), r1 = ld_piece(r + 1), r0 = ld_piece(r);
  constexpr int low = (1 << (20 - kTab64Sub)) - 1;
  const double mid = __hiloint2double((hi & ~low) | ((low + 1) >> 1), 0);
  const double t = s - (idx == 0 ? T.mid0 : mid);
  A = fma(r2.z, t, r2.x);
  B = fma(r2.w, t, r2.y);
  A = fma(A, t, r1.z);
  B = fma(B, t, r1.w);
  A = fma(A, t, r1.x);
  B = fma(B, t, r1.y);
  A = fma(A, t, r0.z);
  B = fma(B, t, r0.w);
  A = fma(A, t, r0.x);
  B = fma(B, t, r0.y);
  const bool close = __double_as_longlong(s) < eps2;
  A = close ? coeff_2 : A;
  B = close ? 0.0 : B;
}

// A(s) (as a sum A + Al) and B(s) for the fit: the alternating series where
// ksi^2 s is small (the closed form cancels there), its constant term, nearly
// all of A, in twofold precision; otherwise the closed form with the
// difference of the two erf as a difference of erfc (both small at large r)
__device__ void tensor_ab64(const DevConsts &c, double s, double &A, double &Al, double &B) {
  const double k = c.one_eight_pi_mu, ksi2 = c.ksi * c.ksi;
  if (ksi2 * s < 0.25) {
    double sp = 0.0, sm = 0.0, kp = c.ksi, ap = c.alpha, w = 1.0, wm = 1.0 / s;
#pragma unroll
    for (int n = 0; n < 16; ++n) {  // 0.25^16 / 16! is far below 2^-53
      const double d = kp - ap;
      if (n > 0) {
        sp += d * w * (1.0 / (2.0 * n + 1.0) + 1.0);
        sm += d * wm * (1.0 / (2.0 * n + 1.0) - 1.0);
      }
      kp *= ksi2;
      ap *= c.alpha2;
      w *= -s * (1.0 / (n + 1.0));
      wm = n == 0 ? -1.0 : wm * (-s * (1.0 / (n + 1.0)));
    }
    // 2 / sqrt(pi) k = m + ml, ksi - alpha = d + dl, their doubled product p + pl
    constexpr double t = 1.1283791670955126, tl = 1.533545961316588e-17;
    const double m = __dmul_rn(k, t), ml = fma(k, t, -m) + k * tl;
    const double d = __dadd_rn(c.ksi, -c.alpha), g = __dadd_rn(d, -c.ksi);
    const double dl = (c.ksi - __dadd_rn(d, -g)) + (-c.alpha - g);
    const double p = 2.0 * __dmul_rn(m, d), pl = 2.0 * (fma(m, d, -0.5 * p) + (m * dl + ml * d));
    const double x = __dmul_rn(m, sp);
    A = __dadd_rn(p, x);
    const double y = __dadd_rn(A, -p);
    Al = ((p - __dadd_rn(A, -y)) + (x - y)) + (pl + ml * sp);
    B = m * sm;
    return;
  }
  const double r = sqrt(s);
  const double kr = c.ksi * r, ar = c.alpha * r;
  const double c1 = (ar > 0.5 ? erfc(ar) - erfc(kr) : erf(kr) - erf(ar)) / r;
  const double c2 = c.two_ksi_sqrt_pi * exp(-ksi2 * s) - c.two_alpha_sqrt_pi * exp(-c.alpha2 * s);
  A = k * (c1 + c2);
  Al = 0.0;
  B = k * (c1 - c2) / s;
}

// Chebyshev interpolants at 12 points of every piece, cut at degree 5 (the
// oversampling averages the rounding of the samples).  The first piece ends
// where ksi^2 s = 2^-6 at most; with 2^7 pieces per octave above it the
// dropped terms stay below 2e-17 of A(0): the functions vary on the scale
// 1 / alpha^2 and 1 / ksi^2 of s and, beyond it, algebraically.  The sums run
// over the samples' differences from the piece's first one, which is added
// last: the constants are then good to half an ulp (A of isolated pairs at r =
// 1e-5 .. 1 rc against 40 digits, rms over A(0): 9.4e-17 at alpha = 0.5, ksi =
// 0.59 and 3.5e-17 at alpha = 0.1; erf and exp per pair 3.3e-16 and 7.1e-17;
// sums over the samples themselves 3.2e-16 and 1.7e-16).  One thread per sample,
// then one per coefficient, behind the rest of a context's set-up; the host
// took 0.8 ms for the 1360 pieces of alpha = 0.5, rc = 7.
constexpr int kFitPoints = 12, kFitPieces = 8;

struct FitBasis {
  double node[kFitPoints], w[kTab64Deg + 1][kFitPoints];
};

__global__ void __launch_bounds__(kFitPoints *kFitPieces) k_fit_tensor64(
    int np, double s0, DevConsts c, const __grid_constant__ FitBasis b,
    double4_32a *__restrict__ rec) {
  constexpr int M = kFitPoints, D = kTab64Deg;
  static_assert(D == 5 && 2 * (D + 1) == M, "record layout");
  __shared__ double v[kFitPieces][2][M];   // samples less the first one
  __shared__ double ref[kFitPieces][2];
  __shared__ double ch[kFitPieces][2][M];  // Chebyshev coefficients
  const int p = threadIdx.x / M, j = threadIdx.x % M;
  const int i = blockIdx.x * kFitPieces + p;
  const int sub = 1 << kTab64Sub;
  double mid = 0.5 * s0, half = mid;
  if (i > 0) {
    const double lo = ldexp(s0, (i - 1) / sub);
    half = 0.5 * lo / sub;
    mid = lo + (2 * ((i - 1) % sub) + 1) * half;
  }
  double A, Al, B;
  tensor_ab64(c, mid + half * b.node[j], A, Al, B);
  if (j == 0) {
    ref[p][0] = A;
    ref[p][1] = B;
  }
  __syncthreads();
  v[p][0][j] = (A - ref[p][0]) + Al;
  v[p][1][j] = B - ref[p][1];
  __syncthreads();
  const int w = j / (D + 1), q = j % (D + 1);  // A or B, degree
  double a = 0.0;
  for (int m = 0; m < M; ++m) a = fma(v[p][w][m], b.w[q][m], a);
  ch[p][w][q] = a;
  __syncthreads();
  // T_0 .. T_5 as monomials, smallest contributions first
  const double *t = ch[p][w];
  double m = q == 0   ? ref[p][w] + ((t[4] - t[2]) + t[0])
             : q == 1 ? (5.0 * t[5] - 3.0 * t[3]) + t[1]
             : q == 2 ? -8.0 * t[4] + 2.0 * t[2]
             : q == 3 ? -20.0 * t[5] + 4.0 * t[3]
             : q == 4 ? 8.0 * t[4]
                      : 16.0 * t[5];
  for (int n = 0; n < q; ++n) m /= half;
  if (i < np) reinterpret_cast<double *>(rec + 3 * (size_t)i)[2 * q + w] = m;
}

// FP64 plain sweep.  own_first: reference mode (own cell, then the element
// stencil that excludes (0,0,0), no cut-off); otherwise the cut-off stencil.
// Runs where there is no pair list (ggem_set_fp64_pair_list(0), no room for
// one, or a first application under stream capture).
template <int NR>
__global__ void __launch_bounds__(128) k_matvec_f64(int64_t n, Grid g, DevConsts K, Tensor64 T,
                                                    const int4 *__restrict__ stencil, int nst,
                                                    int own_first, int use_cutoff, double rc2,
                                                    long long eps2,
                                                    const int32_t *__restrict__ start,
                                                    const double4_32a *__restrict__ pos64,
                                                    const float4 *__restrict__ pos32,
                                                    const double *__restrict__ f,
                                                    double *__restrict__ u, int self_mode,
                                                    int r0) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const double4_32a pi = pos64[s];
  const int32_t cid = __float_as_int(pos32[s].w);
  const int cx = cid % g.nc[0], cy = (cid / g.nc[0]) % g.nc[1], cz = cid / (g.nc[0] * g.nc[1]);
  double acc[NR][3];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r][0] = acc[r][1] = acc[r][2] = 0.0;
  const int64_t vstride = 3 * n;
  for (int k = own_first ? -1 : 0; k < nst; ++k) {
    int4 o = (k < 0) ? make_int4(0, 0, 0, 0) : stencil[k];
    int c[3] = {cx + o.x, cy + o.y, cz + o.z};
    bool ok = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (c[d] < 0 || c[d] >= g.nc[d]) {
        if (!g.periodic[d]) ok = false;
        else c[d] = wrap_i(c[d], g.nc[d]);
      }
    }
    if (!ok) continue;
    const int32_t nc = c[0] + g.nc[0] * (c[1] + g.nc[1] * c[2]);
    const int32_t b = start[nc], e = start[nc + 1];
    for (int32_t t = b; t < e; ++t) {
      if (t == s) continue;
      const double4_32a pj = pos64[t];
      double x[3] = {pj.x - pi.x, pj.y - pi.y, pj.z - pi.z};
      min_image(g, x);
      if (use_cutoff) {
        const double r2c = __dadd_rn(__dadd_rn(__dmul_rn(x[0], x[0]), __dmul_rn(x[1], x[1])),
                                     __dmul_rn(x[2], x[2]));
        if (!(r2c < rc2)) continue;
      }
      double A, B;
      tensor64(T, fma(x[2], x[2], fma(x[1], x[1], x[0] * x[0])), eps2, K.coeff_2, A, B);
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const double *fj = f + (int64_t)(r0 + q) * vstride + 3 * (int64_t)t;
        const double f0 = fj[0], f1 = fj[1], f2 = fj[2];
        const double xf = B * fma(x[2], f2, fma(x[1], f1, x[0] * f0));
        acc[q][0] = fma(A, f0, fma(xf, x[0], acc[q][0]));
        acc[q][1] = fma(A, f1, fma(xf, x[1], acc[q][1]));
        acc[q][2] = fma(A, f2, fma(xf, x[2], acc[q][2]));
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const double *fi = f + (int64_t)(r0 + q) * vstride + 3 * s;
    const double fv[3] = {fi[0], fi[1], fi[2]};
    self_term(K, self_mode, fv, acc[q]);
    double *ui = u + (int64_t)(r0 + q) * vstride + 3 * s;
    ui[0] = acc[q][0];
    ui[1] = acc[q][1];
    ui[2] = acc[q][2];
  }
}

// the row of one target: G lanes take every G-th entry and add their sums by
// shuffles (every lane holds the totals).  NC: f is constant during the
// kernel (read-only loads); otherwise it is read through L2.
template <int NR, int G, bool NC>
__device__ __forceinline__ void pair_row_f64(int sub, int m, const uint32_t *__restrict__ row,
                                             const double4_32a &pi, const MinImage &mi,
                                             const DevConsts &K, const Tensor64 &T,
                                             long long eps2,
                                             const double4_32a *__restrict__ pos64,
                                             const double *f, int64_t vstride,
                                             double acc[NR][3]) {
#pragma unroll
  for (int q = 0; q < NR; ++q) acc[q][0] = acc[q][1] = acc[q][2] = 0.0;
  uint32_t nxt = sub < m ? __ldg(row + sub) : 0u;
  for (int k = sub; k < m; k += G) {
    const int64_t t = (int64_t)(nxt >> kCodeBits);
    if (k + G < m) nxt = __ldg(row + k + G);
    const double4_32a pj = ld_f64x4(pos64 + t);
    double x = pj.x - pi.x, y = pj.y - pi.y, z = pj.z - pi.z;
    min_image3(mi, x, y, z);
    double A, B;
    tensor64(T, fma(z, z, fma(y, y, x * x)), eps2, K.coeff_2, A, B);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const double *fj = f + q * vstride + 3 * t;
      const double f0 = NC ? __ldg(fj) : __ldcg(fj), f1 = NC ? __ldg(fj + 1) : __ldcg(fj + 1),
                   f2 = NC ? __ldg(fj + 2) : __ldcg(fj + 2);
      const double xf = B * fma(z, f2, fma(y, f1, x * f0));
      acc[q][0] = fma(A, f0, fma(xf, x, acc[q][0]));
      acc[q][1] = fma(A, f1, fma(xf, y, acc[q][1]));
      acc[q][2] = fma(A, f2, fma(xf, z, acc[q][2]));
    }
  }
#pragma unroll
  for (int o = 1; o < G; o <<= 1)
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int a = 0; a < 3; ++a) acc[q][a] += __shfl_xor_sync(0xffffffffu, acc[q][a], o);
}

// The targets of a block of 256 threads (G lanes each) in order of row
// length, so that the targets of a warp end together: returns the target of
// this thread's group, its length in m (past the last target: -1, length 0).
// Each target's own sum is formed as in slot order.  In slot order a warp's
// eight rows at G = 4 walk 10.0 entries per lane where 8.5 would do (N = 200k,
// phi = 0.1), in order of length among the block's 64 rows 9.1.
template <int G>
__device__ __forceinline__ int64_t block_target_by_length(int64_t n, const int32_t *__restrict__ cnt,
                                                          int &m) {
  constexpr int T = 256 / G;  // targets per block
  if constexpr (G == 32) {  // one target per warp
    const int64_t s = blockIdx.x * (int64_t)T + threadIdx.x / G;
    m = s < n ? cnt[s] : 0;
    return s < n ? s : -1;
  }
  __shared__ int s_len[T];
  __shared__ int s_tgt[T];
  const int64_t s0 = blockIdx.x * (int64_t)T;
  const int t = threadIdx.x / G, sub = threadIdx.x % G;
  const int mine = s0 + t < n ? cnt[s0 + t] : -1;
  if (sub == 0) s_len[t] = mine;
  __syncthreads();
  int rank = 0;  // longer rows before this one, and equal ones of smaller slots
#pragma unroll
  for (int k = 0; k < T; k += G) {  // (T is a multiple of G up to G = 16)
    const int o = s_len[k + sub];
    rank += o > mine || (o == mine && k + sub < t);
  }
#pragma unroll
  for (int o = 1; o < G; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  if (sub == 0) s_tgt[rank] = t;
  __syncthreads();
  const int tgt = s_tgt[t];
  m = max(s_len[tgt], 0);
  return s_len[tgt] < 0 ? -1 : s0 + tgt;
}

// FP64 pair sum over the pair list (cut-off lists and element lists alike):
// minimum image of the wrapped FP64 positions (pm_periodic_boundary.C:350-374)
// and green_tensor_local_regularized (ggem_stokes.C:304-357) as its piecewise
// quintic; the tensor's two coefficients are formed once per pair and applied
// to NR right-hand sides.  G lanes per target take every G-th entry of its
// row and add their sums by shuffles.
//
// Bound by the FP64 pipe (two lanes per SM and clock): 27 FP64 instructions
// per pair and right-hand side pass (3 displacement, 3 r^2, 11 tensor, 10
// product; 3 more where a warp's pairs cross a box face), which is 0.29 ms at
// N = 200k, phi = 0.1 (6.74 M pairs).
// Measured there: 0.42 ms; 0.45 ms with the box-face additions for every
// pair, 0.50 ms also with the targets in slot order (lanes idle at the ends
// of uneven rows), 2.85 ms also with erf and exp per pair; the cell
// sweep takes 4.8 ms, 15.0 ms with erf and exp.  u is closer to 34 digits
// than with the formula, which cancels (N = 500, norm-wise): 3.0e-16 against
// 5.5e-16 at alpha = 0.5, 1.1e-16 against 2.2e-16 at 0.1.
template <int NR, int G>
__global__ void __launch_bounds__(256) k_pair_list_f64(int64_t n, MinImage mi, DevConsts K,
                                                       Tensor64 T, long long eps2,
                                                       const int32_t *__restrict__ cnt, int W,
                                                       const uint32_t *__restrict__ list,
                                                       const double4_32a *__restrict__ pos64,
                                                       const double *__restrict__ f,
                                                       double *__restrict__ u, int self_mode,
                                                       int r0) {
  wait_prior_grid();
  const int sub = (int)(threadIdx.x % G);
  int m;
  const int64_t tgt = block_target_by_length<G>(n, cnt, m);
  const bool act = tgt >= 0;
  const int64_t s = act ? tgt : n - 1;
  const double4_32a pi = ld_f64x4(pos64 + s);
  const int64_t vstride = 3 * n;
  double acc[NR][3];
  pair_row_f64<NR, G, true>(sub, m, list + s * (int64_t)W, pi, mi, K, T, eps2,
                            pos64, f + (int64_t)r0 * vstride, vstride, acc);
  if (!act || sub != 0) return;
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const double *fi = f + (int64_t)(r0 + q) * vstride + 3 * s;
    const double fv[3] = {fi[0], fi[1], fi[2]};
    self_term(K, self_mode, fv, acc[q]);
    double *ui = u + (int64_t)(r0 + q) * vstride + 3 * s;
    ui[0] = acc[q][0];
    ui[1] = acc[q][1];
    ui[2] = acc[q][2];
  }
}

// ---- the FP64 Chebyshev series of one right-hand side in one launch --------
// The loop of brownian_system.C:1036-1155 as one cooperative kernel.  Phase i
// applies M to x_i and, where the degree-i sum dw_i is to be checked, to dw_i
// in the same row walk (the tensors are formed once for both): the products
// give the check of dw_i and, ahead of its decision, x_{i+1} and dw_{i+1}.  A
// grid barrier ends the phase; its last block adds the estimator partials in
// a fixed order and decides, so the host neither launches nor waits per term
// (one product is in vain when the series stops).  Vectors travel as 32-byte
// records through L2 and rotate, so that a phase writes only buffers that no
// block reads in it.  G lanes walk a target's row; a reduce-scatter leaves
// each of the six sums (and its component of the vectors) on one lane.
//
// CACHE > 0: the first CACHE entries of every lane keep their tensor (six
// FP64 values) in registers over all phases, which leaves one gather and 18
// FP64 instructions per pair and phase instead of a list, a position and a
// tensor gather and 40.  It takes every target resident in one round.
//
// Bound: at small counts the barriers and one L2 gather per phase (~7 us a
// phase at N = 1000), at large ones the FP64 pipe.  us per series, single
// launches with host checks -> one launch: N = 1000 (7 terms) 431 -> 119,
// 6000 698 -> 315, 20k 1779 -> 1291, 200k 10476 -> 9075.
//
// Waits are bounded (polls): a block that gives up sets the error word and
// leaves, and so do the others.
struct SeriesCtl {
  unsigned int arrive, release;
  int stop, err;
  int n_terms, n_matvecs, converged, first_check;
  double err1, err2, aux2, n0, n1;  // n0 = |dw_{i-1}|^2, n1 = |x_i|^2 of the sum to be checked
};

struct SeriesF64 {
  int64_t n;
  int W, N, rounds, self_mode, check_every, k_first, out_y;
  uint32_t polls;
  double da, db, tol;
  MinImage mi;
  DevConsts K;
  Tensor64 T;
  long long eps2;
  const int32_t *cnt, *order;
  const uint32_t *list;
  const double4_32a *pos64;
  const double *coef;         // [N + 1]
  const double *xi;           // caller order
  double4_32a *x[3], *d[2];   // x_{i-1}, x_i, x_{i+1}; dw_i, dw_{i+1} (rotating)
  double *dm;                 // M dw of the last check
  double *out;                // caller order: y (out_y), or M y once converged
  double *part;               // [3][blocks] partial sums
  SeriesCtl *ctl;
};

__device__ __forceinline__ void ld_vec(const double4_32a *p, double &x, double &y, double &z) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
  x = a.x;
  y = a.y;
  z = __ldcg(reinterpret_cast<const double *>(p) + 2);
}

// the sums of v[0..7] over the G lanes of a target: lane sub returns v[0] =
// sum of v[index], index = sub / (G / 8) (G = 4: v[0], v[1] of 2 sub, 2 sub + 1)
template <int G>
__device__ __forceinline__ void group_sum8(int sub, double v[8]) {
  constexpr int kSplit = G >= 8 ? 3 : 2;
  int o = G / 2;
#pragma unroll
  for (int l = 0; l < kSplit; ++l, o >>= 1) {
    const int half = 4 >> l;
    const bool up = sub & o;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i >= half) break;
      const double keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

template <int CACHE>
struct PairCache {
  double g[CACHE > 0 ? CACHE : 1][6];  // xx, xy, xz, yy, yz, zz
  int t[CACHE > 0 ? CACHE : 1];        // source slot, -1 past the row's end
};

// v[0..2] += G f(t), v[4..6] += G d(t)
__device__ __forceinline__ void add_pair(const double g[6], const double4_32a *xv,
                                         const double4_32a *dv, double v[8]) {
  if (xv) {
    double f0, f1, f2;
    ld_vec(xv, f0, f1, f2);
    v[0] = fma(g[0], f0, fma(g[1], f1, fma(g[2], f2, v[0])));
    v[1] = fma(g[1], f0, fma(g[3], f1, fma(g[4], f2, v[1])));
    v[2] = fma(g[2], f0, fma(g[4], f1, fma(g[5], f2, v[2])));
  }
  if (dv) {
    double f0, f1, f2;
    ld_vec(dv, f0, f1, f2);
    v[4] = fma(g[0], f0, fma(g[1], f1, fma(g[2], f2, v[4])));
    v[5] = fma(g[1], f0, fma(g[3], f1, fma(g[4], f2, v[5])));
    v[6] = fma(g[2], f0, fma(g[4], f1, fma(g[5], f2, v[6])));
  }
}

constexpr int kSeriesThreads = 128;

template <int G, int CACHE>
__global__ void __launch_bounds__(kSeriesThreads, CACHE ? 3 : 7) k_series_f64(SeriesF64 a) {
  __shared__ double sh[3][kSeriesThreads / 32];
  __shared__ int s_last, s_ok;
  const int sub = threadIdx.x % G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kT = kSeriesThreads / G;  // targets per block and round
  constexpr int kSpread = G >= 8 ? G / 8 : 1, kVal = G >= 8 ? 1 : 2;
  const int64_t n = a.n;
  const bool faithful = a.check_every == 1;
  const int64_t first = blockIdx.x * (int64_t)(kT * a.rounds) + threadIdx.x / G;
  PairCache<CACHE> pc;
  // the tensor of entry en seen from position pi
  auto tensor = [&](uint32_t en, const double4_32a &pi, double g[6]) {
    const double4_32a pj = ld_f64x4(a.pos64 + (en >> kCodeBits));
    double x = pj.x - pi.x, y = pj.y - pi.y, z = pj.z - pi.z;
    min_image3(a.mi, x, y, z);
    double A, B;
    tensor64(a.T, fma(z, z, fma(y, y, x * x)), a.eps2, a.K.coeff_2, A, B);
    const double bx = B * x, by = B * y;
    g[0] = fma(bx, x, A);
    g[1] = bx * y;
    g[2] = bx * z;
    g[3] = fma(by, y, A);
    g[4] = by * z;
    g[5] = fma(B * z, z, A);
  };
  if (CACHE) {
    const int64_t s = min(first, n - 1);
    const int m = first < n ? __ldg(a.cnt + s) : 0;
    const double4_32a pi = ld_f64x4(a.pos64 + s);
#pragma unroll
    for (int p = 0; p < CACHE; ++p) {
      const int k = sub + p * G;
      pc.t[p] = -1;
      if (k < m) {
        const uint32_t en = __ldg(a.list + s * (int64_t)a.W + k);
        pc.t[p] = (int)(en >> kCodeBits);
        tensor(en, pi, pc.g[p]);
      }
    }
  }
  // M xv (v[0..2]) and M dv (v[4..6]) pair sums of slot s; null: not wanted
  auto walk = [&](int64_t s, bool act, const double4_32a *xv, const double4_32a *dv, double v[8]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = 0.0;
    const int m = act ? __ldg(a.cnt + s) : 0;
    if (CACHE) {
#pragma unroll
      for (int p = 0; p < CACHE; ++p)
        if (pc.t[p] >= 0)
          add_pair(pc.g[p], xv ? xv + pc.t[p] : nullptr, dv ? dv + pc.t[p] : nullptr, v);
    }
    if (m > CACHE * G) {
      const double4_32a pi = ld_f64x4(a.pos64 + s);
      const uint32_t *row = a.list + s * (int64_t)a.W;
      for (int k = CACHE * G + sub; k < m; k += G) {
        const uint32_t en = __ldg(row + k);
        const int64_t t = (int64_t)(en >> kCodeBits);
        double g[6];
        tensor(en, pi, g);
        add_pair(g, xv ? xv + t : nullptr, dv ? dv + t : nullptr, v);
      }
    }
    group_sum8<G>(sub, v);
  };
  auto with_self = [&](double u, double own) {
    if (a.self_mode == GGEM_SELF_BEAD) return (u - a.K.coeff_1 * own) + own;
    if (a.self_mode == GGEM_SELF_LAGRANGIAN) return u + a.K.coeff_2 * own;
    return u;
  };
  auto comp = [](const double4_32a *p, int c) {
    return __ldcg(reinterpret_cast<const double *>(p) + c);
  };
  auto put = [](double4_32a *p, int c, double v) { reinterpret_cast<double *>(p)[c] = v; };
  // f(slot, active) over this block's targets, all lanes together
  auto targets = [&](auto &&f) {
    for (int r = 0; r < a.rounds; ++r) {
      const int64_t s = first + (int64_t)r * kT;
      f(min(s, n - 1), s < n);
    }
  };
  // f(component, vector (0: x, 1: dw), value) for the sums this lane holds
  auto mine = [&](bool act, const double v[8], auto &&f) {
    if (!act || sub % kSpread) return;
#pragma unroll
    for (int q = 0; q < kVal; ++q) {
      const int idx = G >= 8 ? sub / kSpread : 2 * sub + q;
      if ((idx & 3) < 3) f(idx & 3, idx >> 2, v[q]);
    }
  };
  unsigned gen = 0;
  // the end of a phase: this block's three partials, then all blocks arrive;
  // the last one runs work(sum0, sum1, sum2) on its first thread and releases
  // the others.  False: a wait ran out.
  auto barrier = [&](double p0, double p1, double p2, auto &&work) -> bool {
    ++gen;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      p0 += __shfl_xor_sync(0xffffffffu, p0, o);
      p1 += __shfl_xor_sync(0xffffffffu, p1, o);
      p2 += __shfl_xor_sync(0xffffffffu, p2, o);
    }
    if (lane == 0) {
      sh[0][warp] = p0;
      sh[1][warp] = p1;
      sh[2][warp] = p2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kSeriesThreads / 32; ++w) t += sh[q][w];
        __stcg(a.part + (int64_t)q * gridDim.x + blockIdx.x, t);
      }
      __threadfence();
      s_last = atomicAdd(&a.ctl->arrive, 1u) == gen * gridDim.x - 1u;
      s_ok = 1;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      if (warp < 3) {  // one warp per partial
        double t = 0.0;
        for (unsigned b = lane; b < gridDim.x; b += 32)
          t += __ldcg(a.part + (int64_t)warp * gridDim.x + b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sh[warp][0] = t;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        work(sh[0][0], sh[1][0], sh[2][0]);
        __threadfence();
        atomicExch(&a.ctl->release, gen);
      }
    } else if (threadIdx.x == 0) {
      uint32_t k = 0;
      while (*(volatile unsigned int *)&a.ctl->release < gen) {
        if (*(volatile int *)&a.ctl->err || ++k > a.polls) {
          atomicOr(&a.ctl->err, kErrTimeout);
          s_ok = 0;
          break;
        }
        __nanosleep(20);
      }
      __threadfence();
    }
    __syncthreads();
    return s_ok != 0;
  };

  double4_32a *xp = a.x[0], *xc = a.x[1], *xn = a.x[2], *dc = a.d[0], *dn = a.d[1];
  double v[8];
  // x_0 = xi
  targets([&](int64_t s, bool act) {
    if (act && sub < 3) put(xp + s, sub, a.xi[3 * (int64_t)a.order[s] + sub]);
  });
  if (!barrier(0.0, 0.0, 0.0, [](double, double, double) {})) return;
  // m = M x_0; aux2 = m . x_0; x_1 = db x_0 + da m; dw_1 = c0 x_0 + c1 x_1
  {
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    const double c0 = a.coef[0], c1 = a.coef[1];
    targets([&](int64_t s, bool act) {
      walk(s, act, xp, nullptr, v);
      mine(act, v, [&](int c, int vec, double u) {
        if (vec) return;
        const double x = comp(xp + s, c);
        const double m = with_self(u, x);
        const double w = a.db * x + a.da * m;
        const double t = c0 * x;
        put(xc + s, c, w);
        put(dc + s, c, t + c1 * w);
        p0 = fma(t, t, p0);
        p1 = fma(w, w, p1);
        p2 = fma(m, x, p2);
      });
    });
    const bool ok = barrier(p0, p1, p2, [&](double s0, double s1, double s2) {
      a.ctl->aux2 = s2;
      a.ctl->n0 = s0;
      a.ctl->n1 = s1;
      a.ctl->n_terms = 1;
      a.ctl->n_matvecs = 1;
    });
    if (!ok) return;
  }
  for (int i = 1;; ++i) {
    const int t = i - 1;  // the loop index whose term formed dw_i
    const bool chk = faithful || (t > 0 && (t == a.N - 1 || (a.check_every > 1
                                                                ? t % a.check_every == 0
                                                                : i >= a.k_first)));
    const bool term = i < a.N;
    if (!chk && !term) break;
    const double cn = term ? a.coef[i + 1] : 0.0, ci = a.coef[i];
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    targets([&](int64_t s, bool act) {
      if (chk && term) walk(s, act, xc, dc, v);
      else walk(s, act, term ? xc : nullptr, term ? nullptr : dc, v);
      mine(act, v, [&](int c, int vec, double u) {
        if (vec == 0) {
          if (!term) return;
          const double x = comp(xc + s, c), y = comp(dc + s, c);
          double w = (2. * a.db) * x + (2. * a.da) * with_self(u, x);
          w -= comp(xp + s, c);
          put(xn + s, c, w);
          put(dn + s, c, y + cn * w);
          p0 = fma(y, y, p0);
          p1 = fma(w, w, p1);
        } else if (chk) {
          const double m = with_self(u, comp(dc + s, c));
          a.dm[3 * s + c] = m;
          p2 = fma(m, m, p2);
        }
      });
    });
    const bool ok = barrier(p0, p1, p2, [&](double s0, double s1, double s2) {
      SeriesCtl &ctl = *a.ctl;
      if (chk) {
        const double aux4 = sqrt(ctl.n0), aux3 = sqrt(ctl.n1) * fabs(ci), aux2 = ctl.aux2;
        ctl.n_matvecs += 1;
        if (aux2 != 0.0) ctl.err1 = sqrt(fabs(s2 - aux2) / aux2);
        if (aux4 != 0.0) ctl.err2 = aux3 / aux4;
        if (t > 0) {
          if (ctl.first_check < 0) ctl.first_check = i;
          if (ctl.err1 <= a.tol) {  // brownian_system.C:1138-1147
            ctl.converged = 1;
            ctl.stop = 1;
          } else if (ctl.err2 <= 1E-9) {  // :1150
            ctl.stop = 1;
          }
        }
      }
      if (term && !ctl.stop) {
        ctl.n_matvecs += 1;
        ctl.n_terms = i + 1;
      }
      ctl.n0 = s0;
      ctl.n1 = s1;
    });
    if (!ok) return;
    if (!term || *(volatile int *)&a.ctl->stop) break;
    double4_32a *q = xp;
    xp = xc;
    xc = xn;
    xn = q;
    q = dc;
    dc = dn;
    dn = q;
  }
  if (!a.out_y && !*(volatile int *)&a.ctl->converged) return;
  targets([&](int64_t s, bool act) {
    mine(act, v, [&](int c, int vec, double) {
      // (M dw is held by the lanes that formed it, y by those of its update)
      if (vec != (a.out_y ? 0 : 1)) return;
      a.out[3 * (int64_t)a.order[s] + c] = a.out_y ? comp(dc + s, c) : a.dm[3 * s + c];
    });
  });
}

__device__ __forceinline__ void kahan_add(float &sum, float &comp, float v) {
  const float y = v - comp;
  const float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

// one 32-byte record per source (cell-relative position, force of the single
// right-hand side): a single 32-byte gather per pair
struct __align__(32) Rec32 {
  float4 a, b;
};

// the analytic tensor, passed by value (constant bank)
// (a_q, b_q) interleaved so that both polynomials advance in one packed
// FP32x2 FMA per degree (Blackwell FFMA2)
struct PolyAB {
  float2 ab[kPolyDeg + 1];
  float x0, x1, e_hi, e_lo;  // x = s x1 + x0; e^{-alpha^2 s} = 2^{s (e_hi + e_lo)}
};

template <bool POLY>
__device__ __forceinline__ void tensor_ab32(float s2, const PolyAB &P,
                                            const Rec32 *__restrict__ tab, float inv_ds,
                                            float &A, float &B) {
  if (POLY) {
    const float x = fmaf(s2, P.x1, P.x0);
    const float2 xx = make_float2(x, x);
    float2 ab = P.ab[kPolyDeg];
#pragma unroll
    for (int q = kPolyDeg - 1; q >= 0; --q) ab = __ffma2_rn(ab, xx, P.ab[q]);
    // e^{-alpha^2 s} = 2^{p + r}: p = s e_hi rounded, r its exact residual plus
    // s e_lo, so the exponent keeps ~1e-7 relative accuracy at s ~ rc^2
    const float p = s2 * P.e_hi;
    const float r = fmaf(s2, P.e_lo, fmaf(s2, P.e_hi, -p));
    const float E0 = exp2f(p);
    const float E = fmaf(E0, r * 0.6931471805599453f, E0);
    ab = __fmul2_rn(ab, make_float2(E, E));
    A = ab.x;
    B = ab.y;
  } else {
    const float uu = s2 * inv_ds;
    const float fi = fminf(floorf(uu), (float)(kTableN - 1));  // last piece extrapolates
    const float t = uu - fi;
    const Rec32 tr = tab[(int)fi];
    A = fmaf(fmaf(fmaf(tr.a.w, t, tr.a.z), t, tr.a.y), t, tr.a.x);
    B = fmaf(fmaf(fmaf(tr.b.w, t, tr.b.z), t, tr.b.y), t, tr.b.x);
  }
}

template <int CD>
__device__ __forceinline__ void decode_shift(uint32_t e, float hx, float hy, float hz, float &sx,
                                             float &sy, float &sz) {
  constexpr int SIDE = 2 * CD + 1;
  const int code = (int)(e & (kMaxCode - 1));
  sx = (float)(code % SIDE - CD) * hx;
  sy = (float)((code / SIDE) % SIDE - CD) * hy;
  sz = (float)(code / (SIDE * SIDE) - CD) * hz;
}

__device__ __forceinline__ void group_ff(float &hi, float &lo) {
#pragma unroll
  for (int o = kGroup / 2; o > 0; o >>= 1) {
    const float h2 = __shfl_xor_sync(0xffffffffu, hi, o);
    const float l2 = __shfl_xor_sync(0xffffffffu, lo, o);
    ff_add(hi, lo, h2, l2);
  }
}

// lanes sub = 0, 1, 2 of a group write component sub of the target:
// u = (hi + lo) + self_c f with the FP64 force of the target (order: u in the
// caller's particle order)
__device__ __forceinline__ void group_store(bool act, int sub, int64_t s, float hx, float lx,
                                            float hy, float ly, float hz, float lz,
                                            double self_c, const double *__restrict__ f,
                                            double *__restrict__ u,
                                            const int32_t *__restrict__ order = nullptr) {
  if (!act || sub >= 3) return;
  const float h = sub == 0 ? hx : (sub == 1 ? hy : hz);
  const float l = sub == 0 ? lx : (sub == 1 ? ly : lz);
  const double v = f2d_bits(h) + f2d_bits(l);
  u[3 * (order ? (int64_t)order[s] : s) + sub] = fma(self_c, f[3 * s + sub], v);
}

__global__ void k_build_src(int64_t n, const float4 *__restrict__ pos32,
                            const double *__restrict__ f, Rec32 *__restrict__ src) {
  wait_prior_grid();
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  Rec32 r;
  r.a = pos32[s];
  r.b = make_float4(d2f_bits(f[3 * s]), d2f_bits(f[3 * s + 1]), d2f_bits(f[3 * s + 2]), 0.f);
  src[s] = r;
}

// float-float sum of one target's pair terms
struct PairSum {
  float hx, lx, hy, ly, hz, lz;
};

// 2^x on the special-function unit (PTX ex2.approx.ftz.f32); the argument
// range of the tensor, [-alpha^2 rc^2 log2(e), 0], keeps results normal
__device__ __forceinline__ float ex2_sfu(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// one 32-byte record in a single 256-bit read-only load (sm_100+): the
// position and the force of a source share one sector, so one request per
// warp touches each sector once instead of twice
__device__ __forceinline__ Rec32 ld_rec32(const Rec32 *p) {
  Rec32 r;
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y),
                 "=f"(r.b.z), "=f"(r.b.w)
               : "l"(p)
               : "memory");
  return r;
}

// the FP32 cell shift of every entry code, staged per block in shared
// memory (one 16-byte load per pair instead of decoding the code); the
// table holds (float)(k h) for offsets |k| <= 2, which equals the FP32
// product k * (float)h that the list build and decode_shift use
__device__ __forceinline__ void stage_shifts(float4 *sh, const float4 *__restrict__ shift) {
  for (int k = threadIdx.x; k < kMaxCode; k += blockDim.x) sh[k] = shift[k];
  __syncthreads();
}

// reduce-scatter of the group's float-float sums: afterwards lane sub
// (0, 1, 2) holds component sub of the target's total, summed in the same
// tree as the all-reduce ((lane 0 + lane 2) + (lane 1 + lane 3))
__device__ __forceinline__ void group_scatter3(int sub, const PairSum &r, float &h, float &l) {
  const bool up = sub & 2;
  // lanes 0, 1 keep (x, y) and send z; lanes 2, 3 keep z and send (x, y)
  float k1h = up ? r.hz : r.hx, k1l = up ? r.lz : r.lx;
  float k2h = up ? 0.f : r.hy, k2l = up ? 0.f : r.ly;
  const float s1h = up ? r.hx : r.hz, s1l = up ? r.lx : r.lz;
  const float s2h = up ? r.hy : 0.f, s2l = up ? r.ly : 0.f;
  const float a1h = __shfl_xor_sync(0xffffffffu, s1h, 2), a1l = __shfl_xor_sync(0xffffffffu, s1l, 2);
  const float a2h = __shfl_xor_sync(0xffffffffu, s2h, 2), a2l = __shfl_xor_sync(0xffffffffu, s2l, 2);
  ff_add(k1h, k1l, a1h, a1l);
  ff_add(k2h, k2l, a2h, a2l);
  // lane 0 keeps x, lane 1 keeps y, lane 2 keeps z (lane 3: zero)
  const bool odd = sub & 1;
  h = odd ? k2h : k1h;
  l = odd ? k2l : k1l;
  const float th = odd ? k1h : k2h, tl = odd ? k1l : k2l;
  const float bh = __shfl_xor_sync(0xffffffffu, th, 1), bl = __shfl_xor_sync(0xffffffffu, tl, 1);
  ff_add(h, l, bh, bl);
}

// the pair loop of one target slot s over its list entries (one right-hand
// side, 32-byte source records); lanes sub = 0..kGroup-1 take every
// kGroup-th entry, so a group reads consecutive list words.  The next entry
// of the lane is loaded while the current pair is evaluated.  (Prefetching
// the next source record into registers or L1 as well measured no faster.)
template <bool POLY>
__device__ __forceinline__ PairSum pair_sum_r1(int64_t s, bool act, int sub, const Rec32 &ri,
                                               const Rec32 *__restrict__ src,
                                               const int32_t *__restrict__ cnt, int W,
                                               const uint32_t *__restrict__ list,
                                               const PolyAB &P, const Rec32 *__restrict__ tab,
                                               float inv_ds, const float4 *sh) {
  const uint32_t *lp = list + s * (int64_t)W + sub;
  int left = (act ? cnt[s] : 0) - sub;  // entries lp[0], lp[kGroup], ... while left > 0
  float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float2 bxy = make_float2(0.f, 0.f);
  float bz = 0.f;
  int blk = 0;
  uint32_t nxt = left > 0 ? __ldg(lp) : 0u;
  while (left > 0) {
    const uint32_t en = nxt;
    left -= kGroup;
    lp += kGroup;
    if (left > 0) nxt = __ldg(lp);
    const Rec32 rj = ld_rec32(src + (en >> kCodeBits));
    const float4 o = sh[en & (kMaxCode - 1)];
    const float dx = (rj.a.x - ri.a.x) + o.x;
    const float dy = (rj.a.y - ri.a.y) + o.y;
    const float dz = (rj.a.z - ri.a.z) + o.z;
    const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    float A, B;
    if (POLY) {
      const float x = fmaf(s2, P.x1, P.x0);
      const float2 xx = make_float2(x, x);
      float2 ab = P.ab[kPolyDeg];
#pragma unroll
      for (int q = kPolyDeg - 1; q >= 0; --q) ab = __ffma2_rn(ab, xx, P.ab[q]);
      // e^{-alpha^2 s} = 2^{p + r}, p = s e_hi rounded, r its residual plus s e_lo
      const float p = s2 * P.e_hi;
      const float r = fmaf(s2, P.e_lo, fmaf(s2, P.e_hi, -p));
      const float E0 = ex2_sfu(p);
      const float E = fmaf(E0, r * 0.6931471805599453f, E0);
      ab = __fmul2_rn(ab, make_float2(E, E));
      A = ab.x;
      B = ab.y;
    } else {
      tensor_ab32<false>(s2, P, tab, inv_ds, A, B);
    }
    // G f = A f + B (x.f) x, the x and y components packed (FFMA2)
    const float2 dxy = make_float2(dx, dy), fxy = make_float2(rj.b.x, rj.b.y);
    const float2 pxy = __fmul2_rn(dxy, fxy);
    const float bxf = B * fmaf(dz, rj.b.z, pxy.x + pxy.y);
    bxy = __fadd2_rn(bxy, __ffma2_rn(make_float2(A, A), fxy,
                                     __fmul2_rn(make_float2(bxf, bxf), dxy)));
    bz += fmaf(A, rj.b.z, bxf * dz);
    if (++blk == 8) {
      kahan_add(sx, cx, bxy.x);
      kahan_add(sy, cy, bxy.y);
      kahan_add(sz, cz, bz);
      bxy = make_float2(0.f, 0.f);
      bz = 0.f;
      blk = 0;
    }
  }
  kahan_add(sx, cx, bxy.x);
  kahan_add(sy, cy, bxy.y);
  kahan_add(sz, cz, bz);
  // Kahan keeps sum = s - c: the float-float value is (s, -c)
  return PairSum{sx, -cx, sy, -cy, sz, -cz};
}

// The fused series' estimator sums (x0 . M x0, |dw|^2, |x_{k+1}|^2, |M dw|^2)
// without FP64 arithmetic (ggem_ff.cuh): float-float products and sums, one
// partial per block (256 threads) written by thread 0.
__device__ __forceinline__ void block_partial_ff(float hi, float lo, double *__restrict__ part) {
  __shared__ float2 sh[32];
  const double v = block_ff_sum(hi, lo, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

// ---- symmetric pair sums --------------------------------------------------
// The tensor of a pair is symmetric (G(x) = G(-x)), so each unordered pair is
// evaluated once, from the half list (the row of the smaller slot): the
// target side A f_j + B (x.f_j) x is summed in registers as in pair_sum_r1,
// the source side A f_i + B (x.f_i) x goes to the source's accumulator with
// one 16-byte vector atomic (red.global.add.v4.f32).  The order in which a
// source's contributions arrive varies from run to run, so the FP32 result
// is not bit-reproducible (the FP64 paths and the full-row kernels are).
__device__ __forceinline__ void red_add_v4(float4 *p, float x, float y, float z) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y),
               "f"(z), "f"(0.f)
               : "memory");
}

template <bool POLY>
__device__ __forceinline__ PairSum pair_sum_sym(int64_t s, bool act, int sub, const Rec32 &ri,
                                                const Rec32 *__restrict__ src,
                                                const int32_t *__restrict__ cnt, int W,
                                                const uint32_t *__restrict__ list,
                                                const PolyAB &P, const Rec32 *__restrict__ tab,
                                                float inv_ds, const float4 *sh,
                                                float4 *__restrict__ acc) {
  const uint32_t *lp = list + s * (int64_t)W + sub;
  int left = (act ? cnt[s] : 0) - sub;
  float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float2 bxy = make_float2(0.f, 0.f);
  float bz = 0.f;
  int blk = 0;
  const float2 fixy = make_float2(ri.b.x, ri.b.y);
  uint32_t nxt = left > 0 ? __ldg(lp) : 0u;
  while (left > 0) {
    const uint32_t en = nxt;
    left -= kGroup;
    lp += kGroup;
    if (left > 0) nxt = __ldg(lp);
    const uint32_t j = en >> kCodeBits;
    const Rec32 rj = ld_rec32(src + j);
    const float4 o = sh[en & (kMaxCode - 1)];
    const float dx = (rj.a.x - ri.a.x) + o.x;
    const float dy = (rj.a.y - ri.a.y) + o.y;
    const float dz = (rj.a.z - ri.a.z) + o.z;
    const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    float A, B;
    if (POLY) {
      const float x = fmaf(s2, P.x1, P.x0);
      const float2 xx = make_float2(x, x);
      float2 ab = P.ab[kPolyDeg];
#pragma unroll
      for (int q = kPolyDeg - 1; q >= 0; --q) ab = __ffma2_rn(ab, xx, P.ab[q]);
      const float p = s2 * P.e_hi;
      const float r = fmaf(s2, P.e_lo, fmaf(s2, P.e_hi, -p));
      const float E0 = ex2_sfu(p);
      const float E = fmaf(E0, r * 0.6931471805599453f, E0);
      ab = __fmul2_rn(ab, make_float2(E, E));
      A = ab.x;
      B = ab.y;
    } else {
      tensor_ab32<false>(s2, P, tab, inv_ds, A, B);
    }
    const float2 dxy = make_float2(dx, dy);
    // target side: G f_j
    const float2 fxy = make_float2(rj.b.x, rj.b.y);
    const float2 pxy = __fmul2_rn(dxy, fxy);
    const float bxf = B * fmaf(dz, rj.b.z, pxy.x + pxy.y);
    bxy = __fadd2_rn(bxy, __ffma2_rn(make_float2(A, A), fxy,
                                     __fmul2_rn(make_float2(bxf, bxf), dxy)));
    bz += fmaf(A, rj.b.z, bxf * dz);
    // source side: G f_i into the source's accumulator
    const float2 qxy = __fmul2_rn(dxy, fixy);
    const float bxi = B * fmaf(dz, ri.b.z, qxy.x + qxy.y);
    const float2 vxy = __ffma2_rn(make_float2(A, A), fixy, __fmul2_rn(make_float2(bxi, bxi), dxy));
    red_add_v4(acc + j, vxy.x, vxy.y, fmaf(A, ri.b.z, bxi * dz));
    if (++blk == 8) {
      kahan_add(sx, cx, bxy.x);
      kahan_add(sy, cy, bxy.y);
      kahan_add(sz, cz, bz);
      bxy = make_float2(0.f, 0.f);
      bz = 0.f;
      blk = 0;
    }
  }
  kahan_add(sx, cx, bxy.x);
  kahan_add(sy, cy, bxy.y);
  kahan_add(sz, cz, bz);
  return PairSum{sx, -cx, sy, -cy, sz, -cz};
}

// the target sides of the half rows: part[3 s + c] (FP64 of the group's
// float-float sum); the source sides accumulate in acc
template <bool POLY>
__global__ void __launch_bounds__(256, 6) k_pair_sym(
    int64_t n, const Rec32 *__restrict__ src, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    const float4 *__restrict__ shift, float4 *__restrict__ acc, double *__restrict__ part) {
  __shared__ float4 sh[kMaxCode];
  stage_shifts(sh, shift);
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const Rec32 ri = src[s];
  const PairSum r = pair_sum_sym<POLY>(s, act, sub, ri, src, cnt, W, list, P, tab, inv_ds, sh,
                                       acc);
  float h, l;
  group_scatter3(sub, r, h, l);
  if (act && sub < 3) part[3 * s + sub] = f2d_bits(h) + f2d_bits(l);
}

// u = part + acc + self term; acc is cleared for the next use
__global__ void k_sym_finish(int64_t n, const double *__restrict__ part, float4 *__restrict__ acc,
                             double self_c, const double *__restrict__ f, double *__restrict__ u) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float4 a = acc[s];
  acc[s] = make_float4(0.f, 0.f, 0.f, 0.f);
  const float v[3] = {a.x, a.y, a.z};
#pragma unroll
  for (int c = 0; c < 3; ++c)
    u[3 * s + c] = fma(self_c, f[3 * s + c], part[3 * s + c] + f2d_bits(v[c]));
}

// the per-matvec-tensor kernel shapes the autotuner chooses from: blocks of
// 256 threads per SM that the register cap allows (6 at 40 registers, with a
// few spilled epilogue values in some kernels; 5 at 48 without)
constexpr int kComputedMinBlocks[] = {6, 5};
constexpr int kNumComputedVariants = 2;

// u = M f, single right-hand side; with ORIG, u is written in the caller's
// particle order (u[order[s]]) instead of slot order
template <bool POLY, int V, bool ORIG>
__global__ void __launch_bounds__(256, kComputedMinBlocks[V]) k_pair_r1(
    int64_t n, const Rec32 *__restrict__ src, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    const float4 *__restrict__ shift, double self_c, const double *__restrict__ f,
    double *__restrict__ u, const int32_t *__restrict__ order, double *__restrict__ part) {
  __shared__ float4 sh[kMaxCode];
  stage_shifts(sh, shift);  // (constant: no kernel writes it)
  wait_prior_grid();
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const Rec32 ri = src[s];
  const PairSum r = pair_sum_r1<POLY>(s, act, sub, ri, src, cnt, W, list, P, tab, inv_ds, sh);
  float h, l;
  group_scatter3(sub, r, h, l);
  float qh = 0.f, ql = 0.f;
  if (act && sub < 3) {
    const int64_t k = 3 * s + sub;
    const double v = fma(self_c, f[k], f2d_bits(h) + f2d_bits(l));
    if (ORIG) u[3 * (int64_t)order[s] + sub] = v;
    else u[k] = v;
    if (part) sq_ff(v, qh, ql);
  }
  if (part) block_partial_ff(qh, ql, part);  // |u|^2 (uniform branch)
}

// The first Chebyshev step in one pass (brownian_system.C:1036-1056 for one
// right-hand side): m = M x0 (src holds the records of x0, m is kept for
// the dot xi . M xi), x1 = db x0 + da m, dw = c0 x0 + c1 x1, and the 32-byte
// records of x1 for the first term.  (The estimator sums stay in separate
// vector kernels: a block-wide FP64 reduction here costs more than the
// launch it saves, FP64 being 1/64 of the FP32 rate.)
template <bool POLY, int V>
__global__ void __launch_bounds__(256, kComputedMinBlocks[V]) k_pair_first(
    int64_t n, const Rec32 *__restrict__ src, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    const float4 *__restrict__ shift, double self_c, double da, double db, double c0, double c1,
    const double *__restrict__ x0, double *__restrict__ m, double *__restrict__ x1,
    double *__restrict__ dw, Rec32 *__restrict__ next, double *__restrict__ part) {
  __shared__ float4 sh[kMaxCode];
  stage_shifts(sh, shift);  // (constant: no kernel writes it)
  wait_prior_grid();
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const Rec32 ri = src[s];
  const PairSum r = pair_sum_r1<POLY>(s, act, sub, ri, src, cnt, W, list, P, tab, inv_ds, sh);
  float h, l;
  group_scatter3(sub, r, h, l);
  float qh = 0.f, ql = 0.f;
  if (act) {
    float *nf = reinterpret_cast<float *>(next + s);
    if (sub < 3) {
      const int64_t k = 3 * s + sub;
      const double xk = x0[k];
      const double mk = fma(self_c, xk, f2d_bits(h) + f2d_bits(l));
      m[k] = mk;
      const double x1k = db * xk + da * mk;
      x1[k] = x1k;
      dw[k] = c0 * xk + c1 * x1k;
      nf[4 + sub] = d2f_bits(x1k);
      if (part) dot_ff(xk, mk, qh, ql);
    } else {
      reinterpret_cast<float4 *>(nf)[0] = ri.a;
      nf[7] = 0.f;
    }
  }
  if (part) block_partial_ff(qh, ql, part);  // x0 . M x0 (aux2; uniform branch)
}

// One Chebyshev term with the pair sum (brownian_system.C:1091-1108 for one
// right-hand side, without the norms of the error estimators):
//   m = M x1 (pair sum + self term),  xm = (2db x1 + 2da m) - x0,
//   dw += coef xm,  and the 32-byte records of xm for the next term.
// With c1 = 2db + 2da self_c this is xm = 2da (pair sum) + (c1 x1 - x0).
// src holds the records of x1; next must be a different buffer.
template <bool POLY, int V, bool NORMS>
__global__ void __launch_bounds__(256, kComputedMinBlocks[V]) k_pair_cheb(
    int64_t n, const Rec32 *__restrict__ src, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    const float4 *__restrict__ shift, double two_da, double c1, double coef,
    const double *__restrict__ x0, const double *__restrict__ x1, double *__restrict__ xm,
    double *__restrict__ dw, Rec32 *__restrict__ next, double *__restrict__ part,
    int64_t nw, Rec32 *__restrict__ dw_next) {
  __shared__ float4 sh[kMaxCode];
  stage_shifts(sh, shift);  // (constant: no kernel writes it)
  wait_prior_grid();
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const Rec32 ri = src[s];
  const PairSum r = pair_sum_r1<POLY>(s, act, sub, ri, src, cnt, W, list, P, tab, inv_ds, sh);
  float h, l;
  group_scatter3(sub, r, h, l);
  float q0h = 0.f, q0l = 0.f, q1h = 0.f, q1l = 0.f;
  if (act) {
    float *nf = reinterpret_cast<float *>(next + s);
    float *df = reinterpret_cast<float *>(dw_next + s);
    if (sub < 3) {
      const int64_t k = 3 * s + sub;
      const double v = fma(two_da, f2d_bits(h) + f2d_bits(l), fma(c1, x1[k], -x0[k]));
      xm[k] = v;
      const double y = dw[k];
      const double yn = fma(coef, v, y);
      dw[k] = yn;
      nf[4 + sub] = d2f_bits(v);
      if (NORMS) {
        sq_ff(y, q0h, q0l);  // |dw|^2 before the term
        sq_ff(v, q1h, q1l);  // |x_{k+1}|^2
        df[4 + sub] = d2f_bits(yn);
      }
    } else {
      reinterpret_cast<float4 *>(nf)[0] = ri.a;  // the target's position record
      nf[7] = 0.f;
      if (NORMS) {
        reinterpret_cast<float4 *>(df)[0] = ri.a;
        df[7] = 0.f;
      }
    }
  }
  if (NORMS) {  // the estimators' two norms (the records of dw are written)
    block_partial_ff(q0h, q0l, part);
    __syncthreads();  // the shared partials are reused
    block_partial_ff(q1h, q1l, part + nw);
  }
}

// xi (caller order) into slot order and the 32-byte records of it
__global__ void k_to_slots_rec(int64_t n, const int32_t *__restrict__ order,
                               const float4 *__restrict__ pos32, const double *__restrict__ xi,
                               double *__restrict__ x0, Rec32 *__restrict__ rec) {
  wait_prior_grid();
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int64_t i = order[s];
  const double a = xi[3 * i], b = xi[3 * i + 1], c = xi[3 * i + 2];
  x0[3 * s] = a;
  x0[3 * s + 1] = b;
  x0[3 * s + 2] = c;
  Rec32 r;
  r.a = pos32[s];
  r.b = make_float4((float)a, (float)b, (float)c, 0.f);
  rec[s] = r;
}

// ---- precomputed pair tensors ---------------------------------------------
//
// Once per configuration, every listed pair's tensor is stored as t = (A, sqrt(B) x) in the list's row layout, valid when
// B >= 0 on [0, rc^2] (checked at context creation).  A matvec then streams
// 20 B per pair (entry + tensor, evict-first) and gathers a 16-byte force:
// G f = A f + (x~ . f) x~ with x~ = sqrt(B) x, no position gathers and no
// polynomial per pair and matvec.
template <int CD, bool POLY>
__device__ __forceinline__ void tensor_row(int64_t s, int sub, const float4 *__restrict__ pos32,
                                           const int32_t *__restrict__ cnt, int W,
                                           const uint32_t *__restrict__ list, const PolyAB &P,
                                           const Rec32 *__restrict__ tab, float inv_ds, float hx,
                                           float hy, float hz, float4 *__restrict__ ten) {
  const float4 pi = pos32[s];
  const int64_t b = s * (int64_t)W, e = b + cnt[s];
  for (int64_t m = b + sub; m < e; m += 2 * kGroup) {
    const bool two = m + kGroup < e;
    const uint32_t en0 = __ldg(list + m), en1 = two ? __ldg(list + m + kGroup) : en0;
    const float4 pj0 = __ldg(pos32 + (en0 >> kCodeBits)), pj1 = __ldg(pos32 + (en1 >> kCodeBits));
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (q == 1 && !two) break;
      const uint32_t en = q ? en1 : en0;
      const float4 pj = q ? pj1 : pj0;
      float ox, oy, oz;
      decode_shift<CD>(en, hx, hy, hz, ox, oy, oz);
      const float dx = (pj.x - pi.x) + ox, dy = (pj.y - pi.y) + oy, dz = (pj.z - pi.z) + oz;
      const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      float A, B;
      tensor_ab32<POLY>(s2, P, tab, inv_ds, A, B);
      const float w = sqrtf(fmaxf(B, 0.f));
      __stcs(ten + m + q * kGroup, make_float4(A, w * dx, w * dy, w * dz));
    }
  }
}

template <int CD, bool POLY>
__global__ void __launch_bounds__(256) k_pair_tensor(
    int64_t n, const float4 *__restrict__ pos32, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    float hx, float hy, float hz, float4 *__restrict__ ten) {
  wait_prior_grid();
  const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  if (s < n)
    tensor_row<CD, POLY>(s, (int)(threadIdx.x % kGroup), pos32, cnt, W, list, P, tab, inv_ds, hx,
                         hy, hz, ten);
}

// the tensors of K suspensions' concatenated rows
template <int CD, bool POLY>
__global__ void __launch_bounds__(256) k_batch_tensor(
    int64_t n, const BatchGeo *__restrict__ geo, const int32_t *__restrict__ susp,
    const float4 *__restrict__ pos32, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, PolyAB P, const Rec32 *__restrict__ tab, float inv_ds,
    float4 *__restrict__ ten) {
  const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  if (s >= n) return;
  const float *h = geo[susp[s]].g.h32;
  tensor_row<CD, POLY>(s, (int)(threadIdx.x % kGroup), pos32, cnt, W, list, P, tab, inv_ds, h[0],
                       h[1], h[2], ten);
}

// xi (caller order) into slot order and one float4 per slot of it
__global__ void k_to_slots_f4(int64_t n, const int32_t *__restrict__ order,
                              const double *__restrict__ xi, double *__restrict__ x0,
                              float4 *__restrict__ f4) {
  wait_prior_grid();
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int64_t i = order[s];
  const double a = xi[3 * i], b = xi[3 * i + 1], c = xi[3 * i + 2];
  x0[3 * s] = a;
  x0[3 * s + 1] = b;
  x0[3 * s + 2] = c;
  f4[s] = make_float4(d2f_bits(a), d2f_bits(b), d2f_bits(c), 0.f);
}

// forces of one right-hand side as one float4 per slot (w = 0)
__global__ void k_stage_f4(int64_t n, const double *__restrict__ f, float4 *__restrict__ f4) {
  wait_prior_grid();
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  f4[s] = make_float4(d2f_bits(f[3 * s]), d2f_bits(f[3 * s + 1]), d2f_bits(f[3 * s + 2]), 0.f);
}

// float-float sum over the G lanes of a target's group
template <int G>
__device__ __forceinline__ void group_ff_g(float &hi, float &lo) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float h2 = __shfl_xor_sync(0xffffffffu, hi, o);
    const float l2 = __shfl_xor_sync(0xffffffffu, lo, o);
    ff_add(hi, lo, h2, l2);
  }
}

// blk += G f over one entry: A f + (x~ . f) x~, x and y packed (FFMA2)
__device__ __forceinline__ void tensor_apply(const float4 &t, const float4 &fj, float2 &bxy,
                                             float &bz) {
  const float2 txy = make_float2(t.y, t.z), fxy = make_float2(fj.x, fj.y);
  const float2 p = __fmul2_rn(txy, fxy);
  const float d = fmaf(t.w, fj.z, p.x + p.y);
  bxy = __fadd2_rn(bxy, __ffma2_rn(make_float2(t.x, t.x), fxy, __fmul2_rn(make_float2(d, d), txy)));
  bz += fmaf(t.x, fj.z, d * t.w);
}

// The pair loop over stored tensors for one target slot s (cf. pair_sum_r1):
// G lanes share the target and take every G-th entry, U entries per lane and
// iteration are loaded before any is used (an entry past the row end reads a
// zero tensor and adds exactly zero).  PIPE: the streamed entries and tensors
// of the next iteration are requested before the current iteration's force
// gathers are used, so that the HBM latency of the stream overlaps the L2
// latency of the gathers.  Variants are picked by ggem_autotune_pair_storage.
template <int G, int U, bool PIPE>
__device__ __forceinline__ PairSum pair_sum_tv(int64_t s, bool act, int sub,
                                               const float4 *__restrict__ f4,
                                               const int32_t *__restrict__ cnt, int W,
                                               const uint32_t *__restrict__ list,
                                               const float4 *__restrict__ ten) {
  constexpr int FLUSH = (8 + U - 1) / U;  // iterations per Kahan flush (~8 entries)
  const int64_t b = s * (int64_t)W, e = act ? b + cnt[s] : b;
  float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float2 bxy = make_float2(0.f, 0.f);
  float bz = 0.f;
  int blk = 0;
  uint32_t en[U];
  float4 t[U];
  int64_t m = b + sub;
  if (PIPE) {
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int64_t mq = m + q * G;
      const bool ok = mq < e;
      en[q] = ok ? __ldcs(list + mq) : 0u;
      t[q] = ok ? __ldcs(ten + mq) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  for (; m < e; m += U * G) {
    if (!PIPE) {
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int64_t mq = m + q * G;
        const bool ok = mq < e;
        en[q] = ok ? __ldcs(list + mq) : 0u;
        t[q] = ok ? __ldcs(ten + mq) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    float4 fj[U];
#pragma unroll
    for (int q = 0; q < U; ++q) fj[q] = __ldg(f4 + (en[q] >> kCodeBits));
    float4 tc[U];
#pragma unroll
    for (int q = 0; q < U; ++q) tc[q] = t[q];
    if (PIPE) {
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int64_t mq = m + U * G + q * G;
        const bool ok = mq < e;
        en[q] = ok ? __ldcs(list + mq) : 0u;
        t[q] = ok ? __ldcs(ten + mq) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) tensor_apply(tc[q], fj[q], bxy, bz);
    if (++blk == FLUSH) {
      kahan_add(sx, cx, bxy.x);
      kahan_add(sy, cy, bxy.y);
      kahan_add(sz, cz, bz);
      bxy = make_float2(0.f, 0.f);
      bz = 0.f;
      blk = 0;
    }
  }
  kahan_add(sx, cx, bxy.x);
  kahan_add(sy, cy, bxy.y);
  kahan_add(sz, cz, bz);
  PairSum r{sx, -cx, sy, -cy, sz, -cz};
  group_ff_g<G>(r.hx, r.lx);
  group_ff_g<G>(r.hy, r.ly);
  group_ff_g<G>(r.hz, r.lz);
  return r;
}

// u = M f from stored tensors, single right-hand side
template <int G, int U, bool PIPE>
__global__ void __launch_bounds__(256) k_pair_r1tv(int64_t n, const float4 *__restrict__ f4,
                                                   const int32_t *__restrict__ cnt, int W,
                                                   const uint32_t *__restrict__ list,
                                                   const float4 *__restrict__ ten, double self_c,
                                                   const double *__restrict__ f,
                                                   double *__restrict__ u, const int32_t *__restrict__ order) {
  wait_prior_grid();
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int sub = (int)(threadIdx.x % G);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const PairSum r = pair_sum_tv<G, U, PIPE>(s, act, sub, f4, cnt, W, list, ten);
  group_store(act, sub, s, r.hx, r.lx, r.hy, r.ly, r.hz, r.lz, self_c, f, u, order);
}

// The first product over a new list: forms each pair's tensor (the
// arithmetic of tensor_row), stores it for the products after it and applies
// it (the lanes, order and sums of k_pair_r1tv with four lanes per target),
// so that it is written once and not read back: a matvec with its list, N =
// 400k, 337 -> 307 us (tensors 70 us and product 76 us as two kernels).  Two
// entries in flight per lane (52 registers); four are slower (310 us).
template <int CD, bool POLY, int U>
__global__ void __launch_bounds__(256) k_pair_r1tv_first(
    int64_t n, const float4 *__restrict__ pos32, const float4 *__restrict__ f4,
    const int32_t *__restrict__ cnt, int W, const uint32_t *__restrict__ list, PolyAB P,
    const Rec32 *__restrict__ tab, float inv_ds, float hx, float hy, float hz,
    float4 *__restrict__ ten, double self_c, const double *__restrict__ f,
    double *__restrict__ u, const int32_t *__restrict__ order) {
  wait_prior_grid();
  constexpr int FLUSH = 8 / U;  // iterations per Kahan flush
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const float4 pi = pos32[s];
  const int64_t b = s * (int64_t)W, e = act ? b + cnt[s] : b;
  float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float2 bxy = make_float2(0.f, 0.f);
  float bz = 0.f;
  int blk = 0;
  for (int64_t m = b + sub; m < e; m += U * kGroup) {
    uint32_t en[U];
    float4 pj[U], fj[U];
#pragma unroll
    for (int q = 0; q < U; ++q) en[q] = m + q * kGroup < e ? __ldg(list + m + q * kGroup) : 0u;
#pragma unroll
    for (int q = 0; q < U; ++q) {
      pj[q] = __ldg(pos32 + (en[q] >> kCodeBits));
      fj[q] = __ldg(f4 + (en[q] >> kCodeBits));
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (m + q * kGroup >= e) break;
      float ox, oy, oz;
      decode_shift<CD>(en[q], hx, hy, hz, ox, oy, oz);
      const float dx = (pj[q].x - pi.x) + ox, dy = (pj[q].y - pi.y) + oy, dz = (pj[q].z - pi.z) + oz;
      const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      float A, B;
      tensor_ab32<POLY>(s2, P, tab, inv_ds, A, B);
      const float w = sqrtf(fmaxf(B, 0.f));
      const float4 t = make_float4(A, w * dx, w * dy, w * dz);
      __stcs(ten + m + q * kGroup, t);
      tensor_apply(t, fj[q], bxy, bz);
    }
    if (++blk == FLUSH) {
      kahan_add(sx, cx, bxy.x);
      kahan_add(sy, cy, bxy.y);
      kahan_add(sz, cz, bz);
      bxy = make_float2(0.f, 0.f);
      bz = 0.f;
      blk = 0;
    }
  }
  kahan_add(sx, cx, bxy.x);
  kahan_add(sy, cy, bxy.y);
  kahan_add(sz, cz, bz);
  PairSum r{sx, -cx, sy, -cy, sz, -cz};
  group_ff_g<kGroup>(r.hx, r.lx);
  group_ff_g<kGroup>(r.hy, r.ly);
  group_ff_g<kGroup>(r.hz, r.lz);
  group_store(act, sub, s, r.hx, r.lx, r.hy, r.ly, r.hz, r.lz, self_c, f, u, order);
}

// one Chebyshev term from stored tensors (cf. k_pair_cheb); f4 holds the
// FP32 forces of x1, next receives those of xm
template <int G, int U, bool PIPE>
__global__ void __launch_bounds__(256) k_pair_cheb_tv(
    int64_t n, const float4 *__restrict__ f4, const int32_t *__restrict__ cnt, int W,
    const uint32_t *__restrict__ list, const float4 *__restrict__ ten, double self_c,
    double two_da, double two_db, double coef, const double *__restrict__ x0,
    const double *__restrict__ x1, double *__restrict__ xm, double *__restrict__ dw,
    float4 *__restrict__ next) {
  wait_prior_grid();
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int sub = (int)(threadIdx.x % G);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const PairSum r = pair_sum_tv<G, U, PIPE>(s, act, sub, f4, cnt, W, list, ten);
  if (!act) return;
  float *nf = reinterpret_cast<float *>(next + s);
  if (sub < 3) {
    const float h = sub == 0 ? r.hx : (sub == 1 ? r.hy : r.hz);
    const float l = sub == 0 ? r.lx : (sub == 1 ? r.ly : r.lz);
    const int64_t k = 3 * s + sub;
    const double xk = x1[k];
    const double m = fma(self_c, xk, f2d_bits(h) + f2d_bits(l));
    double v = two_db * xk + two_da * m;
    v -= x0[k];
    xm[k] = v;
    dw[k] = dw[k] + coef * v;
    nf[sub] = d2f_bits(v);
  } else if (sub == 3) {
    nf[3] = 0.f;
  }
}

// the stored-tensor variants the autotuner chooses from: lanes per target,
// entries in flight per lane, pipelined stream
struct StoredVariant {
  int G, U;
  bool pipe;
};
constexpr StoredVariant kStoredVariants[] = {{4, 4, false}, {4, 2, true}, {8, 2, true}, {8, 4, false}};
constexpr int kNumStoredVariants = 4;

template <int V>
void launch_stored_r1(ggem_ctx *c, const float4 *f4, double self_c, const double *f, double *u,
                      const int32_t *order) {
  constexpr StoredVariant sv = kStoredVariants[V];
  const int64_t threads = c->n * sv.G;
  launch_dependent(k_pair_r1tv<sv.G, sv.U, sv.pipe>, dim3((unsigned)((threads + 255) / 256)), 256, 0,
                   c->stream, 
      c->n, f4, c->nb_cnt.p, c->nb_w, c->nb_list.p, c->pair_ten.p, self_c, f, u, order);
}

template <int V>
void launch_stored_cheb(ggem_ctx *c, const float4 *f4, double self_c, double two_da,
                        double two_db, double coef, const double *x0, const double *x1,
                        double *xm, double *dw, float4 *next) {
  constexpr StoredVariant sv = kStoredVariants[V];
  const int64_t threads = c->n * sv.G;
  launch_dependent(k_pair_cheb_tv<sv.G, sv.U, sv.pipe>, dim3((unsigned)((threads + 255) / 256)), 256, 0,
                   c->stream, 
      c->n, f4, c->nb_cnt.p, c->nb_w, c->nb_list.p, c->pair_ten.p, self_c, two_da, two_db, coef,
      x0, x1, xm, dw, next);
}

void dispatch_stored_r1(ggem_ctx *c, const float4 *f4, double self_c, const double *f, double *u,
                        const int32_t *order) {
  switch (c->stored_variant) {
    case 1: launch_stored_r1<1>(c, f4, self_c, f, u, order); break;
    case 2: launch_stored_r1<2>(c, f4, self_c, f, u, order); break;
    case 3: launch_stored_r1<3>(c, f4, self_c, f, u, order); break;
    default: launch_stored_r1<0>(c, f4, self_c, f, u, order); break;
  }
}

void dispatch_stored_cheb(ggem_ctx *c, const float4 *f4, double self_c, double two_da,
                          double two_db, double coef, const double *x0, const double *x1,
                          double *xm, double *dw, float4 *next) {
  switch (c->stored_variant) {
    case 1: launch_stored_cheb<1>(c, f4, self_c, two_da, two_db, coef, x0, x1, xm, dw, next); break;
    case 2: launch_stored_cheb<2>(c, f4, self_c, two_da, two_db, coef, x0, x1, xm, dw, next); break;
    case 3: launch_stored_cheb<3>(c, f4, self_c, two_da, two_db, coef, x0, x1, xm, dw, next); break;
    default: launch_stored_cheb<0>(c, f4, self_c, two_da, two_db, coef, x0, x1, xm, dw, next); break;
  }
}

// NR right-hand sides r0 .. r0+NR-1: f32 is [r][n] float4, u [r][n][3]
template <int CD, bool POLY, int NR>
__global__ void __launch_bounds__(256) k_pair_nr(
    int64_t n, const float4 *__restrict__ pos32, const float4 *__restrict__ f32,
    const int32_t *__restrict__ cnt, int W, const uint32_t *__restrict__ list, PolyAB P,
    const Rec32 *__restrict__ tab, float inv_ds, float hx, float hy, float hz, double self_c,
    const double *__restrict__ f, double *__restrict__ u, int r0) {
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGroup;
  const int sub = (int)(threadIdx.x % kGroup);
  const bool act = gid < n;
  const int64_t s = act ? gid : n - 1;
  const int64_t b = s * (int64_t)W, e = act ? b + cnt[s] : b;
  const float4 pi = pos32[s];
  float sx[NR], sy[NR], sz[NR], cx[NR], cy[NR], cz[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) sx[q] = sy[q] = sz[q] = cx[q] = cy[q] = cz[q] = 0.f;
  for (int64_t m = b + sub; m < e; m += kGroup) {
    const uint32_t en = __ldg(list + m);
    const uint32_t j = en >> kCodeBits;
    const float4 pj = __ldg(pos32 + j);
    float ox, oy, oz;
    decode_shift<CD>(en, hx, hy, hz, ox, oy, oz);
    const float dx = (pj.x - pi.x) + ox;
    const float dy = (pj.y - pi.y) + oy;
    const float dz = (pj.z - pi.z) + oz;
    const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    float A, B;
    tensor_ab32<POLY>(s2, P, tab, inv_ds, A, B);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const float4 fj = __ldg(f32 + (int64_t)(r0 + q) * n + j);
      const float bxf = B * fmaf(dz, fj.z, fmaf(dy, fj.y, dx * fj.x));
      kahan_add(sx[q], cx[q], fmaf(A, fj.x, bxf * dx));
      kahan_add(sy[q], cy[q], fmaf(A, fj.y, bxf * dy));
      kahan_add(sz[q], cz[q], fmaf(A, fj.z, bxf * dz));
    }
  }
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    cx[q] = -cx[q];
    cy[q] = -cy[q];
    cz[q] = -cz[q];
    group_ff(sx[q], cx[q]);
    group_ff(sy[q], cy[q]);
    group_ff(sz[q], cz[q]);
    const int64_t roff = (int64_t)(r0 + q) * n * 3;
    group_store(act, sub, s, sx[q], cx[q], sy[q], cy[q], sz[q], cz[q], self_c, f + roff,
                u + roff);
  }
}

// ---- batched right-hand sides: 64 per pass, lanes over right-hand sides ----
//
// Forces of a pass are staged as FP32 [slot][3][64] (768 B per source, the
// pair (2l, 2l+1) of right-hand sides at float2 index l), so the 32 lanes of
// a warp read one source's forces with three coalesced 256-byte loads.  A
// warp owns one target slot: its lanes first evaluate the tensors of 32
// entries of the target's row at once (one entry per lane) into shared
// memory, then walk those entries with every lane updating its two
// right-hand sides in packed FP32x2 arithmetic.  Block-Kahan sums per lane;
// the CTA transposes the float-float results through shared memory so that
// the FP64 velocities [r][slot][3] (self term added in FP64) are written
// coalesced.
//
// Bound by the L1 data path (78% of its wavefronts), then by latency.  A
// broadcast of an entry's data takes 128 B per clock like any other load: as
// (x, x) pairs ready for the packed arithmetic an entry took 11 cycles of it,
// as single values 6, the pairs being made in registers (14-term step of N =
// 100k chains, 64 right-hand sides: 5.37 -> 4.97 ms).  The first three
// sources' forces are requested before the tensors are formed (4.93 ms), and
// a CTA holds four targets (4.70 ms; 2: 5.64, 5: 4.92, 8: 4.93, 16: 5.24):
// fewer wait for the longest row of theirs, and a write-out run is still 96
// bytes.  24 warps per SM instead of 32: 5.5 ms; 40, with spills: 6.9 ms.
constexpr int kBatchR = 64;      // right-hand sides per pass
constexpr int kBatchMinRhs = 16; // fewer go through k_pair_nr in chunks of 8
constexpr int kBatchWarps = 4;   // target slots per CTA

// elements whose loads a thread of the batched vector passes has in flight (a
// divisor of 64 * 96 / 256): one at a time waited out a DRAM latency each.  64
// right-hand sides of N = 100k, us: staging 59 -> 55, slots + staging 99 -> 83,
// start 176 -> 167
constexpr int kStageFly = 4;

__global__ void __launch_bounds__(256) k_stage_b64(int64_t n, int nr, const double *__restrict__ f,
                                                   float *__restrict__ fb) {
  // block: 32 slots x 64 right-hand sides; smem [r][96 + 1]
  __shared__ float t[kBatchR][97];
  const int64_t s0 = blockIdx.x * 32LL;
  const int ns = (int)(n - s0 < 32 ? n - s0 : 32);
#pragma unroll 1
  for (int k0 = threadIdx.x; k0 < kBatchR * 96; k0 += kStageFly * 256) {
    double v[kStageFly];
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96;
      v[i] = (r < nr && q < 3 * ns) ? f[((int64_t)r * n + s0) * 3 + q] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96;
      t[r][q] = d2f_bits(v[i]);
    }
  }
  __syncthreads();
  float *out = fb + s0 * 3 * kBatchR;
  for (int k = threadIdx.x; k < ns * 3 * kBatchR; k += blockDim.x) {
    const int sc = k / kBatchR, r = k - sc * kBatchR;
    out[k] = t[r][sc];
  }
}

// xi (caller order, [r][i][3]) into slot order (x0) and its batched FP32
// staging in one pass: k_to_slots followed by k_stage_b64
__global__ void __launch_bounds__(256) k_to_slots_b64(int64_t n, int nr,
                                                      const int32_t *__restrict__ order,
                                                      const double *__restrict__ xi,
                                                      double *__restrict__ x0,
                                                      float *__restrict__ fb) {
  __shared__ float t[kBatchR][97];
  const int64_t s0 = blockIdx.x * 32LL;
  const int ns = (int)(n - s0 < 32 ? n - s0 : 32);
#pragma unroll 1
  for (int k0 = threadIdx.x; k0 < kBatchR * 96; k0 += kStageFly * 256) {
    double v[kStageFly];
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96, sl = q / 3, c = q - 3 * sl;
      v[i] = r < nr && q < 3 * ns ? xi[((int64_t)r * n + order[s0 + sl]) * 3 + c] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96;
      if (r < nr && q < 3 * ns) x0[((int64_t)r * n + s0) * 3 + q] = v[i];
      t[r][q] = d2f_bits(v[i]);
    }
  }
  __syncthreads();
  float *out = fb + s0 * 3 * kBatchR;
  for (int k = threadIdx.x; k < ns * 3 * kBatchR; k += blockDim.x) {
    const int sc = k / kBatchR, r = k - sc * kBatchR;
    out[k] = t[r][sc];
  }
}

// The first step of a batched series in one pass (brownian_system.C:1041,
// 1050-1056): x1 = db x0 + da x1 (x1 holds M x0 on entry), dw = c0 x0 +
// c1 x1, and the batched FP32 staging of x1 for the first fused term
__global__ void __launch_bounds__(256) k_cheb_start_b64(int64_t n, int nr, double da, double db,
                                                        double c0, double c1,
                                                        const double *__restrict__ x0,
                                                        double *__restrict__ x1,
                                                        double *__restrict__ dw,
                                                        float *__restrict__ fb) {
  __shared__ float t[kBatchR][97];
  const int64_t s0 = blockIdx.x * 32LL;
  const int ns = (int)(n - s0 < 32 ? n - s0 : 32);
#pragma unroll 1
  for (int k0 = threadIdx.x; k0 < kBatchR * 96; k0 += kStageFly * 256) {
    double vx[kStageFly], vy[kStageFly];
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96;
      const int64_t idx = ((int64_t)r * n + s0) * 3 + q;
      const bool ok = r < nr && q < 3 * ns;
      vx[i] = ok ? x0[idx] : 0.0;
      vy[i] = ok ? x1[idx] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kStageFly; ++i) {
      const int k = k0 + 256 * i, r = k / 96, q = k - r * 96;
      const int64_t idx = ((int64_t)r * n + s0) * 3 + q;
      float v = 0.f;
      if (r < nr && q < 3 * ns) {
        const double y = db * vx[i] + da * vy[i];
        x1[idx] = y;
        const double c0x = c0 * vx[i];
        dw[idx] = c0x + c1 * y;
        v = d2f_bits(y);
      }
      t[r][q] = v;
    }
  }
  __syncthreads();
  float *out = fb + s0 * 3 * kBatchR;
  for (int k = threadIdx.x; k < ns * 3 * kBatchR; k += blockDim.x) {
    const int sc = k / kBatchR, r = k - sc * kBatchR;
    out[k] = t[r][sc];
  }
}

// forces of source slot j for the two right-hand sides of this lane
// (fw = fb + lane)
__device__ __forceinline__ void b64_fetch(const float2 *__restrict__ fw, uint32_t j, float2 &x,
                                          float2 &y, float2 &z) {
  const float2 *fp = fw + (int64_t)j * (3 * 32);
  x = __ldg(fp);
  y = __ldg(fp + 32);
  z = __ldg(fp + 64);
}

// blk += A f + B (x.f) x for both right-hand sides of the lane (packed)
__device__ __forceinline__ void b64_accumulate(const float4 &g, float B, const float2 &fx,
                                               const float2 &fy, const float2 &fz, float2 &b0,
                                               float2 &b1, float2 &b2) {
  const float2 dx2 = make_float2(g.x, g.x), dy2 = make_float2(g.y, g.y);
  const float2 dz2 = make_float2(g.z, g.z), A2 = make_float2(g.w, g.w);
  float2 d = __ffma2_rn(dz2, fz, __ffma2_rn(dy2, fy, __fmul2_rn(dx2, fx)));
  d = __fmul2_rn(make_float2(B, B), d);
  b0 = __ffma2_rn(d, dx2, __ffma2_rn(A2, fx, b0));
  b1 = __ffma2_rn(d, dy2, __ffma2_rn(A2, fy, b1));
  b2 = __ffma2_rn(d, dz2, __ffma2_rn(A2, fz, b2));
}

// block sums into the Kahan pairs, blocks cleared
__device__ __forceinline__ void b64_flush(float2 (&sum)[3], float2 (&cmp)[3], float2 &b0,
                                          float2 &b1, float2 &b2) {
  kahan_add(sum[0].x, cmp[0].x, b0.x);
  kahan_add(sum[0].y, cmp[0].y, b0.y);
  kahan_add(sum[1].x, cmp[1].x, b1.x);
  kahan_add(sum[1].y, cmp[1].y, b1.y);
  kahan_add(sum[2].x, cmp[2].x, b2.x);
  kahan_add(sum[2].y, cmp[2].y, b2.y);
  b0 = b1 = b2 = make_float2(0.f, 0.f);
}

// per right-hand side Chebyshev coefficient of a fused batched term (0 for
// a right-hand side whose series has stopped)
struct BatchCoef {
  double c[kBatchR];
};

// With CHEB the kernel is one unchecked Chebyshev term for up to 64
// right-hand sides (brownian_system.C:1091-1108, the order of k_cheb_term):
// u is x_{k+1}: u = (2db x1 + 2da M x1) - x0, dw += c_r u, and fb_next
// receives the FP32 staging of u for the next term.
template <int CD, bool POLY, bool CHEB>
__global__ void __launch_bounds__(32 * kBatchWarps, 8) k_pair_b64(
    int64_t n, int nr, const float4 *__restrict__ pos32, const float2 *__restrict__ fb,
    const int32_t *__restrict__ cnt, int W, const uint32_t *__restrict__ list, PolyAB P,
    const Rec32 *__restrict__ tab, float inv_ds, float hx, float hy, float hz, float self_hi,
    float self_lo, double *__restrict__ u, double two_da, double two_db, BatchCoef cf,
    const double *__restrict__ x0, const double *__restrict__ x1, double *__restrict__ dw,
    float *__restrict__ fb_next) {
  // per entry: (dx, dy, dz, A), B, source slot
  __shared__ float4 s_g[kBatchWarps][32];
  __shared__ float s_b[kBatchWarps][32];
  __shared__ uint32_t s_j[kBatchWarps][32];
  // float-float results; the padding puts a right-hand side's consecutive
  // (target, component) values in consecutive banks
  __shared__ float2 s_out[kBatchWarps][kBatchR + 1][3];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t s = blockIdx.x * (int64_t)kBatchWarps + w;
  const bool act = s < n;
  float2 sum[3], cmp[3];
  float2 blk0 = make_float2(0.f, 0.f), blk1 = blk0, blk2 = blk0;
#pragma unroll
  for (int c = 0; c < 3; ++c) sum[c] = cmp[c] = make_float2(0.f, 0.f);
  if (act) {
    // self term from the target's own staged forces, as a float-float
    // product with self_c = self_hi + self_lo
    {
      const float2 *fo = fb + s * (3 * 32);
      const float2 ch = make_float2(self_hi, self_hi), cl = make_float2(self_lo, self_lo);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float2 v = __ldg(fo + 32 * c + lane);
        const float2 pr = __fmul2_rn(ch, v);
        const float2 er = __ffma2_rn(cl, v, __ffma2_rn(ch, v, make_float2(-pr.x, -pr.y)));
        sum[c] = pr;
        cmp[c] = make_float2(-er.x, -er.y);  // Kahan keeps value = sum - cmp
      }
    }
    const float4 pi = pos32[s];
    const int64_t b = s * (int64_t)W;
    const int e = cnt[s];
    int nb = 0;
    for (int m0 = 0; m0 < e; m0 += 32) {
      const int np = min(32, e - m0);
      const uint32_t en = lane < np ? __ldg(list + b + m0 + lane) : 0u;
      const uint32_t j = en >> kCodeBits;
      // three force slots in flight: each is refilled with the entry three
      // ahead right after its own entry is used (no register rotation); the
      // first three are on their way while the tensors are formed
      const float2 *fw = fb + lane;
      float2 ax, ay, az, bx, by, bz, cx, cy, cz;
      b64_fetch(fw, __shfl_sync(0xffffffffu, j, 0), ax, ay, az);
      b64_fetch(fw, __shfl_sync(0xffffffffu, j, min(1, np - 1)), bx, by, bz);
      b64_fetch(fw, __shfl_sync(0xffffffffu, j, min(2, np - 1)), cx, cy, cz);
      if (lane < np) {
        const float4 pj = __ldg(pos32 + j);
        float ox, oy, oz;
        decode_shift<CD>(en, hx, hy, hz, ox, oy, oz);
        const float dx = (pj.x - pi.x) + ox, dy = (pj.y - pi.y) + oy, dz = (pj.z - pi.z) + oz;
        const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        float A, B;
        tensor_ab32<POLY>(s2, P, tab, inv_ds, A, B);
        s_g[w][lane] = make_float4(dx, dy, dz, A);
        s_b[w][lane] = B;
        s_j[w][lane] = j;
      }
      __syncwarp();
      const uint32_t *jw = s_j[w];
      for (int p = 0; p < np; p += 3) {
        b64_accumulate(s_g[w][p], s_b[w][p], ax, ay, az, blk0, blk1, blk2);
        b64_fetch(fw, jw[min(p + 3, np - 1)], ax, ay, az);
        if (p + 1 < np) {
          b64_accumulate(s_g[w][p + 1], s_b[w][p + 1], bx, by, bz, blk0, blk1,
                         blk2);
          b64_fetch(fw, jw[min(p + 4, np - 1)], bx, by, bz);
        }
        if (p + 2 < np) {
          b64_accumulate(s_g[w][p + 2], s_b[w][p + 2], cx, cy, cz, blk0, blk1,
                         blk2);
          b64_fetch(fw, jw[min(p + 5, np - 1)], cx, cy, cz);
        }
        if (++nb == 3) {  // every 9 entries into the compensated sums
          b64_flush(sum, cmp, blk0, blk1, blk2);
          nb = 0;
        }
      }
      __syncwarp();
    }
  }
  b64_flush(sum, cmp, blk0, blk1, blk2);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    s_out[w][2 * lane][c] = make_float2(sum[c].x, -cmp[c].x);
    s_out[w][2 * lane + 1][c] = make_float2(sum[c].y, -cmp[c].y);
  }
  __syncthreads();
  // coalesced FP64 write-out: per right-hand side, the CTA's targets'
  // 3 components are consecutive doubles; one FP64 add per value
  const int64_t s0 = blockIdx.x * (int64_t)kBatchWarps;
  const int ns = (int)(n - s0 < kBatchWarps ? n - s0 : kBatchWarps);
  constexpr int kRow = 3 * kBatchWarps;
  if (CHEB) {
    // x_{k+1} = 2da M x_k + (2db x_k - x_{k-1}), dw += c x_{k+1}: four FP64
    // operations per element with the add below (FP64 issues at a small
    // fraction of the FP32 rate on this GPU).  The vectors exceed L2, so
    // three elements' nine loads are in flight before the first is used (one
    // element at a time waited out three DRAM latencies per pass: 5.95 ->
    // 5.46 ms per 14-term step of N = 100k chains)
    constexpr int kFly = 3;
    const int total = nr * kRow;
    for (int k0 = threadIdx.x; k0 < total; k0 += kFly * 32 * kBatchWarps) {
      double va[kFly], vb[kFly], vd[kFly];
      int64_t at[kFly];
#pragma unroll
      for (int i = 0; i < kFly; ++i) {
        const int k = k0 + i * 32 * kBatchWarps, r = k / kRow, q = k - r * kRow;
        at[i] = k < total && q < 3 * ns ? ((int64_t)r * n + s0) * 3 + q : -1;
        if (at[i] >= 0) {
          va[i] = x0[at[i]];
          vb[i] = x1[at[i]];
          vd[i] = dw[at[i]];
        }
      }
#pragma unroll
      for (int i = 0; i < kFly; ++i) {
        if (at[i] < 0) continue;
        const int k = k0 + i * 32 * kBatchWarps, r = k / kRow, q = k - r * kRow;
        const int t = q / 3, c = q - t * 3;
        const float2 v = s_out[t][r][c];
        const double m = f2d_bits(v.x) + f2d_bits(v.y);
        const double x = fma(two_da, m, fma(two_db, vb[i], -va[i]));
        dw[at[i]] = fma(cf.c[r], x, vd[i]);
        u[at[i]] = x;
        // FP32 staging of x_{k+1}, transposed through shared memory below
        reinterpret_cast<float *>(&s_out[t][r][c])[0] = d2f_bits(x);
      }
    }
  } else {
    for (int k = threadIdx.x; k < nr * kRow; k += blockDim.x) {
      const int r = k / kRow, q = k - r * kRow;
      const int t = q / 3, c = q - t * 3;
      if (t >= ns) continue;
      const float2 v = s_out[t][r][c];
      u[((int64_t)r * n + s0) * 3 + q] = f2d_bits(v.x) + f2d_bits(v.y);
    }
  }
  if (CHEB) {
    __syncthreads();
    // staging layout [slot][3][64], right-hand sides fastest
    float *out = fb_next + s0 * 3 * kBatchR;
    for (int k = threadIdx.x; k < ns * 3 * kBatchR; k += blockDim.x) {
      const int sc = k / kBatchR, r = k - sc * kBatchR;
      const int t = sc / 3, c = sc - t * 3;
      out[k] = r < nr ? reinterpret_cast<const float *>(&s_out[t][r][c])[0] : 0.f;
    }
  }
}

__global__ void k_slots_to_f32(int64_t n, int nrhs, const double *__restrict__ f,
                               float4 *__restrict__ f32) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n * nrhs) return;
  const double *p = f + 3 * k;
  f32[k] = make_float4((float)p[0], (float)p[1], (float)p[2], 0.f);
}

// orig [r][n][3] -> slots [r][n][3]
__global__ void k_to_slots(int64_t n, int nrhs, const int32_t *__restrict__ order,
                           const double *__restrict__ orig, double *__restrict__ slot) {
  wait_prior_grid();
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n * nrhs) return;
  const int64_t r = k / n, s = k - r * n;
  const int64_t i = order[s];
  const double *src = orig + (r * n + i) * 3;
  double *dst = slot + (r * n + s) * 3;
  dst[0] = src[0];
  dst[1] = src[1];
  dst[2] = src[2];
}

__global__ void k_from_slots(int64_t n, int nrhs, const int32_t *__restrict__ rank,
                             const double *__restrict__ slot, double *__restrict__ orig) {
  wait_prior_grid();
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n * nrhs) return;
  const int64_t r = k / n, i = k - r * n;
  const int64_t s = rank[i];
  const double *src = slot + (r * n + s) * 3;
  double *dst = orig + (r * n + i) * 3;
  dst[0] = src[0];
  dst[1] = src[1];
  dst[2] = src[2];
}

MinImage min_image_of(const Grid &g) {
  MinImage m;
  for (int d = 0; d < 3; ++d) {
    const double half = g.periodic[d] ? g.L[d] / 2.0 : INFINITY;
    std::memcpy(&m.half[d], &half, 8);
    std::memcpy(&m.L[d], &g.L[d], 8);
  }
  return m;
}

template <int NR, int G>
void launch_list_f64(ggem_ctx *c, const double *f, double *u, int self_mode, int r0,
                     long long eps2) {
  const int64_t threads = c->n * G;
  launch_dependent(k_pair_list_f64<NR, G>, dim3((unsigned)((threads + 255) / 256)), 256, 0,
                   c->stream, 
      c->n, min_image_of(c->grid), c->dc, c->t64, eps2, c->nb_cnt.p, c->nb_w, c->nb_list.p,
      c->pos64.p, f, u, self_mode, r0);
}

template <int NR>
int launch_f64(ggem_ctx *c, const double *f, double *u, int self_mode, int r0) {
  long long eps2;
  const double e2 = c->dc.r_eps * c->dc.r_eps;
  std::memcpy(&eps2, &e2, 8);
  kt_start(c, kKPairF64);
  // (a caller's graph outlives this configuration: it holds the sweep, whose
  // buffers depend on the particle count alone, not a list of this width)
  if (c->list_built && !(c->f64_list_is_own() && stream_capturing(c))) {
    // lanes per target: four fill the FP64 pipe from ~80k targets on (fewer
    // lanes would idle in rows of ~35 entries of uneven length); smaller
    // counts need more lanes to cover the latency of a row walk.  us per
    // kernel with 4 / 8 / 16 / 32 lanes, phi = 0.1: N = 1000 (phi 0.05) 20 / 14
    // / 12 / 10, 2000 31 / 19 / 14 / 18, 4000 31 / 20 / 22 / 29, 12000 50 / 42 /
    // 46 / 60, 40000 110 / 108 / 125 / 174, 80000 189 / 197 / 236 / 334, 200000
    // 426 / 464 / 570 / 813; element lists of 1000 47 / 28 / 19 / 14, of 20000
    // 129 / 111 / 110 / 131
    if (c->n >= 80000) launch_list_f64<NR, 4>(c, f, u, self_mode, r0, eps2);
    else if (c->n >= 2500) launch_list_f64<NR, 8>(c, f, u, self_mode, r0, eps2);
    else launch_list_f64<NR, 32>(c, f, u, self_mode, r0, eps2);
    kt_stop(c, kKPairF64);
    return check_launch(c, "matvec f64 list");
  }
  const int T = 128;
  const unsigned bn = (unsigned)((c->n + T - 1) / T);
  const bool ref = c->prm.nb_mode == GGEM_NB_REFERENCE;
  k_matvec_f64<NR><<<bn, T, 0, c->stream>>>(c->n, c->grid, c->dc, c->t64, c->d_stencil.p,
                                             (int)c->stencil.size(), ref ? 1 : 0, ref ? 0 : 1,
                                             c->rc2, eps2, c->cell_start.p, c->pos64.p,
                                             c->pos32.p, f, u, self_mode, r0);
  kt_stop(c, kKPairF64);
  return check_launch(c, "matvec f64");
}

// at most max_rounds targets per group of lanes; *done = false: more, or no
// cooperative launch
template <int G, int CACHE>
int launch_series_f64(ggem_ctx *c, SeriesF64 &a, int max_rounds, bool *done) {
  int sms = 0, per = 0, coop = 0;
  cudaError_t e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device)) ||
      (e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device)) ||
      (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_series_f64<G, CACHE>,
                                                          kSeriesThreads, 0)))
    return cuda_fail(c, e, "series occupancy");
  if (!coop || per < 1) return GGEM_OK;
  const int64_t kt = kSeriesThreads / G, most = (int64_t)sms * per;
  a.rounds = (int)((a.n + most * kt - 1) / (most * kt));
  if (a.rounds > max_rounds) return GGEM_OK;
  // the same number of rounds in every block
  const unsigned grid = (unsigned)((a.n + a.rounds * kt - 1) / (a.rounds * kt));
  if ((e = c->w_red.ensure((size_t)3 * grid))) return cuda_fail(c, e, "series partials");
  a.part = c->w_red.p;
  void *args[] = {&a};
  if ((e = cudaLaunchCooperativeKernel((const void *)k_series_f64<G, CACHE>, dim3(grid),
                                       dim3(kSeriesThreads), args, 0, c->stream)))
    return cuda_fail(c, e, "series launch");
  *done = true;
  return check_launch(c, "series f64");
}

PolyAB poly_of(const ggem_ctx *c) {
  PolyAB P;
  for (int q = 0; q <= kPolyDeg; ++q) P.ab[q] = make_float2(c->poly_a[q], c->poly_b[q]);
  P.x0 = c->poly_x0;
  P.x1 = c->poly_x1;
  P.e_hi = c->poly_e[0];
  P.e_lo = c->poly_e[1];
  return P;
}

template <bool POLY, int V, bool ORIG>
void launch_r1(ggem_ctx *c, const Rec32 *src, const double *f, double *u, double self_c,
               double *part) {
  launch_dependent(k_pair_r1<POLY, V, ORIG>, dim3(pair_grid_blocks(c)), 256, 0, c->stream,
                   c->n, src, (const int32_t *)c->nb_cnt.p, c->nb_w, (const uint32_t *)c->nb_list.p,
                   poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds,
                   (const float4 *)c->d_shift.p, self_c, f, u, (const int32_t *)c->order.p, part);
}

template <bool POLY, bool ORIG = false>
void dispatch_r1(ggem_ctx *c, const Rec32 *src, const double *f, double *u, double self_c,
                 double *part = nullptr) {
  if (c->computed_variant == 1) launch_r1<POLY, 1, ORIG>(c, src, f, u, self_c, part);
  else launch_r1<POLY, 0, ORIG>(c, src, f, u, self_c, part);
}

// single right-hand side: records from FP64 slot-order f, then the pair sum
// u = M f for one right-hand side from the half list (k_pair_sym +
// k_sym_finish); src holds the records of f
int launch_sym_r1(ggem_ctx *c, const Rec32 *src, const double *f, double *u, double self_c) {
  const int64_t n = c->n;
  cudaError_t e;
  if (c->sym_acc.count < (size_t)n) {
    if ((e = c->sym_acc.ensure((size_t)n)) ||
        (e = cudaMemsetAsync(c->sym_acc.p, 0, sizeof(float4) * c->sym_acc.count, c->stream)))
      return cuda_fail(c, e, "symmetric accumulators");
  }
  if ((e = c->sym_part.ensure(3 * (size_t)n))) return cuda_fail(c, e, "symmetric sums");
  const unsigned nb = (unsigned)((n * kGroup + 255) / 256);
  kt_start(c, kKPairF32);
  if (c->use_poly)
    k_pair_sym<true><<<nb, 256, 0, c->stream>>>(
        n, src, c->nb_cnt_h.p, c->nb_w, c->nb_list_h.p, poly_of(c),
        reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds, c->d_shift.p, c->sym_acc.p,
        c->sym_part.p);
  else
    k_pair_sym<false><<<nb, 256, 0, c->stream>>>(
        n, src, c->nb_cnt_h.p, c->nb_w, c->nb_list_h.p, poly_of(c),
        reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds, c->d_shift.p, c->sym_acc.p,
        c->sym_part.p);
  if (int rc = check_launch(c, "pair f32 symmetric")) return rc;
  k_sym_finish<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(n, c->sym_part.p, c->sym_acc.p,
                                                                  self_c, f, u);
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32 symmetric finish");
}

void launch_stored_first(ggem_ctx *c, const float4 *f4, double self_c, const double *f,
                         double *u, const int32_t *order) {
  const Grid &g = c->grid;
  const bool cd2 = c->prm.cell_div == 2;
  launch_dependent(
      c->use_poly ? (cd2 ? k_pair_r1tv_first<2, true, 2> : k_pair_r1tv_first<1, true, 2>)
                  : (cd2 ? k_pair_r1tv_first<2, false, 2> : k_pair_r1tv_first<1, false, 2>),
      dim3((unsigned)((c->n * kGroup + 255) / 256)), 256, 0, c->stream, c->n, c->pos32.p, f4,
      c->nb_cnt.p, c->nb_w, c->nb_list.p, poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p),
      c->tab_inv_ds, g.h32[0], g.h32[1], g.h32[2], c->pair_ten.p, self_c, f, u, order);
}

// u = M f from the stored tensors, the FP32 forces staged in w_f4 (order: u
// in the caller's particle order)
int stored_product(ggem_ctx *c, double self_c, const double *f, double *u, const int32_t *order) {
  const bool capturing = stream_capturing(c);
  if (capturing) c->pretensor_eager = true;
  if (kStoredVariants[c->stored_variant].G != kGroup)
    if (int rc = form_pair_tensors(c)) return rc;
  kt_start(c, kKPairF32);
  if (c->pretensor_pending && kStoredVariants[c->stored_variant].G == kGroup) {
    launch_stored_first(c, c->w_f4[0].p, self_c, f, u, order);
    // (a captured product forms them whenever it is replayed)
    c->pretensor_pending = capturing;
  } else {
    dispatch_stored_r1(c, c->w_f4[0].p, self_c, f, u, order);
  }
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32 r1 (tensors)");
}

int launch_f32_r1(ggem_ctx *c, const double *f, double *u, double self_c) {
  const int64_t n = c->n;
  cudaError_t e;
  if (c->pretensor_ok) {
    if ((e = c->w_f4[0].ensure((size_t)n))) return cuda_fail(c, e, "pair forces");
    launch_dependent(k_stage_f4, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, f, c->w_f4[0].p);
    if (int rc = check_launch(c, "pair forces")) return rc;
    return stored_product(c, self_c, f, u, nullptr);
  }
  if ((e = c->w_src.ensure(2 * (size_t)n))) return cuda_fail(c, e, "pair records");
  Rec32 *src = reinterpret_cast<Rec32 *>(c->w_src.p);
  launch_dependent(k_build_src, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, c->pos32.p, f, src);
  if (int rc = check_launch(c, "pair records")) return rc;
  if (c->sym_pairs && c->nb_list_h.p) return launch_sym_r1(c, src, f, u, self_c);
  kt_start(c, kKPairF32);
  if (c->use_poly) dispatch_r1<true>(c, src, f, u, self_c);
  else dispatch_r1<false>(c, src, f, u, self_c);
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32 r1");
}

// c1 = 2db + 2da self_c folds the self term into the x1 coefficient
template <bool POLY, int V, bool NORMS>
void launch_cheb(ggem_ctx *c, const Rec32 *src, Rec32 *next, double two_da, double c1,
                 double coef, const double *x0, const double *x1, double *xm, double *dw,
                 double *part, Rec32 *dw_next) {
  launch_dependent(k_pair_cheb<POLY, V, NORMS>, dim3(pair_grid_blocks(c)), 256, 0, c->stream,
                   c->n, src, (const int32_t *)c->nb_cnt.p, c->nb_w, (const uint32_t *)c->nb_list.p,
                   poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds,
                   (const float4 *)c->d_shift.p, two_da, c1, coef, x0, x1, xm, dw, next, part,
                   pair_partials(c), dw_next);
}

// with part (and dw_next) the term also leaves the estimators' two norms as
// per-block partials and the records of the new dw
template <bool POLY>
void dispatch_cheb(ggem_ctx *c, const Rec32 *src, Rec32 *next, double two_da, double c1,
                   double coef, const double *x0, const double *x1, double *xm, double *dw,
                   double *part, Rec32 *dw_next) {
  const bool v1 = c->computed_variant == 1;
  if (part) {
    if (v1) launch_cheb<POLY, 1, true>(c, src, next, two_da, c1, coef, x0, x1, xm, dw, part, dw_next);
    else launch_cheb<POLY, 0, true>(c, src, next, two_da, c1, coef, x0, x1, xm, dw, part, dw_next);
  } else {
    if (v1) launch_cheb<POLY, 1, false>(c, src, next, two_da, c1, coef, x0, x1, xm, dw, part, dw_next);
    else launch_cheb<POLY, 0, false>(c, src, next, two_da, c1, coef, x0, x1, xm, dw, part, dw_next);
  }
}

template <bool POLY, int V>
void launch_first(ggem_ctx *c, const Rec32 *src, Rec32 *next, double self_c, double da,
                  double db, double c0, double c1, const double *x0, double *m, double *x1,
                  double *dw, double *part) {
  launch_dependent(k_pair_first<POLY, V>, dim3(pair_grid_blocks(c)), 256, 0, c->stream, c->n,
                   src, (const int32_t *)c->nb_cnt.p, c->nb_w, (const uint32_t *)c->nb_list.p,
                   poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds,
                   (const float4 *)c->d_shift.p, self_c, da, db, c0, c1, x0, m, x1, dw, next,
                   part);
}

template <int CD, bool POLY>
void launch_b64_t(ggem_ctx *c, int nr, const double *f, double *u, double self_c) {
  const Grid &g = c->grid;
  const unsigned grid = (unsigned)((c->n + kBatchWarps - 1) / kBatchWarps);
  k_pair_b64<CD, POLY, false><<<grid, 32 * kBatchWarps, 0, c->stream>>>(
      c->n, nr, c->pos32.p, reinterpret_cast<const float2 *>(c->w_fb.p), c->nb_cnt.p, c->nb_w,
      c->nb_list.p, poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds,
      g.h32[0], g.h32[1], g.h32[2], (float)self_c, (float)(self_c - (double)(float)self_c), u,
      0.0, 0.0, BatchCoef{}, nullptr, nullptr, nullptr, nullptr);
}

template <int CD, bool POLY>
void launch_b64_cheb(ggem_ctx *c, int nr, const float *fb, float *fb_next, double self_c,
                     double two_da, double two_db, const BatchCoef &cf, const double *x0,
                     const double *x1, double *xm, double *dw) {
  const Grid &g = c->grid;
  const unsigned grid = (unsigned)((c->n + kBatchWarps - 1) / kBatchWarps);
  k_pair_b64<CD, POLY, true><<<grid, 32 * kBatchWarps, 0, c->stream>>>(
      c->n, nr, c->pos32.p, reinterpret_cast<const float2 *>(fb), c->nb_cnt.p, c->nb_w,
      c->nb_list.p, poly_of(c), reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds,
      g.h32[0], g.h32[1], g.h32[2], (float)self_c, (float)(self_c - (double)(float)self_c), xm,
      two_da, two_db, cf, x0, x1, dw, fb_next);
}

// many right-hand sides: passes of 64 (k_stage_b64 + k_pair_b64)
// (staged: w_fb already holds the FP32 staging of f, one pass of at most 64)
int matvec_b64(ggem_ctx *c, int nrhs, const double *f, double *u, double self_c,
               bool staged = false) {
  const int64_t n = c->n;
  cudaError_t e = c->w_fb.ensure((size_t)n * 3 * kBatchR);
  if (e) return cuda_fail(c, e, "batched staging");
  const bool cd2 = c->prm.cell_div == 2;
  for (int r0 = 0; r0 < nrhs; r0 += kBatchR) {
    const int nr = std::min(kBatchR, nrhs - r0);
    const double *fr = f + (int64_t)r0 * n * 3;
    double *ur = u + (int64_t)r0 * n * 3;
    if (!staged) {
      k_stage_b64<<<(unsigned)((n + 31) / 32), 256, 0, c->stream>>>(n, nr, fr, c->w_fb.p);
      if (int rc = check_launch(c, "batched staging")) return rc;
    }
    kt_start(c, kKPairF32);
    if (c->use_poly) cd2 ? launch_b64_t<2, true>(c, nr, fr, ur, self_c)
                         : launch_b64_t<1, true>(c, nr, fr, ur, self_c);
    else cd2 ? launch_b64_t<2, false>(c, nr, fr, ur, self_c)
             : launch_b64_t<1, false>(c, nr, fr, ur, self_c);
    kt_stop(c, kKPairF32);
    if (int rc = check_launch(c, "pair f32 batched")) return rc;
  }
  return GGEM_OK;
}

template <int CD, bool POLY, int NR>
void launch_nr_t(ggem_ctx *c, const double *f, double *u, double self_c, int r0) {
  const int64_t threads = c->n * kGroup;
  const Grid &g = c->grid;
  k_pair_nr<CD, POLY, NR><<<(unsigned)((threads + 255) / 256), 256, 0, c->stream>>>(
      c->n, c->pos32.p, c->w_f32.p, c->nb_cnt.p, c->nb_w, c->nb_list.p, poly_of(c),
      reinterpret_cast<const Rec32 *>(c->tab.p), c->tab_inv_ds, g.h32[0], g.h32[1], g.h32[2],
      self_c, f, u, r0);
}

template <int NR>
int launch_nr(ggem_ctx *c, const double *f, double *u, double self_c, int r0) {
  const bool cd2 = c->prm.cell_div == 2;
  kt_start(c, kKPairF32);
  if (c->use_poly) {
    if (cd2) launch_nr_t<2, true, NR>(c, f, u, self_c, r0);
    else launch_nr_t<1, true, NR>(c, f, u, self_c, r0);
  } else {
    if (cd2) launch_nr_t<2, false, NR>(c, f, u, self_c, r0);
    else launch_nr_t<1, false, NR>(c, f, u, self_c, r0);
  }
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32");
}

}  // namespace

int permute_to_slots(ggem_ctx *c, int nrhs, const double *d_orig, double *d_slot) {
  const int64_t tot = c->n * nrhs;
  if (tot == 0) return GGEM_OK;
  launch_dependent(k_to_slots, dim3((unsigned)((tot + 255) / 256)), 256, 0, c->stream,
                   c->n, nrhs, c->order.p,
                                                                   d_orig, d_slot);
  return check_launch(c, "to slots");
}

int permute_from_slots(ggem_ctx *c, int nrhs, const double *d_slot, double *d_orig) {
  const int64_t tot = c->n * nrhs;
  if (tot == 0) return GGEM_OK;
  launch_dependent(k_from_slots, dim3((unsigned)((tot + 255) / 256)), 256, 0, c->stream,
                   c->n, nrhs, c->rank.p,
                                                                     d_slot, d_orig);
  return check_launch(c, "from slots");
}

// One fused Chebyshev term on the FP32 single-RHS path (k_pair_cheb).
// records_fresh: c->w_rec[c->rec_cur] already holds the records of x1 (the
// previous fused term wrote them); otherwise they are built here first.
int pair_cheb_term(ggem_ctx *c, bool records_fresh, const double *x0, const double *x1,
                   double *xm, double *dw, double two_da, double two_db, double coef,
                   int self_mode, double *norms) {
  const int64_t n = c->n;
  if (n == 0) return GGEM_OK;
  cudaError_t e;
  const double self_c0 = self_coefficient(c, self_mode);
  if (c->pretensor_ok) {
    if (int rc = form_pair_tensors(c)) return rc;
    if (norms) return fail(c, GGEM_ERR_BAD_ARG, "fused norms need per-matvec pair tensors");
    if ((e = c->w_f4[0].ensure((size_t)n)) || (e = c->w_f4[1].ensure((size_t)n)))
      return cuda_fail(c, e, "chebyshev forces");
    float4 *cur = c->w_f4[c->rec_cur].p, *nxt = c->w_f4[c->rec_cur ^ 1].p;
    if (!records_fresh) {
      launch_dependent(k_stage_f4, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, x1, cur);
      if (int rc = check_launch(c, "chebyshev forces")) return rc;
    }
    kt_start(c, kKPairCheb);
    dispatch_stored_cheb(c, cur, self_c0, two_da, two_db, coef, x0, x1, xm, dw, nxt);
    kt_stop(c, kKPairCheb);
    c->rec_cur ^= 1;
    return check_launch(c, "pair chebyshev term (tensors)");
  }
  if ((e = c->w_rec[0].ensure(2 * (size_t)n)) || (e = c->w_rec[1].ensure(2 * (size_t)n)))
    return cuda_fail(c, e, "chebyshev records");
  Rec32 *cur = reinterpret_cast<Rec32 *>(c->w_rec[c->rec_cur].p);
  Rec32 *nxt = reinterpret_cast<Rec32 *>(c->w_rec[c->rec_cur ^ 1].p);
  if (!records_fresh) {
    launch_dependent(k_build_src, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, c->pos32.p, x1, cur);
    if (int rc = check_launch(c, "chebyshev records")) return rc;
  }
  const double c1 = two_db + two_da * self_c0;
  // a checked term leaves the records of the new dw in w_src for the check
  // matvec (matvec_dw_records)
  Rec32 *dwr = nullptr;
  if (norms) {
    if ((e = c->w_src.ensure(2 * (size_t)n))) return cuda_fail(c, e, "pair records");
    dwr = reinterpret_cast<Rec32 *>(c->w_src.p);
  }
  kt_start(c, kKPairCheb);
  if (c->use_poly) dispatch_cheb<true>(c, cur, nxt, two_da, c1, coef, x0, x1, xm, dw, norms, dwr);
  else dispatch_cheb<false>(c, cur, nxt, two_da, c1, coef, x0, x1, xm, dw, norms, dwr);
  kt_stop(c, kKPairCheb);
  c->rec_cur ^= 1;
  return check_launch(c, "pair chebyshev term");
}

// (the batched kernels evaluate their tensors per pair whether or not the
// single-RHS path stores them)
bool batch_term_fusable(const ggem_ctx *c, int nrhs) {
  return nrhs >= kBatchMinRhs && nrhs <= kBatchR && c->prm.precision == GGEM_FP32 &&
         c->prm.nb_mode == GGEM_NB_CUTOFF;
}

// One unchecked Chebyshev term for 16 .. 64 right-hand sides in one kernel
// (k_pair_b64 with the recurrence in its write-out).  staged_fresh:
// c->w_fb holds the FP32 staging of x1 (the previous fused term wrote it);
// otherwise it is staged here first.  coef[r] is 0 for a stopped series.
int batch_cheb_term(ggem_ctx *c, int nrhs, bool staged_fresh, const double *x0, const double *x1,
                    double *xm, double *dw, double two_da, double two_db, const double *coef,
                    int self_mode) {
  const int64_t n = c->n;
  if (n == 0) return GGEM_OK;
  cudaError_t e;
  if ((e = c->w_fb.ensure((size_t)n * 3 * kBatchR)) || (e = c->w_fb2.ensure((size_t)n * 3 * kBatchR)))
    return cuda_fail(c, e, "batched staging");
  if (!staged_fresh) {
    k_stage_b64<<<(unsigned)((n + 31) / 32), 256, 0, c->stream>>>(n, nrhs, x1, c->w_fb.p);
    if (int rc = check_launch(c, "batched staging")) return rc;
  }
  BatchCoef cf{};
  for (int r = 0; r < nrhs; ++r) cf.c[r] = coef[r];
  const double self_c = self_coefficient(c, self_mode);
  const bool cd2 = c->prm.cell_div == 2;
  kt_start(c, kKPairCheb);
  if (c->use_poly) {
    if (cd2) launch_b64_cheb<2, true>(c, nrhs, c->w_fb.p, c->w_fb2.p, self_c, two_da, two_db, cf, x0, x1, xm, dw);
    else launch_b64_cheb<1, true>(c, nrhs, c->w_fb.p, c->w_fb2.p, self_c, two_da, two_db, cf, x0, x1, xm, dw);
  } else {
    if (cd2) launch_b64_cheb<2, false>(c, nrhs, c->w_fb.p, c->w_fb2.p, self_c, two_da, two_db, cf, x0, x1, xm, dw);
    else launch_b64_cheb<1, false>(c, nrhs, c->w_fb.p, c->w_fb2.p, self_c, two_da, two_db, cf, x0, x1, xm, dw);
  }
  kt_stop(c, kKPairCheb);
  std::swap(c->w_fb.p, c->w_fb2.p);  // the staging of x_{k+1} is the next term's x1
  std::swap(c->w_fb.count, c->w_fb2.count);
  return check_launch(c, "pair chebyshev term (batched)");
}

int pair_grid_blocks(const ggem_ctx *c) {
  return (int)std::max<int64_t>(1, (c->n * kGroup + 255) / 256);
}

int64_t pair_partials(const ggem_ctx *c) { return pair_grid_blocks(c); }

// The first step of a fused series: xi (caller order) into slot order (x0)
// with its records, then k_pair_first (m = M x0, x1, dw and the records of
// x1 for the first term).
int cheb_start_fused(ggem_ctx *c, const double *xi, double *x0, double *m, double *x1,
                     double *dw, double da, double db, double c0, double c1, int self_mode,
                     double *aux2) {
  const int64_t n = c->n;
  if (n == 0) return GGEM_OK;
  if (c->pretensor_ok) return fail(c, GGEM_ERR_BAD_ARG, "fused start needs per-matvec pair tensors");
  cudaError_t e;
  if ((e = c->w_rec[0].ensure(2 * (size_t)n)) || (e = c->w_rec[1].ensure(2 * (size_t)n)))
    return cuda_fail(c, e, "chebyshev records");
  Rec32 *cur = reinterpret_cast<Rec32 *>(c->w_rec[c->rec_cur].p);
  Rec32 *nxt = reinterpret_cast<Rec32 *>(c->w_rec[c->rec_cur ^ 1].p);
  launch_dependent(k_to_slots_rec, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, c->order.p, c->pos32.p,
                                                                     xi, x0, cur);
  if (int rc = check_launch(c, "to slots + records")) return rc;
  const double self_c = self_coefficient(c, self_mode);
  kt_start(c, kKPairF32);
  const bool v1 = c->computed_variant == 1;
  if (c->use_poly) {
    if (v1) launch_first<true, 1>(c, cur, nxt, self_c, da, db, c0, c1, x0, m, x1, dw, aux2);
    else launch_first<true, 0>(c, cur, nxt, self_c, da, db, c0, c1, x0, m, x1, dw, aux2);
  } else {
    if (v1) launch_first<false, 1>(c, cur, nxt, self_c, da, db, c0, c1, x0, m, x1, dw, aux2);
    else launch_first<false, 0>(c, cur, nxt, self_c, da, db, c0, c1, x0, m, x1, dw, aux2);
  }
  kt_stop(c, kKPairF32);
  c->rec_cur ^= 1;
  return check_launch(c, "pair first step");
}

// u = M dw after a checked fused term: the term left the records of dw in
// w_src, so the check matvec is one launch, and |u|^2 leaves as per-block
// partials (norm)
int matvec_dw_records(ggem_ctx *c, const double *dw, double *u, int self_mode, double *norm) {
  return matvec_records(c, c->w_src.p, dw, u, self_mode, norm);
}

// u = M f from the 32-byte records of f already staged in rec (2 float4 per
// slot: the cell-relative position, then the FP32 force), f in slot order
int matvec_records(ggem_ctx *c, const float4 *rec, const double *f, double *u, int self_mode,
                   double *norm) {
  if (c->n == 0) return GGEM_OK;
  const Rec32 *src = reinterpret_cast<const Rec32 *>(rec);
  const double self_c = self_coefficient(c, self_mode);
  kt_start(c, kKPairF32);
  if (c->use_poly) dispatch_r1<true>(c, src, f, u, self_c, norm);
  else dispatch_r1<false>(c, src, f, u, self_c, norm);
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32 r1");
}

// u = M f for one right-hand side with f and u in the caller's particle
// order (FP32 list): the slot permutation of f is fused with the staging of
// its FP32 forces (k_to_slots_rec, k_to_slots_f4) and the pair kernel writes
// u in caller order, so a matvec is two launches.  f_slot receives f in slot
// order (the self term reads it).  N = 400k with stored tensors, list
// included: 307 -> 298 us against four launches.
int matvec_orig_fused(ggem_ctx *c, const double *f, double *u, double *f_slot, int self_mode) {
  const int64_t n = c->n;
  if (n == 0) return GGEM_OK;
  if (c->pretensor_ok) {
    if (cudaError_t e = c->w_f4[0].ensure((size_t)n)) return cuda_fail(c, e, "pair forces");
    launch_dependent(k_to_slots_f4, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream, n,
                     c->order.p, f, f_slot, c->w_f4[0].p);
    if (int rc = check_launch(c, "to slots + forces")) return rc;
    return stored_product(c, self_coefficient(c, self_mode), f_slot, u, c->order.p);
  }
  cudaError_t e = c->w_src.ensure(2 * (size_t)n);
  if (e) return cuda_fail(c, e, "pair records");
  Rec32 *src = reinterpret_cast<Rec32 *>(c->w_src.p);
  launch_dependent(k_to_slots_rec, dim3((unsigned)((n + 255) / 256)), 256, 0, c->stream,
                   n, c->order.p, c->pos32.p,
                                                                     f, f_slot, src);
  if (int rc = check_launch(c, "to slots + records")) return rc;
  const double self_c = self_coefficient(c, self_mode);
  kt_start(c, kKPairF32);
  if (c->use_poly) dispatch_r1<true, true>(c, src, f_slot, u, self_c);
  else dispatch_r1<false, true>(c, src, f_slot, u, self_c);
  kt_stop(c, kKPairF32);
  return check_launch(c, "pair f32 r1");
}

// The per-pair tensors of the current list: room for them now, the tensors
// themselves with the first product that reads them (k_pair_r1tv_first), or
// by form_pair_tensors where another kernel comes first.  A graph that a
// caller captured may read the stored tensors when it is replayed, so from
// the first captured product on they are formed with the list.
int build_pair_tensors(ggem_ctx *c) {
  c->pretensor_ok = c->pretensor_pending = false;
  if (!c->use_pretensor || !c->allow_pretensor || !c->list_built) return GGEM_OK;
  if (c->n > 0) {
    cudaError_t e = c->pair_ten.ensure((size_t)c->n * c->nb_w);
    if (e) {
      // no room for the tensors: the pair kernels evaluate them on the fly
      cudaGetLastError();
      return GGEM_OK;
    }
  }
  c->pretensor_ok = true;
  c->pretensor_pending = c->n > 0;
  return c->pretensor_eager ? form_pair_tensors(c) : GGEM_OK;
}

int form_pair_tensors(ggem_ctx *c) {
  if (!c->pretensor_pending) return GGEM_OK;
  const Grid &g = c->grid;
  const unsigned grid = (unsigned)((c->n * kGroup + 255) / 256);
  const bool cd2 = c->prm.cell_div == 2;
  const Rec32 *tab = reinterpret_cast<const Rec32 *>(c->tab.p);
  kt_start(c, kKListBuild);
  launch_dependent(c->use_poly ? (cd2 ? k_pair_tensor<2, true> : k_pair_tensor<1, true>)
                               : (cd2 ? k_pair_tensor<2, false> : k_pair_tensor<1, false>),
                   dim3(grid), 256, 0, c->stream, c->n, c->pos32.p, c->nb_cnt.p, c->nb_w,
                   c->nb_list.p, poly_of(c), tab, c->tab_inv_ds, g.h32[0], g.h32[1], g.h32[2],
                   c->pair_ten.p);
  kt_stop(c, kKListBuild);
  if (int rc = check_launch(c, "pair tensors")) return rc;
  const bool capturing = stream_capturing(c);
  if (capturing) c->pretensor_eager = true;
  c->pretensor_pending = capturing;
  return GGEM_OK;
}

void batch_tensors(const BatchBuild &b, const ggem_ctx *like, cudaStream_t st) {
  const unsigned grid = (unsigned)((b.ntot * kGroup + 255) / 256);
  const Rec32 *tab = reinterpret_cast<const Rec32 *>(like->tab.p);
  const bool cd2 = like->prm.cell_div == 2;
  auto launch = [&](auto kernel) {
    kernel<<<grid, 256, 0, st>>>(b.ntot, b.geo, b.susp, b.pos32, b.cnt, b.W, b.list, poly_of(like),
                                 tab, like->tab_inv_ds, b.ten);
  };
  if (like->use_poly) cd2 ? launch(k_batch_tensor<2, true>) : launch(k_batch_tensor<1, true>);
  else cd2 ? launch(k_batch_tensor<2, false>) : launch(k_batch_tensor<1, false>);
}

double self_coefficient(const ggem_ctx *c, int self_mode) {
  if (self_mode == GGEM_SELF_BEAD) return 1.0 - c->cst.coeff_1;
  if (self_mode == GGEM_SELF_LAGRANGIAN) return c->cst.coeff_2;
  return 0.0;
}

// The whole FP64 series of one right-hand side (k_series_f64): xi and out in
// caller order (y stays in the series' own records).  *done = false: not taken
// (no pair list, the kernel timer or the launch trace wants the single
// launches, a deferred list build to be checked first, or no cooperative
// launch).
int series_f64(ggem_ctx *c, int N, const double *coef, double da, double db, double tol,
               int check_every, int k_first, int self_mode, const double *xi, double *out,
               bool out_y, ggem_cheb_report *rep, int *first_check, bool *done) {
  *done = false;
  if (c->prm.precision != GGEM_FP64 || c->timing || c->trace || c->n == 0) return GGEM_OK;
  if (int rc = ensure_f64_list(c)) return rc;
  if (!c->list_built || c->list_unchecked) return GGEM_OK;
  cudaError_t e;
  // control block and coefficients in one upload, through pinned memory
  // where they fit the context's mirror
  constexpr int kCtl = (sizeof(SeriesCtl) + 7) / 8;
  const size_t words = kCtl + N + 1;
  if ((e = c->s64_tab.ensure(words))) return cuda_fail(c, e, "series tables");
  std::vector<double> big;
  double *up = c->h_red + 64;
  if (words > 3072) {
    big.resize(words);
    up = big.data();
  }
  SeriesCtl ctl;
  std::memset(&ctl, 0, sizeof(ctl));
  ctl.first_check = -1;
  std::memcpy(up, &ctl, sizeof(ctl));
  std::memcpy(up + kCtl, coef, sizeof(double) * (N + 1));
  if ((e = cudaMemcpyAsync(c->s64_tab.p, up, sizeof(double) * words, cudaMemcpyHostToDevice,
                           c->stream)))
    return cuda_fail(c, e, "series tables");
  SeriesF64 a;
  a.n = c->n;
  a.W = c->nb_w;
  a.N = N;
  a.self_mode = self_mode;
  a.check_every = check_every;
  a.k_first = k_first;
  a.out_y = out_y ? 1 : 0;
  a.polls = c->series_polls;
  a.da = da;
  a.db = db;
  a.tol = tol;
  a.mi = min_image_of(c->grid);
  a.K = c->dc;
  a.T = c->t64;
  const double e2 = c->dc.r_eps * c->dc.r_eps;
  std::memcpy(&a.eps2, &e2, 8);
  a.cnt = c->nb_cnt.p;
  a.order = c->order.p;
  a.list = c->nb_list.p;
  a.pos64 = c->pos64.p;
  a.coef = c->s64_tab.p + kCtl;
  a.xi = xi;
  if ((e = c->s64_vec.ensure(5 * (size_t)c->n))) return cuda_fail(c, e, "series vectors");
  for (int q = 0; q < 3; ++q) a.x[q] = c->s64_vec.p + q * c->n;
  for (int q = 0; q < 2; ++q) a.d[q] = c->s64_vec.p + (3 + q) * c->n;
  a.dm = c->w_out.p;
  a.out = out;
  a.ctl = reinterpret_cast<SeriesCtl *>(c->s64_tab.p);
  // the cached tensors wherever every target is resident, then lanes per
  // target as for single products.  us per step, with its host copies, of <16,
  // 4> / <8, 4> / <32, 4> / <16, 2> / <16, 6> / <16, 0> / <8, 0>: N = 1000, phi =
  // 0.05 117 / 124 / 134 / 117 / 119 / 143 / 179, N = 1500, phi = 0.1 180 / 192
  // / 203 / 196 / 180 / 258 / 270, N = 3600, phi = 0.1 221 / 253 / 577 / 253 /
  // 228 / 329 / 352.  Of <4, 0> / <8, 0> / <16, 0> / <16, 4> at phi = 0.1: N =
  // 4000 417 / 351 / 399 / 513, 17000 935 / 897 / 1021 / 1209, 40000 2007 / 1941
  // / 2212 / 2390, 80000 3516 / 3531 / 4147 / 4467, 200000 7799 / 8067 / 9511 /
  // 11107
  int rc = launch_series_f64<16, 4>(c, a, 1, done);
  if (!rc && !*done) {
    if (c->n >= 80000) rc = launch_series_f64<4, 0>(c, a, 1 << 30, done);
    else rc = launch_series_f64<8, 0>(c, a, 1 << 30, done);
  }
  if (rc || !*done) return rc;
  if ((e = cudaMemcpyAsync(c->h_red, c->s64_tab.p, sizeof(ctl), cudaMemcpyDeviceToHost,
                           c->stream)) ||
      (e = cudaStreamSynchronize(c->stream)))
    return cuda_fail(c, e, "series report");
  std::memcpy(&ctl, c->h_red, sizeof(ctl));
  if (ctl.err) return fail(c, GGEM_ERR_TIMEOUT, "a wait of the FP64 series ran out");
  *rep = ggem_cheb_report{ctl.converged, ctl.n_terms, ctl.n_matvecs, ctl.err1, ctl.err2};
  *first_check = ctl.first_check;
  return GGEM_OK;
}

int fit_tensor64(ggem_ctx *c, double s_max) {
  Tensor64 &t = c->t64;
  const double s0 = std::ldexp(1.0, (int)std::floor(std::log2(0.0168 / c->cst.ksi2)));
  const int sub = 1 << kTab64Sub;
  int np = 1;  // up to the piece that holds s_max
  if (s_max > s0) {
    const int oct = (int)std::floor(std::log2(s_max / s0));
    np += oct * sub + std::min(sub, 1 + (int)((std::ldexp(s_max / s0, -oct) - 1.0) * sub));
  }
  cudaError_t e = c->tab64.ensure((size_t)3 * np);
  if (e) return cuda_fail(c, e, "FP64 tensor");
  FitBasis b;
  for (int j = 0; j < kFitPoints; ++j) {
    const double a = 3.14159265358979323846 * (j + 0.5) / kFitPoints;
    b.node[j] = std::cos(a);
    for (int q = 0; q <= kTab64Deg; ++q) b.w[q][j] = std::cos(q * a) * (q ? 2.0 : 1.0) / kFitPoints;
  }
  // (ggem_create waits for it once, when the rest of the context is set up)
  k_fit_tensor64<<<(np + kFitPieces - 1) / kFitPieces, kFitPoints * kFitPieces, 0, c->stream>>>(
      np, s0, c->dc, b, c->tab64.p);
  if ((e = cudaGetLastError())) return cuda_fail(c, e, "FP64 tensor");
  uint64_t bits;
  std::memcpy(&bits, &s0, sizeof bits);
  t.rec = c->tab64.p;
  t.base = (int)(bits >> (52 - kTab64Sub)) - 1;
  t.last = np - 1;
  t.mid0 = 0.5 * s0;
  return GGEM_OK;
}

// u = M f on slot-ordered FP64 vectors [r][n][3]
int matvec_slots(ggem_ctx *c, int nrhs, const double *f, double *u, int self_mode) {
  if (c->n == 0) return GGEM_OK;
  if (c->prm.precision == GGEM_FP64) {
    if (int rc = ensure_f64_list(c)) return rc;
    int r0 = 0;
    while (r0 < nrhs) {
      const int left = nrhs - r0;
      int rc;
      if (left >= 4) rc = launch_f64<4>(c, f, u, self_mode, r0), r0 += 4;
      else if (left >= 2) rc = launch_f64<2>(c, f, u, self_mode, r0), r0 += 2;
      else rc = launch_f64<1>(c, f, u, self_mode, r0), r0 += 1;
      if (rc) return rc;
    }
    return GGEM_OK;
  }
  if (nrhs == 1) return launch_f32_r1(c, f, u, self_coefficient(c, self_mode));
  if (nrhs >= kBatchMinRhs) return matvec_b64(c, nrhs, f, u, self_coefficient(c, self_mode));
  cudaError_t e = c->w_f32.ensure((size_t)c->n * nrhs);
  if (e) return cuda_fail(c, e, "f32 staging");
  const int64_t tot = c->n * nrhs;
  k_slots_to_f32<<<(unsigned)((tot + 255) / 256), 256, 0, c->stream>>>(c->n, nrhs, f,
                                                                       c->w_f32.p);
  if (int rc = check_launch(c, "to f32")) return rc;
  return matvec_f32_staged(c, nrhs, f, u, self_mode);
}

// xi (caller order) into slot order x0 and, for a batched series, x0's
// staging in w_fb (then matvec_slots_prestaged); false: nothing done
bool to_slots_staged(ggem_ctx *c, int nrhs, const double *xi, double *x0, int *rc) {
  *rc = GGEM_OK;
  if (c->n == 0 || !batch_term_fusable(c, nrhs)) return false;
  const int64_t n = c->n;
  cudaError_t e = c->w_fb.ensure((size_t)n * 3 * kBatchR);
  if (e) {
    *rc = cuda_fail(c, e, "batched staging");
    return true;
  }
  k_to_slots_b64<<<(unsigned)((n + 31) / 32), 256, 0, c->stream>>>(n, nrhs, c->order.p, xi, x0,
                                                                  c->w_fb.p);
  *rc = check_launch(c, "to slots + staging");
  return true;
}

// the batched series' first step with x1's staging left in w_fb (see
// k_cheb_start_b64; 16 .. 64 right-hand sides)
int cheb_start_staged(ggem_ctx *c, int nrhs, double da, double db, double c0, double c1,
                      const double *x0, double *x1, double *dw) {
  const int64_t n = c->n;
  if (n == 0) return GGEM_OK;
  cudaError_t e = c->w_fb.ensure((size_t)n * 3 * kBatchR);
  if (e) return cuda_fail(c, e, "batched staging");
  k_cheb_start_b64<<<(unsigned)((n + 31) / 32), 256, 0, c->stream>>>(n, nrhs, da, db, c0, c1, x0,
                                                                    x1, dw, c->w_fb.p);
  return check_launch(c, "cheb start + staging");
}

// u = M f when the batched staging of f is already in w_fb (the last fused
// batched term wrote it): the batched kernel without the staging pass
int matvec_slots_prestaged(ggem_ctx *c, int nrhs, const double *f, double *u, int self_mode) {
  if (c->n == 0) return GGEM_OK;
  if (!batch_term_fusable(c, nrhs)) return matvec_slots(c, nrhs, f, u, self_mode);
  return matvec_b64(c, nrhs, f, u, self_coefficient(c, self_mode), true);
}

// FP32 pair sum from the already staged c->w_f32 ([r][n] float4); f is the
// FP64 slot-order force of the self term
int matvec_f32_staged(ggem_ctx *c, int nrhs, const double *f, double *u, int self_mode) {
  const double self_c = self_coefficient(c, self_mode);
  int r0 = 0;
  while (r0 < nrhs) {
    const int left = nrhs - r0;
    int rc;
    if (left >= 8) rc = launch_nr<8>(c, f, u, self_c, r0), r0 += 8;
    else if (left >= 4) rc = launch_nr<4>(c, f, u, self_c, r0), r0 += 4;
    else if (left >= 2) rc = launch_nr<2>(c, f, u, self_c, r0), r0 += 2;
    else rc = launch_nr<1>(c, f, u, self_c, r0), r0 += 1;
    if (rc) return rc;
  }
  return GGEM_OK;
}

}  // namespace ggem


using namespace ggem;

extern "C" int ggem_set_symmetric_pairs(ggem_ctx *ctx, int enable) {
  if (!ctx) return GGEM_ERR_BAD_ARG;
  if (ctx->prm.precision != GGEM_FP32 || ctx->prm.nb_mode != GGEM_NB_CUTOFF)
    return ggem::fail(ctx, GGEM_ERR_BAD_ARG, "symmetric pair sums need a GGEM_FP32 cutoff context");
  ctx->sym_pairs = enable != 0;
  ctx->cells_built = false;  // the next ggem_build_cells writes (or drops) the half list
  ctx->list_built = false;
  return GGEM_OK;
}

extern "C" int ggem_set_pair_variant(ggem_ctx *ctx, int computed, int stored) {
  if (!ctx || computed < 0 || computed >= kNumComputedVariants || stored < 0 ||
      stored >= kNumStoredVariants)
    return GGEM_ERR_BAD_ARG;
  ctx->computed_variant = computed;
  ctx->stored_variant = stored;
  return GGEM_OK;
}

extern "C" int ggem_autotune_pair_storage(ggem_ctx *ctx, int reps, double matvecs_per_build,
                                          int *use_stored, double *ms_computed,
                                          double *ms_stored, int *variants) {
  if (!ctx || reps < 1 || !(matvecs_per_build > 0) || !use_stored || !ms_computed ||
      !ms_stored || !variants)
    return GGEM_ERR_BAD_ARG;
  if (int rc = settle_list(ctx)) return rc;
  if (ctx->prm.precision != GGEM_FP32 || !ctx->list_built)
    return fail(ctx, GGEM_ERR_BAD_ARG, "autotune needs a built FP32 pair list");
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != ctx->device) cudaSetDevice(ctx->device);
  const int64_t n = ctx->n;
  cudaError_t e;
  if ((e = ctx->w_in.ensure((size_t)3 * std::max<int64_t>(n, 1))) ||
      (e = ctx->w_out.ensure((size_t)3 * std::max<int64_t>(n, 1))))
    return cuda_fail(ctx, e, "autotune buffers");
  if (n > 0 && (e = cudaMemsetAsync(ctx->w_in.p, 0, sizeof(double) * 3 * n, ctx->stream)))
    return cuda_fail(ctx, e, "autotune buffers");
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const bool timing = ctx->timing;
  ctx->timing = false;
  auto time_matvecs = [&](double *ms, bool first = false) -> int {
    if (int rc = matvec_slots(ctx, 1, ctx->w_in.p, ctx->w_out.p, GGEM_SELF_BEAD)) return rc;
    cudaEventRecord(a, ctx->stream);
    for (int r = 0; r < reps; ++r) {
      if (first) ctx->pretensor_pending = n > 0;
      if (int rc = matvec_slots(ctx, 1, ctx->w_in.p, ctx->w_out.p, GGEM_SELF_BEAD)) return rc;
    }
    cudaEventRecord(b, ctx->stream);
    cudaEventSynchronize(b);
    float t = 0.f;
    cudaEventElapsedTime(&t, a, b);
    *ms = t / reps;
    return GGEM_OK;
  };
  int rc = GGEM_OK;
  double t_comp = 0.0, t_store = 1e30;
  const bool allow = ctx->allow_pretensor;
  // tensors evaluated per pair and matvec, each loop shape; the fastest stays
  ctx->pretensor_ok = false;
  {
    int best_v = 0;
    t_comp = 1e30;
    for (int v = 0; v < kNumComputedVariants && !rc; ++v) {
      ctx->computed_variant = v;
      double t_mv = 0.0;
      rc = time_matvecs(&t_mv);
      if (!rc && t_mv < t_comp) {
        t_comp = t_mv;
        best_v = v;
      }
    }
    ctx->computed_variant = best_v;
  }
  if (!rc && ctx->use_pretensor) {
    ctx->allow_pretensor = true;
    rc = build_pair_tensors(ctx);
    if (!rc && ctx->pretensor_ok) {
      // every stored-tensor kernel shape, its first product over a list (which
      // forms the tensors, in its own kernel or before it) spread over the
      // products per build; the fastest stays selected
      int best_v = 0;
      for (int v = 0; v < kNumStoredVariants && !rc; ++v) {
        ctx->stored_variant = v;
        double t_mv = 0.0, t_first = 0.0;
        rc = time_matvecs(&t_mv);
        if (!rc) rc = time_matvecs(&t_first, true);
        const double t = t_mv + std::max(0.0, t_first - t_mv) / matvecs_per_build;
        if (!rc && t < t_store) {
          t_store = t;
          best_v = v;
        }
      }
      ctx->stored_variant = best_v;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  ctx->timing = timing;
  if (rc) {
    ctx->allow_pretensor = allow;
    if (dev != ctx->device) cudaSetDevice(dev);
    return rc;
  }
  const bool stored = t_store < t_comp;
  ctx->allow_pretensor = stored;
  if (!stored) ctx->pretensor_ok = false;  // the stored tensors stay allocated but unused
  *use_stored = stored ? 1 : 0;
  *ms_computed = t_comp;
  *ms_stored = ctx->use_pretensor ? t_store : -1.0;
  variants[0] = ctx->computed_variant;
  variants[1] = ctx->stored_variant;
  if (dev != ctx->device) cudaSetDevice(dev);
  return GGEM_OK;
}
