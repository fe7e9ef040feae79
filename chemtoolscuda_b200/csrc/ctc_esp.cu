// ctc_esp.cu -- molecular electrostatic potential from Hermite pair densities.
//
// The reference builds all M(M+1)/2 point-charge integrals V_{mu nu}(C) per
// point with the McMurchie-Davidson E and R recursions (Helgaker 9.5.6-7,
// 9.9.18-20; include/integral_coeffs.cuh:17-238, src/evaluate_electrostatic.cu:
// 16-10158) and then contracts them with D in a serial host loop of cublasDtpttr,
// cublasDsymm, a Hadamard product and thrust::reduce per point
// (src/evaluate_electrostatic.cu:10319-10344).  Since
//     sum_{mu nu} D_{mu nu} V_{mu nu}(C)
//        = sum_{pairs ab} (2 pi / p) sum_{tuv} h^{ab}_{tuv} R_{tuv}(p, P - C),
//     h^{ab}_{tuv} = sum_{mu in a, nu in b} D_{mu nu} c_mu c_nu E^x_t E^y_u E^z_v
// depends on the point only through R, the Hermite densities h are built once
// per molecule (host, all cores) and each point costs one Boys evaluation and
// one R recursion per significant primitive pair -- no integral matrix.
// Pairs are grouped by L = l_a + l_b into batches of one class.
//
// Far pairs.  Where every T = p |P - C|^2 of a block of points is beyond the
// class's threshold, R^0_tuv is a derivative of sqrt(pi/p)/2 / |P - C| and the
// pair is a point multipole:
//     sum_tuv h_tuv R_tuv = ri H(x, y, z),  ri = 1/|P - C|, (x, y, z) = (P - C) ri^2,
// H a polynomial of degree L with n_tuv(L) coefficients formed at set-up: one
// reciprocal square root and one multiply-add per coefficient, instead of the R
// recursion and a dot product (FP64 operations per pair and point for L = 0..4:
// 12, 17, 25, 35, 50).  esp_far_kernel sums these pairs, all classes in one
// launch, two points per thread.  Points are sorted along a Morton curve, so a
// block's points lie close together and few pairs are near one of them and far
// from the others.
//
// Near pairs of a block (a few per cent) go to esp_near_kernel: Boys function
// and sum_n G_n p_n(P - C), G_n = (-2p)^n F_n, with polynomials p_n formed at
// set-up (half the operations of the R recursion and its dot product with h).
//
// Boys function F_n(T) (FP64): beyond a per-L threshold (T >= 38 + 3L, where
// the neglected e^{-T} terms are below 2e-17 relative) the asymptotic forms
// hold without an exponential; 99% of (point, pair) evaluations on molecular
// surfaces are of this kind.  Below it, a 7-term Taylor expansion about the nearest point of
// a 0.05-spaced table gives F_L, and F_{n-1} = (2T F_n + e^{-T})/(2n-1)
// (downward recursion, stable) gives the rest.  The table is built at set-up
// from the series F_m(T) = e^{-T} sum_i (2T)^i / ((2m+1)(2m+3)...(2m+2i+1)).
// (The reference uses forward recursion from erf, include/boys_functions.cuh:13-31,
// which loses digits at small T and divides by zero at T = 0.)
//
// V(C) = sum_A Z_A / |C - R_A| - electronic part (src/evaluate_electrostatic.cu:10357-10369).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "ctc_tiles.cuh"

#include "ctc_terms.inc"

namespace ctc {

namespace {

constexpr int kLmax = 8;                 // g x g
constexpr int kTaylor = 7;               // terms of the Taylor expansion
constexpr int kRow = 2;                  // table row of class L: F_{L+6}(T_i), e^{-T_i}
constexpr double kTstep = 0.05;
constexpr double kTmax = 64.0;           // table range: above every far_T(L <= 8)
constexpr int kNT = (int)(kTmax / kTstep) + 2;

__host__ __device__ constexpr int ntuv(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// index of (t,u,v): totals ascending; within a total s, t descending then u descending
__host__ __device__ constexpr int tuv_index(int t, int u, int v) {
  int s = t + u + v;
  int base = s * (s + 1) * (s + 2) / 6;
  int before = 0;
  for (int tt = s; tt > t; --tt) before += s - tt + 1;
  return base + before + (s - t - u);
}

struct EspPair {
  double Px, Py, Pz;
  double c0;    // constant coefficient of the far-field polynomial
  double p;
  double f0c;   // sqrt(pi / p) / 2: F_0 = f0c / |P - C| in the far field
  double rfar;  // far field from this distance on: sqrt(far_T(L) / p)
  double pad;
};
struct EspBatch {
  int32_t b0, b1;   // pairs [b0, b1)
  int64_t h0;       // first near-field coefficient (nnear(L) per pair)
  int64_t f0;       // first far-field coefficient (nfar(L) per pair)
  int32_t L, pad;
};
// Near-field polynomials: sum_tuv h_tuv R_tuv = sum_n G_n p_n(X, Y, Z), p_n of
// the degrees 2n - s for n <= s <= min(2n, L).
__host__ __device__ constexpr int near_lo(int L, int n) { return 2 * n > L ? 2 * n - L : 0; }
__host__ __device__ constexpr int nnear(int L) {
  int c = 0;
  for (int n = 0; n <= L; ++n)
    for (int d = near_lo(L, n); d <= n; ++d) c += (d + 1) * (d + 2) / 2;
  return c;
}
// far-field coefficients of a pair besides the constant one, padded to whole
// 16-byte loads
__host__ __device__ constexpr int nfar(int L) { return ntuv(L) / 2 * 2; }

// FP64 operations of esp_far_pair per pair and point, a multiply-add counted as two:
// P - C and its square 8, the root 8, the last multiply-add 2, and the polynomial.
__host__ __device__ constexpr int far_flops(int L) { return L == 0 ? 18 : (L == 1 ? 26 : 20 + 2 * ntuv(L)); }

double boys_series(int m, double T) {
  double term = 1.0 / (2 * m + 1), sum = term;
  for (int i = 1; i < 1000; ++i) {
    term *= 2.0 * T / (2 * m + 2 * i + 1);
    sum += term;
    if (term < 1e-18 * sum) break;
  }
  return std::exp(-T) * sum;
}

}  // namespace

// pairs per batch of class L: up to 256, with the batch's coefficients within
// 32 KB (a few barriers per batch)
constexpr int kBatchPairs = 256;
constexpr int kBatchH = 4096;
__host__ __device__ constexpr int batch_pairs(int L) {
  return kBatchPairs < kBatchH / ntuv(L) ? kBatchPairs : kBatchH / ntuv(L);
}

struct EspTables {
  double* d_boys = nullptr;
  EspPair* d_pairs = nullptr;
  double* d_h = nullptr;      // near-field polynomials, nnear(L) per pair
  double* d_far = nullptr;    // far-field polynomials, nfar(L) per pair
  EspBatch* d_batches = nullptr;
  double* d_atoms = nullptr;  // x y z Z per atom
  int npairs = 0, nbatch = 0, natom = 0;
  bool s_only = false;        // every kept pair is of class 0
  size_t nh = 0;
  // FP64 work per point with every kept pair in its far form (far_flops): what the
  // call cannot do without, as a near pair costs more
  double flops_per_point = 0.0;
  double mean_L = 0.0;
};

namespace {

// ------------------------------------------------------------------ device side
// First T from which the asymptotic forms F_0 = sqrt(pi/T)/2, F_n =
// (2n-1)/(2T) F_{n-1} agree with F_n(T) to 2e-17 relative for every n <= L
// (the neglected terms are e^{-T} and erfc(sqrt T); thresholds checked against
// the incomplete-gamma form of F_n in 40-digit arithmetic: 37, 41, 44, 47, 50,
// 53, 55, 58, 60 for L = 0..8).
__host__ __device__ constexpr double far_T(int L) { return 38.0 + 3.0 * L; }

// G_n = R^n_000 = (-2p)^n F_n(T), n = 0..L, at T = p r2.
//  far field (T >= far_T(L)): the p dependence cancels except in F_0,
//    G_0 = (sqrt(pi/p)/2) / r,  G_n = -(2n-1) G_{n-1} / r2  -- no exponential;
//  otherwise: from one 16-byte table row at the nearest 0.05 step T_i,
//    F_{L+6}(T_i) and e^{-T_i}: F_{L+5} .. F_L there by downward recursion, F_L(T)
//    by the 7-term Taylor expansion in d = T_i - T, e^{-T} = e^{-T_i} e^d with e^d
//    by its series to d^7 (|d| <= 0.025: remainder below 4e-18), and
//    F_{n-1} = (2T F_n + e^{-T}) / (2n-1) downwards (stable for every T).  The
//    lanes' rows lie far apart, so the row's size is what the L1 sees: reading
//    the seven coefficients (64 bytes in four loads) bound the near kernel.
template <int L>
__device__ __forceinline__ void boys_g(double p, double f0c, double r2, const double* __restrict__ tab,
                                       double* G) {
  const double T = p * r2;
  if (!(T < far_T(L))) {  // NaN too: its conversion to a table row is out of range
    const double ri = rsqrt(r2);
    const double ri2 = ri * ri;
    G[0] = f0c * ri;
#pragma unroll
    for (int n = 1; n <= L; ++n) G[n] = -(double)(2 * n - 1) * ri2 * G[n - 1];
  } else {
    const int i = __double2int_rn(T * (1.0 / kTstep));
    const double d = i * kTstep - T;  // T_i - T
    const double2 row = __ldg(reinterpret_cast<const double2*>(tab) + ((int64_t)L * kNT + i));
    double F[L + 1], f[kTaylor];
    const double Ti2 = 2.0 * (i * kTstep);
    f[kTaylor - 1] = row.x;
#pragma unroll
    for (int k = kTaylor - 1; k > 0; --k)
      f[k - 1] = fma(Ti2, f[k], row.y) * (1.0 / (double)(2 * (L + k) - 1));
    double fl = f[kTaylor - 1];
#pragma unroll
    for (int k = kTaylor - 2; k >= 0; --k) fl = fma(fl * d, 1.0 / (double)(k + 1), f[k]);
    F[L] = fl;
    if (L > 0) {
      double q = 1.0 / 5040.0;
      q = fma(q, d, 1.0 / 720.0);
      q = fma(q, d, 1.0 / 120.0);
      q = fma(q, d, 1.0 / 24.0);
      q = fma(q, d, 1.0 / 6.0);
      q = fma(q, d, 0.5);
      q = fma(q, d, 1.0);
      q = fma(q, d, 1.0);
      const double e = row.y * q, T2 = 2.0 * T;
#pragma unroll
      for (int n = L; n > 0; --n) F[n - 1] = fma(T2, F[n], e) * (1.0 / (double)(2 * n - 1));
    }
    double m = 1.0;
#pragma unroll
    for (int n = 0; n <= L; ++n) {
      G[n] = m * F[n];
      m *= -2.0 * p;
    }
  }
}

// sum_n G_n p_n(X, Y, Z) of one pair, the p_n in nested Horner form with the
// coefficients in the order of their use (n ascending; powers of X, then Y, then
// Z, descending).  Operations for L = 0..4: 1, 5, 15, 34, 66, about half of the
// R recursion and its dot product with h.
template <int L>
__device__ __forceinline__ double near_sum(double X, double Y, double Z, const double* G,
                                           const double* __restrict__ h) {
  double zp[L + 1];
  zp[0] = 1.0;
#pragma unroll
  for (int i = 1; i <= L; ++i) zp[i] = zp[i - 1] * Z;
  double s = 0.0;
  int k = 0;
#pragma unroll
  for (int n = 0; n <= L; ++n) {
    const int dlo = near_lo(L, n);
    double f = 0.0;
#pragma unroll
    for (int a = n; a >= 0; --a) {
      double g = 0.0;
#pragma unroll
      for (int b = n - a; b >= 0; --b) {
        const int lo = dlo > a + b ? dlo - a - b : 0;
        double t = h[k++];
#pragma unroll
        for (int e = n - a - b - 1; e >= lo; --e) t = fma(t, Z, h[k++]);
        if (lo > 0) t *= zp[lo];
        g = b == n - a ? t : fma(g, Y, t);
      }
      f = a == n ? g : fma(f, X, g);
    }
    s = fma(G[n], f, s);
  }
  return s;
}

constexpr int kEspThreads = 128;

// Points in their sorted order: xyz[3][n].
__global__ void __launch_bounds__(256)
    esp_gather_kernel(const double* __restrict__ pts, const int32_t* __restrict__ perm, int64_t n,
                      double* __restrict__ xyz) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t p = perm ? perm[i] : i;
  for (int d = 0; d < 3; ++d) xyz[d * n + i] = pts[3 * p + d];
}

// A point as the pair sums see it: finite coordinates are cut at 1e153 bohr, so
// that |P - C|^2 stays finite (esp_finish_kernel gives zero beyond).
constexpr double kEspMost = 1e153;
__device__ __forceinline__ double esp_coord(double v) {
  return isfinite(v) ? fmin(fmax(v, -kEspMost), kEspMost) : v;
}

// Sphere around the finite points of a block of kEspThreads threads with P
// points each (centre of their box); radius -1e300 when no point is finite.
template <int P>
__device__ void esp_sphere(const double (*c)[3], const bool* live, double* ctr, double* rad) {
  __shared__ double s_lo[3][kEspThreads / 32], s_hi[3][kEspThreads / 32], s_r[kEspThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = 0; d < 3; ++d) {
    double lo = 1e300, hi = -1e300;
    for (int p = 0; p < P; ++p)
      if (live[p] && finite_point(c[p])) {
        lo = fmin(lo, c[p][d]);
        hi = fmax(hi, c[p][d]);
      }
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
      s_lo[d][warp] = lo;
      s_hi[d][warp] = hi;
    }
  }
  __syncthreads();
  bool any = false;
  for (int d = 0; d < 3; ++d) {
    double lo = 1e300, hi = -1e300;
    for (int w = 0; w < kEspThreads / 32; ++w) {
      lo = fmin(lo, s_lo[d][w]);
      hi = fmax(hi, s_hi[d][w]);
    }
    any = lo <= hi;
    ctr[d] = any ? 0.5 * lo + 0.5 * hi : 0.0;
  }
  double r2 = 0.0;
  for (int p = 0; p < P; ++p)
    if (live[p] && finite_point(c[p])) {
      const double x = c[p][0] - ctr[0], y = c[p][1] - ctr[1], z = c[p][2] - ctr[2];
      r2 = fmax(r2, x * x + y * y + z * z);
    }
  for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if (lane == 0) s_r[warp] = r2;
  __syncthreads();
  for (int w = 0; w < kEspThreads / 32; ++w) r2 = fmax(r2, s_r[w]);
  *rad = any ? sqrt(r2) * (1.0 + 1e-12) + 1e-9 : -1e300;
}

// Indices of the batch's far (or near) pairs in order; returns their number.
// The block's sphere decides, the same way in both kernels.
template <bool FAR>
__device__ int esp_select(const EspPair* __restrict__ pairs, int np, const double* ctr, double rad,
                          uint16_t* s_list, int* s_cnt) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nch = (np + 31) / 32;
  unsigned mask[kBatchPairs / kEspThreads];
#pragma unroll
  for (int k = 0; k < kBatchPairs / kEspThreads; ++k) {
    const int ch = warp + k * (kEspThreads / 32), i = ch * 32 + lane;
    bool take = false;
    if (i < np) {
      const EspPair& q = pairs[i];
      const double x = q.Px - ctr[0], y = q.Py - ctr[1], z = q.Pz - ctr[2];
      const double need = q.rfar + rad;
      const bool far = need <= 0.0 || x * x + y * y + z * z >= need * need * (1.0 + 1e-12);
      take = far == FAR;
    }
    mask[k] = __ballot_sync(0xffffffffu, take);
    if (lane == 0 && ch < kBatchPairs / 32) s_cnt[ch] = ch < nch ? __popc(mask[k]) : 0;
  }
  __syncthreads();
  int total = 0;
#pragma unroll
  for (int ch = 0; ch < kBatchPairs / 32; ++ch) total += s_cnt[ch];
#pragma unroll
  for (int k = 0; k < kBatchPairs / kEspThreads; ++k) {
    const int ch = warp + k * (kEspThreads / 32);
    int base = 0;
    for (int j = 0; j < ch; ++j) base += s_cnt[j];
    if ((mask[k] >> lane) & 1u) s_list[base + __popc(mask[k] & ((1u << lane) - 1u))] = (uint16_t)(ch * 32 + lane);
  }
  return total;
}

// 1 / sqrt(x): the hardware's approximation (relative error below 2^-19 over
// the normal range) and one step of Householder's third-order iteration, whose
// remainder is (5/16) e^3 < 2^-55 (measured: 1.4e-16; rsqrt(): 1.1e-16).  With
// rsqrt() 1e5 surface points of 100 atoms take 149.3 ms instead of 136.7, 1 500
// points of 12 atoms 270 us instead of 260, and the potential's error against 64
// bits is the same (1.3e-15 of its scale).
__device__ __forceinline__ double esp_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// acc[p] += ri H(x, y, z) of one far pair: nested Horner form, coefficients in
// the order of their use (powers of x, then y, then z, descending; the constant
// one is c0).
template <int L, int P>
__device__ __forceinline__ void esp_far_pair(const double4 q, const double2* __restrict__ h,
                                             const double (*c)[3], double* acc) {
  double x[P], y[P], z[P], ri[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    x[p] = q.x - c[p][0];
    y[p] = q.y - c[p][1];
    z[p] = q.z - c[p][2];
    ri[p] = esp_rsqrt(x[p] * x[p] + y[p] * y[p] + z[p] * z[p]);
    if (L == 1) {  // c0 + u (c . X): two operations fewer than scaling X
      const double2 xy = h[0], zo = h[1];
      const double s = fma(zo.x, z[p], fma(xy.y, y[p], xy.x * x[p]));
      acc[p] = fma(ri[p], fma(ri[p] * ri[p], s, q.w), acc[p]);
    } else if (L > 0) {
      const double u = ri[p] * ri[p];
      x[p] *= u;
      y[p] *= u;
      z[p] *= u;
    }
  }
  if (L == 1) return;
  double f[P], g[P], t[P];
  int k = 0;
#pragma unroll
  for (int a = L; a >= 0; --a) {
#pragma unroll
    for (int b = L - a; b >= 0; --b) {
#pragma unroll
      for (int e = L - a - b; e >= 0; --e) {
        const bool last = a == 0 && b == 0 && e == 0;
        const double co = last ? q.w : ((k & 1) ? h[k >> 1].y : h[k >> 1].x);
        ++k;
#pragma unroll
        for (int p = 0; p < P; ++p) t[p] = e == L - a - b ? co : fma(t[p], z[p], co);
      }
#pragma unroll
      for (int p = 0; p < P; ++p) g[p] = b == L - a ? t[p] : fma(g[p], y[p], t[p]);
    }
#pragma unroll
    for (int p = 0; p < P; ++p) f[p] = a == L ? g[p] : fma(f[p], x[p], g[p]);
  }
#pragma unroll
  for (int p = 0; p < P; ++p) acc[p] = fma(ri[p], f[p], acc[p]);
}

// Far pairs of block x's points (P per thread) in slice y of the batches of all
// classes: row y of part.  Rows are summed in a fixed order by
// esp_finish_kernel, so results do not depend on timing.
// Bound: FP64 pipe (73% busy).  100 atoms (1 604 functions, 8e5 pairs), 1e5
// surface points: far 110 ms and near 26 ms; one kernel per class with the R
// recursion for every pair took 287 ms.
template <int P>
__global__ void __launch_bounds__(kEspThreads)
    esp_far_kernel(const EspPair* __restrict__ pairs, const double* __restrict__ far,
                   const EspBatch* __restrict__ batches, int nb, const double* __restrict__ xyz, int64_t n,
                   double* __restrict__ part) {
  __shared__ double4 sp[kBatchPairs];
  __shared__ __align__(16) double sh[kBatchH];
  __shared__ uint16_t s_list[kBatchPairs];
  __shared__ int s_cnt[kBatchPairs / 32];
  const int slices = gridDim.y, y = blockIdx.y;
  const int bb = (int)((int64_t)nb * y / slices), be = (int)((int64_t)nb * (y + 1) / slices);
  double c[P][3], acc[P];
  bool live[P];
  int64_t ip[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    ip[p] = ((int64_t)blockIdx.x * P + p) * kEspThreads + threadIdx.x;
    live[p] = ip[p] < n;
    for (int d = 0; d < 3; ++d) c[p][d] = esp_coord(xyz[d * n + (live[p] ? ip[p] : n - 1)]);
    acc[p] = 0.0;
  }
  double ctr[3], rad;
  esp_sphere<P>(c, live, ctr, &rad);
  for (int b = bb; b < be; ++b) {
    const EspBatch bt = batches[b];
    const int np = bt.b1 - bt.b0;
    __syncthreads();  // readers of the previous batch are done
    for (int i = threadIdx.x; i < np; i += kEspThreads) {
      const EspPair& q = pairs[bt.b0 + i];
      sp[i] = make_double4(q.Px, q.Py, q.Pz, q.c0);
    }
    const int nd = np * nfar(bt.L) / 2;
    const double2* src = reinterpret_cast<const double2*>(far + bt.f0);
    for (int i = threadIdx.x; i < nd; i += kEspThreads) reinterpret_cast<double2*>(sh)[i] = src[i];
    const int nf = esp_select<true>(pairs + bt.b0, np, ctr, rad, s_list, s_cnt);
    __syncthreads();
#define CTC_ESP_FAR(LL)                                                                                \
  case LL:                                                                                             \
    for (int k = 0; k < nf; ++k) {                                                                     \
      const int i = s_list[k];                                                                         \
      esp_far_pair<LL, P>(sp[i], reinterpret_cast<const double2*>(sh) + i * (nfar(LL) / 2), c, acc);   \
    }                                                                                                  \
    break;
    switch (bt.L) {
      CTC_ESP_FAR(0)
      CTC_ESP_FAR(1)
      CTC_ESP_FAR(2)
      CTC_ESP_FAR(3)
      CTC_ESP_FAR(4)
      CTC_ESP_FAR(5)
      CTC_ESP_FAR(6)
      CTC_ESP_FAR(7)
      CTC_ESP_FAR(8)
    }
#undef CTC_ESP_FAR
  }
#pragma unroll
  for (int p = 0; p < P; ++p)
    if (live[p]) part[(int64_t)y * n + ip[p]] = acc[p];
}

// Near pairs of the same blocks and slices.  A warp whose points are all far
// from the pair takes the far-field polynomial, the others the Boys function
// and the near-field polynomials (far points of such a warp by the asymptotic
// form).
template <int P>
__global__ void __launch_bounds__(kEspThreads, 7)
    esp_near_kernel(const EspPair* __restrict__ pairs, const double* __restrict__ hbuf,
                    const double* __restrict__ far, const EspBatch* __restrict__ batches, int nb, const double* __restrict__ tab,
                    const double* __restrict__ xyz, int64_t n, double* __restrict__ part) {
  __shared__ EspPair sp[kBatchPairs / 4];
  __shared__ double sh[kBatchH / 4];
  __shared__ __align__(16) double sf[kBatchH / 4];
  __shared__ uint16_t s_list[kBatchPairs];
  __shared__ int s_cnt[kBatchPairs / 32];
  const int slices = gridDim.y, y = blockIdx.y;
  const int bb = (int)((int64_t)nb * y / slices), be = (int)((int64_t)nb * (y + 1) / slices);
  double c[P][3], acc[P];
  bool live[P];
  int64_t ip[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    ip[p] = ((int64_t)blockIdx.x * P + p) * kEspThreads + threadIdx.x;
    live[p] = ip[p] < n;
    for (int d = 0; d < 3; ++d) c[p][d] = esp_coord(xyz[d * n + (live[p] ? ip[p] : n - 1)]);
    acc[p] = 0.0;
  }
  double ctr[3], rad;
  esp_sphere<P>(c, live, ctr, &rad);
  for (int b = bb; b < be; ++b) {
    const EspBatch bt = batches[b];
    __syncthreads();
    const int nn = esp_select<false>(pairs + bt.b0, bt.b1 - bt.b0, ctr, rad, s_list, s_cnt);
    // the near pairs in groups that fit the shared arrays
    const int NT = nnear(bt.L), cap = min(kBatchPairs, kBatchH / NT) / 4;  // (coefficients: 1024)
    for (int g0 = 0; g0 < nn; g0 += cap) {
      const int ng = min(cap, nn - g0);
      __syncthreads();
      for (int i = threadIdx.x; i < ng; i += kEspThreads) sp[i] = pairs[bt.b0 + s_list[g0 + i]];
      for (int i = threadIdx.x; i < ng * NT; i += kEspThreads)
        sh[i] = hbuf[bt.h0 + s_list[g0 + i / NT] * NT + i % NT];
      const int NF = nfar(bt.L);
      for (int i = threadIdx.x; i < ng * NF; i += kEspThreads)
        sf[i] = far[bt.f0 + s_list[g0 + i / NF] * NF + i % NF];
      __syncthreads();
      auto run = [&](auto lc) {
        constexpr int L = decltype(lc)::value;
        for (int k = 0; k < ng; ++k) {
          const EspPair q = sp[k];
#pragma unroll
          for (int p = 0; p < P; ++p) {
            const double X = q.Px - c[p][0], Y = q.Py - c[p][1], Z = q.Pz - c[p][2];
            const double r2 = X * X + Y * Y + Z * Z;
            // (beyond 1e30 bohr the powers of X overflow: far form also in a mixed warp)
            if (__all_sync(0xffffffffu, q.p * r2 >= far_T(L)) || r2 > 1e60) {
              esp_far_pair<L, 1>(make_double4(q.Px, q.Py, q.Pz, q.c0),
                                 reinterpret_cast<const double2*>(sf) + k * (nfar(L) / 2), c + p, acc + p);
              continue;
            }
            double G[L + 1];
            boys_g<L>(q.p, q.f0c, r2, tab, G);
            acc[p] += near_sum<L>(X, Y, Z, G, sh + k * nnear(L));
          }
        }
      };
      switch (bt.L) {
        case 0: run(std::integral_constant<int, 0>{}); break;
        case 1: run(std::integral_constant<int, 1>{}); break;
        case 2: run(std::integral_constant<int, 2>{}); break;
        case 3: run(std::integral_constant<int, 3>{}); break;
        case 4: run(std::integral_constant<int, 4>{}); break;
        case 5: run(std::integral_constant<int, 5>{}); break;
        case 6: run(std::integral_constant<int, 6>{}); break;
        case 7: run(std::integral_constant<int, 7>{}); break;
        default: run(std::integral_constant<int, 8>{}); break;
      }
    }
  }
#pragma unroll
  for (int p = 0; p < P; ++p)
    if (live[p]) part[(int64_t)y * n + ip[p]] = acc[p];
}

// V = sum_A Z_A / |C - R_A| - (sum of the rows of part, in row order).  Beyond
// kEspMost the electronic part is zero; at infinity only with s functions alone
// (the higher multipoles are infinity times zero there: NaN).
__global__ void __launch_bounds__(256)
    esp_finish_kernel(const double* __restrict__ part, int rows, const double* __restrict__ atoms, int natom,
                      const double* __restrict__ xyz, const int32_t* __restrict__ perm, int64_t n, bool s_only,
                      double* __restrict__ out) {
  const int64_t ip = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= n) return;
  const double cx = xyz[ip], cy = xyz[n + ip], cz = xyz[2 * n + ip];
  double elec = 0.0;
  for (int r = 0; r < rows; ++r) elec += part[(int64_t)r * n + ip];
  const double most = fmax(fmax(fabs(cx), fabs(cy)), fabs(cz));  // (fmax drops a NaN)
  if (most > kEspMost && (s_only || most < INFINITY) && !isnan(cx) && !isnan(cy) && !isnan(cz)) elec = 0.0;
  double nuc = 0.0;
  for (int a = 0; a < natom; ++a) {
    const double dx = cx - atoms[4 * a], dy = cy - atoms[4 * a + 1], dz = cz - atoms[4 * a + 2];
    nuc += atoms[4 * a + 3] / sqrt(dx * dx + dy * dy + dz * dz);
  }
  out[perm ? perm[ip] : ip] = nuc - elec;
}

// ------------------------------------------------------------------ host side
void hermite_e(int la, int lb, double a, double b, double XAB, std::vector<double>& E) {
  const int L = la + lb;
  const double p = a + b, mu = a * b / p;
  const double XPA = -(b / p) * XAB, XPB = (a / p) * XAB;
  E.assign((size_t)(la + 1) * (lb + 1) * (L + 1), 0.0);
  auto at = [&](int i, int j, int t) -> double& { return E[((size_t)i * (lb + 1) + j) * (L + 1) + t]; };
  at(0, 0, 0) = std::exp(-mu * XAB * XAB);
  for (int i = 0; i <= la; ++i)
    for (int j = 0; j <= lb; ++j) {
      if (i == 0 && j == 0) continue;
      for (int t = 0; t <= i + j; ++t) {
        if (j == 0) {
          double em = t >= 1 ? at(i - 1, 0, t - 1) : 0.0;
          double e0 = t <= i - 1 ? at(i - 1, 0, t) : 0.0;
          double ep = t + 1 <= i - 1 ? at(i - 1, 0, t + 1) : 0.0;
          at(i, j, t) = em / (2 * p) + XPA * e0 + (t + 1) * ep;
        } else {
          double em = t >= 1 ? at(i, j - 1, t - 1) : 0.0;
          double e0 = t <= i + j - 1 ? at(i, j - 1, t) : 0.0;
          double ep = t + 1 <= i + j - 1 ? at(i, j - 1, t + 1) : 0.0;
          at(i, j, t) = em / (2 * p) + XPB * e0 + (t + 1) * ep;
        }
      }
    }
}

struct Mono { int a, b, c; };

// Cartesian monomials of degree l and the component -> monomial coefficient matrix.
void seg_monomials(int type, std::vector<Mono>& monos, std::vector<double>& Tm /*ncomp x nmono*/) {
  const int l = l_of_type(type), nc = ncomp_of_type(type);
  monos.clear();
  for (int a = l; a >= 0; --a)
    for (int b = l - a; b >= 0; --b) monos.push_back({a, b, l - a - b});
  Tm.assign((size_t)nc * monos.size(), 0.0);
  for (int j = 0; j < nc; ++j)
    for (int t = h_comp_off[type][j]; t < h_comp_off[type][j + 1]; ++t) {
      const Term& T = h_terms[t];
      for (size_t m = 0; m < monos.size(); ++m)
        if (monos[m].a == T.a && monos[m].b == T.b && monos[m].c == T.z) Tm[j * monos.size() + m] += T.c;
    }
}

struct PairOut {
  int L;
  double bound;  // upper bound of |pair contribution| at any point
  EspPair pr;
  std::vector<double> h;
};

// Coefficients of a pair's polynomials as linear maps of its Hermite
// coefficients h, one sparse list of (output, input, factor) per class.
struct MapTerm {
  int16_t out, in;
  double f;
};
struct EspMaps {
  std::vector<MapTerm> near[kLmax + 1];  // outputs in near_sum's order
  std::vector<MapTerm> far[kLmax + 1];   // outputs in esp_far_pair's order, the constant one last
  EspMaps() {
    // Near field: R_tuv = sum_ijk a_ti a_uj a_vk X^(t-2i) Y^(u-2j) Z^(v-2k) G_(t+u+v-i-j-k),
    // a_ti = t! / (2^i i! (t - 2i)!), the solved recursion R^n_{t+1} = X R^(n+1)_t + t R^(n+1)_{t-1}.
    auto fac = [](int t, int i) {
      double v = 1.0;
      for (int k = 0; k < 2 * i; ++k) v *= t - k;
      for (int k = 1; k <= i; ++k) v /= 2.0 * k;
      return v;
    };
    for (int L = 0; L <= kLmax; ++L) {
      int k = 0;
      for (int n = 0; n <= L; ++n)
        for (int a = n; a >= 0; --a)
          for (int b = n - a; b >= 0; --b)
            for (int c = n - a - b; c >= std::max(0, near_lo(L, n) - a - b); --c, ++k) {
              const int m = n - (a + b + c);  // i + j + k
              for (int i = 0; i <= m; ++i)
                for (int j = 0; i + j <= m; ++j) {
                  const int t = a + 2 * i, u = b + 2 * j, v = c + 2 * (m - i - j);
                  near[L].push_back({(int16_t)k, (int16_t)tuv_index(t, u, v), fac(t, i) * fac(u, j) * fac(v, m - i - j)});
                }
            }
    }
    // Far field: d_x^t d_y^u d_z^v (1/r) = Q_tuv r^(-2l-1), l = t + u + v, with
    // Q_000 = 1 and Q_{t+1,u,v} = r^2 d_x Q - (2l+1) x Q (the same for y, z):
    // homogeneous of degree l with integer coefficients.  With (x, y, z) scaled
    // by 1/r^2, sum_tuv h_tuv Q_tuv r^(-2l-1) is 1/r times one polynomial.
    // q[tuv]: coefficients by tuv_index of the monomial, from its degree's first
    std::vector<std::vector<double>> q(ntuv(kLmax));
    q[0] = {1.0};
    for (int s = 1; s <= kLmax; ++s)
      for (int t = s; t >= 0; --t)
        for (int u = s - t; u >= 0; --u) {
          int low[3] = {t, u, s - t - u};
          const int ax = low[0] ? 0 : (low[1] ? 1 : 2);
          --low[ax];
          const int l = s - 1, base_l = ntuv(l - 1), base_s = ntuv(s - 1);
          const std::vector<double>& ql = q[tuv_index(low[0], low[1], low[2])];
          std::vector<double> r(ntuv(s) - base_s, 0.0);
          for (int a = 0; a <= l; ++a)
            for (int b = 0; a + b <= l; ++b) {
              const int m[3] = {a, b, l - a - b};
              const double c = ql[tuv_index(m[0], m[1], m[2]) - base_l];
              if (c == 0.0) continue;
              auto add = [&](int d0, int d1, int d2, double v) {
                r[tuv_index(m[0] + d0, m[1] + d1, m[2] + d2) - base_s] += v;
              };
              add(ax == 0, ax == 1, ax == 2, -(2.0 * l + 1.0) * c);
              if (m[ax] > 0)
                for (int k = 0; k < 3; ++k)
                  add(2 * (k == 0) - (ax == 0), 2 * (k == 1) - (ax == 1), 2 * (k == 2) - (ax == 2), m[ax] * c);
            }
          q[tuv_index(t, u, s - t - u)] = std::move(r);
        }
    for (int L = 0; L <= kLmax; ++L) {
      int k = 0;
      for (int a = L; a >= 0; --a)
        for (int b = L - a; b >= 0; --b)
          for (int c = L - a - b; c >= 0; --c, ++k) {
            const int s = a + b + c, base = ntuv(s - 1), mono = tuv_index(a, b, c) - base;
            for (int i = base; i < ntuv(s); ++i)
              if (q[i][mono] != 0.0) far[L].push_back({(int16_t)k, (int16_t)i, q[i][mono]});
          }
    }
  }
};

// Upper bound of |R^0_tuv(p, X)| over all points for t + u + v = s, used to
// bound a pair's contribution: (2p)^(s/2) times a generous constant in s.
inline double r_bound(double p, int s) { return std::pow(2.0 * p + 1.0, 0.5 * s) * std::pow(3.0, s); }

// The Boys table of every class (it depends on nothing else: formed once).
const std::vector<double>& boys_table() {
  static const std::vector<double> table = [] {
    std::vector<double> tab((size_t)(kLmax + 1) * kNT * kRow);
    for (int i = 0; i < kNT; ++i) {
      const double e = std::exp(-i * kTstep);
      for (int L = 0; L <= kLmax; ++L) {
        double* row = &tab[((size_t)L * kNT + i) * kRow];
        row[0] = boys_series(L + kTaylor - 1, i * kTstep);
        row[1] = e;
      }
    }
    return tab;
  }();
  return table;
}

}  // namespace

void destroy_esp(ctc_molecule* mol) {
  if (!mol->esp) return;
  cudaFree(mol->esp->d_boys);
  cudaFree(mol->esp->d_pairs);
  cudaFree(mol->esp->d_h);
  cudaFree(mol->esp->d_far);
  cudaFree(mol->esp->d_batches);
  cudaFree(mol->esp->d_atoms);
  delete mol->esp;
  mol->esp = nullptr;
  mol->esp_valid = false;
}

static int build_esp(ctc_molecule* mol) {
  destroy_esp(mol);
  if (int rc = refresh_host_density(mol); rc != CTC_OK) return rc;
  for (const DevSeg& s : mol->segs)
    if (s.l > 4) return fail(CTC_ERR_UNSUPPORTED, "ESP: angular momentum above g");
  const int nseg = mol->nseg, M = mol->M;
  // per-segment monomial data
  std::vector<std::vector<Mono>> monos(nseg);
  std::vector<std::vector<double>> Tm(nseg);
  for (int s = 0; s < nseg; ++s) seg_monomials(mol->segs[s].type, monos[s], Tm[s]);
  const double eps = 1e-22;            // pre-filter before the Hermite densities are formed
  const double budget = 1e-11;         // total |ESP| error allowed for the pairs dropped below
  unsigned nthr = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
  std::vector<std::vector<PairOut>> outs(nthr);
  auto worker = [&](unsigned tid) {
    std::vector<double> Ex, Ey, Ez, Dc;
    for (int I = (int)tid; I < nseg; I += (int)nthr) {
      const DevSeg& A = mol->segs[I];
      const int nA = ncomp_of_type(A.type), mA = (int)monos[I].size();
      for (int J = I; J < nseg; ++J) {
        const DevSeg& B = mol->segs[J];
        const int nB = ncomp_of_type(B.type), mB = (int)monos[J].size();
        const double fac = (I == J) ? 1.0 : 2.0;
        // Cartesian-monomial density Dc = Tm_A^T D_AB Tm_B
        Dc.assign((size_t)mA * mB, 0.0);
        double dmax = 0.0;
        for (int i = 0; i < nA; ++i)
          for (int j = 0; j < nB; ++j) {
            const double d = mol->D[(size_t)(A.ao0 + i) * M + (B.ao0 + j)];
            if (d == 0.0) continue;
            for (int ma = 0; ma < mA; ++ma) {
              const double ta = Tm[I][(size_t)i * mA + ma];
              if (ta == 0.0) continue;
              for (int mb = 0; mb < mB; ++mb) Dc[(size_t)ma * mB + mb] += d * ta * Tm[J][(size_t)j * mB + mb];
            }
          }
        for (double v : Dc) dmax = std::max(dmax, std::fabs(v));
        if (dmax == 0.0) continue;
        const int L = A.l + B.l, NT = ntuv(L);
        const double XAB = A.cx - B.cx, YAB = A.cy - B.cy, ZAB = A.cz - B.cz;
        const double R2 = XAB * XAB + YAB * YAB + ZAB * ZAB;
        for (int ka = 0; ka < A.nprim; ++ka) {
          const double a = mol->alpha[A.prim0 + ka], ca = mol->coef[A.prim0 + ka];
          for (int kb = 0; kb < B.nprim; ++kb) {
            const double b = mol->alpha[B.prim0 + kb], cb = mol->coef[B.prim0 + kb];
            const double p = a + b, mu = a * b / p;
            const double K = std::exp(-mu * R2);
            const double pref = 2.0 * kPi / p;
            const double scale = fac * ca * cb;
            // bound on |h| * |R| (|R_tuv| <= (2p)^(s/2) * s!! F-like factors)
            const double bound = std::fabs(scale) * K * dmax * pref * mA * mB *
                                 std::pow(1.0 + 2.0 * p, 0.5 * L) * std::pow(2.0, L);
            if (bound < eps) continue;
            hermite_e(A.l, B.l, a, b, XAB, Ex);
            hermite_e(A.l, B.l, a, b, YAB, Ey);
            hermite_e(A.l, B.l, a, b, ZAB, Ez);
            PairOut po;
            po.L = L;
            po.pr = {(a * A.cx + b * B.cx) / p, (a * A.cy + b * B.cy) / p, (a * A.cz + b * B.cz) / p, 0.0, p,
                     0.5 * std::sqrt(kPi / p), std::sqrt(far_T(L) / p), 0.0};
            po.h.assign(NT, 0.0);
            const int LB1 = B.l + 1, L1 = L + 1;
            for (int ma = 0; ma < mA; ++ma) {
              const Mono& u = monos[I][ma];
              for (int mb = 0; mb < mB; ++mb) {
                const double dc = Dc[(size_t)ma * mB + mb] * scale;
                if (dc == 0.0) continue;
                const Mono& w = monos[J][mb];
                for (int t = 0; t <= u.a + w.a; ++t) {
                  const double ex = Ex[((size_t)u.a * LB1 + w.a) * L1 + t] * dc;
                  for (int uu = 0; uu <= u.b + w.b; ++uu) {
                    const double exy = ex * Ey[((size_t)u.b * LB1 + w.b) * L1 + uu];
                    for (int v = 0; v <= u.c + w.c; ++v)
                      po.h[tuv_index(t, uu, v)] += exy * Ez[((size_t)u.c * LB1 + w.c) * L1 + v];
                  }
                }
              }
            }
            double bnd = 0.0;
            for (int tt = 0; tt <= L; ++tt)
              for (int uu = 0; uu <= L - tt; ++uu)
                for (int vv = 0; vv <= L - tt - uu; ++vv)
                  bnd += std::fabs(po.h[tuv_index(tt, uu, vv)]) * r_bound(p, tt + uu + vv);
            po.bound = bnd * pref;
            if (po.bound < eps) continue;
            for (double& v : po.h) v *= pref;  // the kernels sum h_tuv R_tuv with 2 pi / p folded in
            outs[tid].push_back(std::move(po));
          }
        }
      }
    }
  };
  std::vector<std::thread> th;
  for (unsigned t = 0; t < nthr; ++t) th.emplace_back(worker, t);
  for (auto& t : th) t.join();
  // drop the weakest pairs while their summed bound stays within the budget:
  // pairs are ranked by (bound, thread, position) and exactly the accumulated
  // prefix is dropped, so ties at the cut never drop more than the budget
  {
    struct Ranked { double bound; uint32_t list, pos; };
    std::vector<Ranked> rk;
    for (uint32_t l = 0; l < outs.size(); ++l)
      for (uint32_t i = 0; i < outs[l].size(); ++i) rk.push_back({outs[l][i].bound, l, i});
    std::sort(rk.begin(), rk.end(), [](const Ranked& a, const Ranked& b) {
      return a.bound != b.bound ? a.bound < b.bound : (a.list != b.list ? a.list < b.list : a.pos < b.pos);
    });
    std::vector<std::vector<char>> drop(outs.size());
    for (size_t l = 0; l < outs.size(); ++l) drop[l].assign(outs[l].size(), 0);
    double acc = 0.0;
    for (const Ranked& r : rk) {
      if (acc + r.bound > budget) break;
      acc += r.bound;
      drop[r.list][r.pos] = 1;
    }
    for (size_t l = 0; l < outs.size(); ++l) {
      size_t w = 0;
      for (size_t i = 0; i < outs[l].size(); ++i) {
        if (drop[l][i]) continue;
        if (w != i) outs[l][w] = std::move(outs[l][i]);  // a self-move would empty h
        ++w;
      }
      outs[l].resize(w);
    }
  }
  // gather, sorted by L, into batches of equal L
  std::vector<EspPair> pairs;
  std::vector<double> hh;  // Hermite coefficients, ntuv(L) per pair
  std::vector<EspBatch> batches;
  size_t nnear_all = 0, nfar_all = 0;
  std::vector<size_t> batch_hh;
  for (int L = 0; L <= kLmax; ++L) {
    const int per = batch_pairs(L);
    int in_batch = 0;
    for (auto& o : outs)
      for (auto& po : o) {
        if (po.L != L) continue;
        if (in_batch == 0) {
          batches.push_back({(int32_t)pairs.size(), (int32_t)pairs.size(), (int64_t)nnear_all, (int64_t)nfar_all, L, 0});
          batch_hh.push_back(hh.size());
        }
        pairs.push_back(po.pr);
        hh.insert(hh.end(), po.h.begin(), po.h.end());
        nnear_all += nnear(L);
        nfar_all += nfar(L);
        batches.back().b1 = (int32_t)pairs.size();
        if (++in_batch == per) in_batch = 0;
      }
  }
  if (hh.size() > (size_t)INT32_MAX) return fail(CTC_ERR_UNSUPPORTED, "ESP: too many pair coefficients");
  // near- and far-field polynomials, batches shared out over the host threads
  static const EspMaps maps;
  std::vector<double> hv(nnear_all, 0.0), fv(nfar_all, 0.0);
  {
    auto form = [&](size_t first, size_t step) {
      for (size_t b = first; b < batches.size(); b += step) {
        const EspBatch& bt = batches[b];
        const int L = bt.L, last = ntuv(L) - 1;
        for (int i = bt.b0; i < bt.b1; ++i) {
          const size_t k = i - bt.b0;
          const double* h = &hh[batch_hh[b] + k * ntuv(L)];
          double* nv = hv.data() + bt.h0 + k * nnear(L);
          double* fp = fv.data() + bt.f0 + k * nfar(L);
          const double f0c = pairs[i].f0c;
          for (const MapTerm& t : maps.near[L]) nv[t.out] += t.f * h[t.in];
          for (const MapTerm& t : maps.far[L]) (t.out == last ? pairs[i].c0 : fp[t.out]) += f0c * t.f * h[t.in];
        }
      }
    };
    const unsigned nt = (unsigned)std::min<size_t>(nthr, batches.size() / 8 + 1);
    std::vector<std::thread> tf;
    for (unsigned t = 1; t < nt; ++t) tf.emplace_back(form, t, nt);
    form(0, nt);
    for (auto& t : tf) t.join();
  }
  const std::vector<double>& tab = boys_table();
  std::vector<double> atoms(4 * (size_t)std::max(mol->natom, 1));
  for (int a = 0; a < mol->natom; ++a) {
    atoms[4 * a] = mol->atom_xyz[3 * a];
    atoms[4 * a + 1] = mol->atom_xyz[3 * a + 1];
    atoms[4 * a + 2] = mol->atom_xyz[3 * a + 2];
    atoms[4 * a + 3] = mol->charges[a];
  }
  EspTables* e = new EspTables();
  mol->esp = e;
  for (const EspBatch& bt : batches) {
    const int np = bt.b1 - bt.b0;
    e->flops_per_point += (double)np * far_flops(bt.L);
    e->mean_L += (double)np * bt.L;
  }
  if (!pairs.empty()) e->mean_L /= (double)pairs.size();
  e->npairs = (int)pairs.size();
  e->nbatch = (int)batches.size();
  e->s_only = batches.empty() || batches.back().L == 0;
  e->natom = mol->natom;
  e->nh = hh.size();
  auto up = [&](void** dst, const void* src, size_t bytes) -> int {
    if (bytes == 0) bytes = 8;
    CTC_CUDA_TRY(cudaMalloc(dst, bytes));
    if (src) CTC_CUDA_TRY(cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice));
    return CTC_OK;
  };
  int rc;
  if ((rc = up((void**)&e->d_boys, tab.data(), tab.size() * sizeof(double))) ||
      (rc = up((void**)&e->d_pairs, pairs.empty() ? nullptr : pairs.data(), pairs.size() * sizeof(EspPair))) ||
      (rc = up((void**)&e->d_h, hv.empty() ? nullptr : hv.data(), hv.size() * sizeof(double))) ||
      (rc = up((void**)&e->d_far, fv.empty() ? nullptr : fv.data(), fv.size() * sizeof(double))) ||
      (rc = up((void**)&e->d_batches, batches.empty() ? nullptr : batches.data(), batches.size() * sizeof(EspBatch))) ||
      (rc = up((void**)&e->d_atoms, atoms.data(), atoms.size() * sizeof(double)))) {
    destroy_esp(mol);
    return rc;
  }
  mol->esp_valid = true;
  if (std::getenv("CTC_LOG"))
    std::fprintf(stderr, "[ctc] esp tables: %d primitive pairs, %d batches, %zu Hermite coefficients\n",
                 e->npairs, e->nbatch, e->nh);
  return CTC_OK;
}

int esp_info(ctc_molecule* mol, double* info) {
  if (!mol->esp_valid) {
    int rc = build_esp(mol);
    if (rc != CTC_OK) return rc;
  }
  info[0] = mol->esp->npairs;
  info[1] = mol->esp->flops_per_point;
  info[2] = (double)mol->esp->nh;
  info[3] = mol->esp->mean_L;
  return CTC_OK;
}

int eval_esp(ctc_molecule* mol, const double* d_points, int64_t n, double* d_out, cudaStream_t st) {
  if (n < 0) return fail(CTC_ERR_INVALID, "eval_esp: negative point count");
  if (n == 0) return CTC_OK;
  if (!mol->esp_valid) {
    int rc = build_esp(mol);
    if (rc != CTC_OK) return rc;
  }
  const EspTables* e = mol->esp;
  int nsm = 148;
  if (int rc = device_sm_count(&nsm); rc != CTC_OK) return rc;
  double lo[3], ext = 0;
  morton_box(mol, lo, &ext);
  const int bits = morton_axis_bits(ext);
  // points per pass: bounds the partial-sum rows (rows x points x 8 B)
  int64_t pass = (int64_t)1 << 22;
  int most_slices = 16383;  // (four times as many fit the grid's y)
  int near_factor = 4;
  for (int64_t p0 = 0, m = 0; p0 < n; p0 += m) {
    const double* pts = d_points + 3 * p0;
    int P = 1, S = 0, SN = 0;
    int64_t gx = 0;
    bool sort = false;
    size_t tmp_bytes = 0;
    double *part = nullptr, *xyz = nullptr;
    uint32_t *k_in = nullptr, *k_out = nullptr;
    int32_t *v_in = nullptr, *perm = nullptr;
    void* tmp = nullptr;
    // One layout gives both the size of the block and the places in it (S and SN
    // are zero when no pair is kept; the finish kernel then reads no row).
    auto lay_out = [&](char* base) {
      Carve cv{base};
      part = cv.take<double>((size_t)(S + SN) * m);
      xyz = cv.take<double>(3 * (size_t)m);
      perm = nullptr;  // (a larger pass that did not fit may have been sorted)
      if (sort) {
        k_in = cv.take<uint32_t>(m);
        k_out = cv.take<uint32_t>(m);
        v_in = cv.take<int32_t>(m);
        perm = cv.take<int32_t>(m);
        tmp = cv.take<char>(tmp_bytes);
      }
      return cv.off;
    };
    for (;;) {
      m = std::min(pass, n - p0);
      // two points per thread share a pair's coefficients; one when the points
      // would fill less than a block per SM (the pairs are then cut into more
      // slices)
      P = m >= (int64_t)2 * kEspThreads * nsm ? 2 : 1;
      gx = (m + P * kEspThreads - 1) / (P * kEspThreads);
      // slices of the batches: about 32 blocks per SM, at least a batch each
      const int64_t want = (32 * (int64_t)nsm + gx - 1) / gx;
      S = e->nbatch == 0 ? 0 : (int)std::max<int64_t>(1, std::min<int64_t>({want, (int64_t)e->nbatch, (int64_t)most_slices}));
      // near pairs cluster in few batches: four times as many slices for them (near
      // kernel at 1e5 surface points of 100 atoms: 40 -> 26 ms)
      SN = std::min(near_factor * S, e->nbatch);
      sort = m > kEspThreads;
      if (sort)
        CTC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                                     (int32_t*)nullptr, (int32_t*)nullptr, (int)m, 0, 3 * bits, st));
      const int rc = mol->ws_esp.ensure(lay_out(nullptr), st);
      if (rc == CTC_OK) break;
      // no room: fewer slices, then fewer points per pass (the sums' order follows
      // the slices, so results then differ in the last bits)
      if (rc != CTC_ERR_NOMEM) return rc;
      if (S > 1) most_slices = S / 2;
      else if (near_factor > 1) near_factor = 1;
      else if (m > kEspThreads) pass = std::max<int64_t>(kEspThreads, m / 2);
      else return rc;
    }
    lay_out((char*)mol->ws_esp.p);
    const unsigned g = (unsigned)((m + 255) / 256);
    if (sort) {
      morton_kernel<<<g, 256, 0, st>>>(pts, m, lo[0], lo[1], lo[2], (1 << bits) / ext, bits, k_in, v_in);
      CTC_CUDA_TRY(cudaGetLastError());
      CTC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k_in, k_out, v_in, perm, (int)m, 0,
                                                   3 * bits, st));
    }
    esp_gather_kernel<<<g, 256, 0, st>>>(pts, perm, m, xyz);
    CTC_CUDA_TRY(cudaGetLastError());
    if (S > 0) {
      const dim3 grid((unsigned)gx, (unsigned)S), ngrid((unsigned)gx, (unsigned)SN);
      double* near = part + (int64_t)S * m;
      if (P == 2) esp_far_kernel<2><<<grid, kEspThreads, 0, st>>>(e->d_pairs, e->d_far, e->d_batches, e->nbatch, xyz, m, part);
      else esp_far_kernel<1><<<grid, kEspThreads, 0, st>>>(e->d_pairs, e->d_far, e->d_batches, e->nbatch, xyz, m, part);
      CTC_CUDA_TRY(cudaGetLastError());
      if (P == 2) esp_near_kernel<2><<<ngrid, kEspThreads, 0, st>>>(e->d_pairs, e->d_h, e->d_far, e->d_batches, e->nbatch, e->d_boys, xyz, m, near);
      else esp_near_kernel<1><<<ngrid, kEspThreads, 0, st>>>(e->d_pairs, e->d_h, e->d_far, e->d_batches, e->nbatch, e->d_boys, xyz, m, near);
      CTC_CUDA_TRY(cudaGetLastError());
    }
    esp_finish_kernel<<<g, 256, 0, st>>>(part, S + SN, e->d_atoms, e->natom, xyz, perm, m, e->s_only, d_out + p0);
    CTC_CUDA_TRY(cudaGetLastError());
  }
  return CTC_OK;
}

}  // namespace ctc
