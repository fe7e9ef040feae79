// ctc_fp64.cuh -- FP64 contraction of the screened tile pipeline: G = A_t D[S_t, S_t]
// on the double-precision matrix units (mma.sync m8n8k4 f64), fused with the
// epilogue that reduces every finished 64-column slice of G against the AO
// values of its columns.
//
// What bounds it: the FP64 matrix pipe (64 FMA per clock and SM; the matrix
// and the vector form reach the same 36 TFLOP/s).  Two things follow.
//
// 1. Work.  D is symmetric, so a row pair (X, Y) needs only the blocks of D on
//    and above the diagonal:
//      sum_{mu nu} X_mu D_mu,nu Y_nu = 1/2 sum_nu (G^X_nu Y_nu + G^Y_nu X_nu),
//      G^X_nu = 2 sum_{mu in earlier blocks} X_mu D_mu,nu + sum_{mu in nu's block}.
//    (rho: X = Y = phi; the d_i phi d_j phi part of the Hessian and tau:
//    X = d_i phi, Y = d_j phi.)  Only rows that are also reduced against
//    quantities without a row of their own need the full sum: G0 = phi D with
//    d_i d_j phi, or with d_k phi when the tile has phi rows only.  With rows
//    phi, d_x, d_y, d_z phi the multiply-adds fall from 4 to about 2.5 per
//    (mu, nu), with phi rows alone (density only) from 1 to about 1/2.  A D
//    that is not symmetric (flag of density_kernel) takes the full sums.
// 2. Rate.  One persistent CTA per SM with separate warps for the loads, the
//    matrix instructions and the epilogue, so that index loads, gathers of D
//    and the epilogue's AO reads run beside the matrix pipe: 4 producer warps
//    (A rows by bulk copies, D gathered by compact index; 3 stages of 32 mu),
//    8 matrix warps, 4 epilogue warps working on the previous slice.
//
// Measured (one B200, device time of the kernel; before: one CTA per tile whose
// eight warps loaded, multiplied and reduced in turn, full sums, four rows per
// point for forces):
//   all descriptors, 200 atoms (2 691 functions, ~1 330 per tile), 90 945 grid
//     points: 70.8 -> 36.2 ms;  60 atoms (820), 20 011 points: 2.97 -> 1.39 ms
//   density, 12 atoms (160), 100 000 points: 276 -> 127 us; 200 points: 58 -> 13 us
//   rho and gradient (full sums), 60 atoms, 268 800 points: 10.1 -> 7.1 ms
//   dL/dR, same points: 60.8 -> 15.8 ms; 64 points: 1 830 -> 834 us (tiles of 32)
//
// Every barrier wait is bounded (ctc_molecule_set_wait_limit): after the limit a
// role sets the CTA's abort flag and stops, the others' waits run out in turn, and
// the CTA records kStatusFp64Timeout and exits once its copies have landed.
#pragma once

#include "ctc_internal.h"
#include "ctc_finalize.cuh"
#include "ctc_mbar.cuh"

namespace ctc {
namespace {

constexpr int kFN = 64;        // nu columns per slice
constexpr int kFK = 32;        // mu per pipeline stage
constexpr int kFStages = 3;
constexpr int kFRows = 128;    // rows of a wide stage
constexpr int kFALd = kFRows + 4;  // A stage [mu][row]: conflict-free fragment loads
constexpr int kFBLd = kFN + 4;     // B stage [mu][nu]
constexpr int kFGLd = kFRows + 2;  // G slice [nu][row]: conflict-free fragment stores
constexpr int kFAStage = kFK * kFALd, kFBStage = kFK * kFBLd;
constexpr int kFThreads = 512;     // warps 0-3 producers, 4-7 epilogue, 8-15 matrix
constexpr size_t kFSmem = sizeof(double) * (kFStages * (kFAStage + kFBStage) + kFN * kFGLd);
constexpr int kFSums = 19;         // per-point sums of the widest epilogue
constexpr int kFProducerRegs = 112, kFEpilogueRegs = 128, kFMatrixRegs = 136;
static_assert(128 * kFProducerRegs + 128 * kFEpilogueRegs + 256 * kFMatrixRegs <= kFThreads * 128,
              "register split above the launch's total");
static_assert(kKtAlign % kFN == 0 && kFN % kFK == 0, "tile K alignment");
constexpr int32_t kStatusFp64Timeout = 0x7102;
constexpr long long kLandCycles = 100000000LL;  // ~50 ms; a copy takes microseconds

// What a launch computes.
enum Fp64Mode {
  kFLocal4 = 0,   // 32 points x {phi, d_x, d_y, d_z phi}, local descriptors
  kFLocal1 = 1,   // 128 points x phi, local descriptors
  kFSmall1 = 2,   // 32 points x phi, local descriptors (few tiles: more CTAs busy)
  kFForce2 = 3,   // 64 points x {phi, w}, dL/dR with dL/d(grad rho)
  kFForce1 = 4,   // 128 points x phi, dL/dR without it
  kFForce2S = 5,  // 32 points x {phi, w}: kFForce2 for few points
};
constexpr int fp64_points(int mode) {
  return mode == kFLocal4 || mode == kFSmall1 || mode == kFForce2S ? 32 : (mode == kFForce2 ? 64 : 128);
}

struct Fp64Args {
  TileBatch tb;
  const double* D;
  int Mpad;
  const int32_t* sym;   // device flag: D is symmetric
  int32_t* status;
  long long wait_cycles;
  // local descriptors
  ctc_outputs out;
  ctc_params prm;
  // forces: per-point dL/drho and dL/dgrad rho indexed by the original point,
  // AO -> atom map, dL/dR accumulator
  const double* v_rho;
  const double* v_grad;
  const int32_t* ao_atom;
  double* dLdR;
  int natom;
};

// bytes (a multiple of 16; both addresses 16-byte aligned) global -> shared,
// counted on bar
__device__ __forceinline__ void bulk_copy(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(smem)),
               "l"(gmem), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// The stages of slice nt, walked alike by the producers and the matrix warps.
// Stages [0, wide) load all rows, [wide, total) the 32 phi rows only; before
// stage `twice` the rows that use the symmetry double their sums.
struct FSlice {
  int total, wide, twice;
};
template <int MODE>
__device__ __forceinline__ FSlice fslice(int nt, int nk, bool tri, int nq_ao) {
  const int diag = min(2 * nt + 2, nk);
  FSlice s{nk, nk, -1};
  if (MODE == kFLocal4) {
    if (tri) s = FSlice{nk, diag, nt > 0 ? 2 * nt : -1};
  } else if (MODE == kFLocal1) {
    if (tri && nq_ao == 1) s = FSlice{diag, diag, nt > 0 ? 2 * nt : -1};
  } else if (MODE == kFSmall1) {
    s.wide = 0;
    if (tri && nq_ao == 1) s = FSlice{diag, 0, nt > 0 ? 2 * nt : -1};
  }
  return s;
}

// Tile of this CTA's i-th turn: the tiles, most expensive first, are dealt out
// forwards and backwards in turn, so that every CTA's total is about the same.
__device__ __forceinline__ int fturn(const TileBatch& tb, int i) {
  const int64_t g = gridDim.x;
  const int64_t k = i * g + ((i & 1) ? g - 1 - (int64_t)blockIdx.x : (int64_t)blockIdx.x);
  return k < tb.C ? tb.order[k] : -1;
}

// Epilogue of 32 points x 4 rows: each of the four warps loads two to four AO
// quantities (lane = point) and forms the sums that use them.
//   role 0: q = 3 with rows 0..3, q = 4;  role 1: q = 2 with rows 0..3, q = 5
//   role 2: q = 1 with rows 0..3, q = 6;  role 3: q = 0, 7, 8, 9
__device__ __forceinline__ constexpr int frole_n(int role) { return role < 3 ? 2 : 4; }
__device__ __forceinline__ constexpr int frole_q(int role, int s) {
  return role == 3 ? (s == 0 ? 0 : 6 + s) : (s == 0 ? 3 - role : 4 + role);
}
__device__ __forceinline__ constexpr int frole_rows(int role, int s) { return role < 3 && s == 0 ? 4 : 1; }
// place of (slot, row) among the 19 sums: 0..9 G0 with quantity q; 10..15 G_i
// d_j phi, i <= j (xx xy xz yy yz zz); 16..18 yx zx zy
__device__ __forceinline__ constexpr int frole_sum(int role, int s, int row) {
  return row == 0 ? frole_q(role, s)
       : role == 0 ? (row == 1 ? 12 : (row == 2 ? 14 : 15))
       : role == 1 ? (row == 1 ? 11 : (row == 2 ? 13 : 18))
                   : (row == 1 ? 10 : (row == 2 ? 16 : 17));
}
// acc[i] += sum over the slice's columns; ao points at quantity 0, column 0 of
// the slice at this lane's point (element (q, c) at ao[q * ldq + c * 32])
template <int ROLE>
__device__ __forceinline__ void fcontract4(const double* __restrict__ ao, int64_t ldq,
                                           const double* __restrict__ sG, int lane, int nq_ao, int ncol,
                                           double* acc) {
  constexpr int NS = frole_n(ROLE);
  constexpr int W = NS == 2 ? 8 : 4;  // columns per batch; the next batch's loads are in flight
  bool live[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) live[s] = frole_q(ROLE, s) < nq_ao;
  double a[2][NS][W];
  auto load = [&](int buf, int c0) {
#pragma unroll
    for (int s = 0; s < NS; ++s)
#pragma unroll
      for (int j = 0; j < W; ++j)
        a[buf][s][j] = live[s] ? __ldg(ao + frole_q(ROLE, s) * ldq + (int64_t)(c0 + j) * 32) : 0.0;
  };
  auto reduce = [&](int buf, int c0) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const double* g = sG + (c0 + j) * kFGLd + lane;
      int i = 0;
#pragma unroll
      for (int s = 0; s < NS; ++s)
#pragma unroll
        for (int r = 0; r < frole_rows(ROLE, s); ++r, ++i) acc[i] = fma(g[r * 32], a[buf][s][j], acc[i]);
    }
  };
  // ncol is 32 or 64, a multiple of 2 W
  load(0, 0);
  for (int c0 = 0; c0 < ncol; c0 += 2 * W) {
    load(1, c0 + W);
    reduce(0, c0);
    if (c0 + 2 * W < ncol) load(0, c0 + 2 * W);
    reduce(1, c0 + W);
  }
}
template <int ROLE>
__device__ __forceinline__ void fstore4(double (*s_sums)[kFSums + 1], int lane, const double* acc) {
  int i = 0;
#pragma unroll
  for (int s = 0; s < frole_n(ROLE); ++s)
#pragma unroll
    for (int r = 0; r < frole_rows(ROLE, s); ++r, ++i) s_sums[lane][frole_sum(ROLE, s, r)] = acc[i];
}

// Epilogue of phi rows: acc[q] += sum over columns [c0, c1) of G A_q at point
// pc (element (q, c) at ao[q * ldq + c * PTS])
template <int NQ, int PTS>
__device__ __forceinline__ void fcontract1(const double* __restrict__ ao, int64_t ldq,
                                           const double* __restrict__ sG, int pc, int c0, int c1, double* acc) {
  constexpr int W = 8;
  for (int c = c0; c < c1; c += W) {
    double a[NQ][W];
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
      for (int j = 0; j < W; ++j) a[q][j] = __ldg(ao + q * ldq + (int64_t)(c + j) * PTS);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const double g = sG[(c + j) * kFGLd + pc];
#pragma unroll
      for (int q = 0; q < NQ; ++q) acc[q] = fma(g, a[q][j], acc[q]);
    }
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFThreads, 1) fp64_tile_kernel(const Fp64Args args) {
  constexpr int PTS = fp64_points(MODE);
  constexpr bool NARROW_ONLY = MODE == kFSmall1;
  constexpr bool HAS_NARROW = MODE == kFLocal4 || MODE == kFSmall1;
  constexpr bool FORCE2 = MODE == kFForce2 || MODE == kFForce2S;
  constexpr bool FORCE = MODE == kFForce1 || FORCE2;
  constexpr int ROWS = FORCE2 ? 2 * PTS : kFRows;  // rows of a wide stage in use
  extern __shared__ __align__(16) double fsmem[];
  double* sA = fsmem;
  double* sB = fsmem + kFStages * kFAStage;
  double* sG = fsmem + kFStages * (kFAStage + kFBStage);
  __shared__ __align__(8) uint64_t full_bar[kFStages], tma_bar[kFStages], empty_bar[kFStages], gfull_bar, gempty_bar, gwide_bar;
  __shared__ double s_sums[32][kFSums + 1];
  __shared__ int s_abort, s_epi_abort;
  __shared__ int s_issued[kFStages][2];  // stage counter of each half's last copies into a slot, -1: none

  const TileBatch& tb = args.tb;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFStages; ++s) {
      mbar_init(&full_bar[s], 64);
      mbar_init(&tma_bar[s], 2);
      mbar_init(&empty_bar[s], 8);
      s_issued[s][0] = s_issued[s][1] = -1;
    }
    mbar_init(&gfull_bar, 8);
    mbar_init(&gempty_bar, 4);
    mbar_init(&gwide_bar, 8);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  const bool tri = *args.sym != 0;
  const int nq_ao = tb.nq;
  const int64_t ldq = (int64_t)PTS * tb.Kcap;  // stride between AO quantities

  if (warp < 4) {
    // ---------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kFProducerRegs));
    // Warps 0-1 take the even stages of the CTA's sequence, warps 2-3 the odd
    // ones.  A thread gathers one nu column of D for 16 + 16 mu into registers,
    // the loads of its next stage in flight while this one waits for its slot;
    // the A rows are bulk copies of one (mu, quantity) run of points each.
    // (cp.async for both takes the L1 a cycle per lane: ~1.7 K for the D block
    // and ~2 K for the A rows of a stage whose matrix instructions take 4.1 K
    // with all rows and 1 K with the phi rows.)
    const int pair = warp >> 1, ptid = threadIdx.x & 63;
    const int khalf = warp & 1;  // bulk copies: mu 16 khalf .. + 15 by this warp
    struct Cur {
      int i, t, nk, nn, nt, kb, total, wide;
    };
    auto open_tile = [&](Cur& c) {  // first stage of the next tile that has any
      for (;; ++c.i) {
        c.t = fturn(tb, c.i);
        if (c.t < 0) return;
        c.nk = (tb.ktrue[c.t] + kFK - 1) / kFK;  // columns beyond ktrue are zero
        c.nn = (c.nk * kFK + kFN - 1) / kFN;
        if (c.nn > 0) break;
      }
      const FSlice fs = fslice<MODE>(0, c.nk, tri, nq_ao);
      c.nt = c.kb = 0;
      c.total = fs.total;
      c.wide = fs.wide;
    };
    auto advance = [&](Cur& c) {
      if (c.t < 0 || ++c.kb < c.total) return;
      c.kb = 0;
      if (++c.nt < c.nn) {
        const FSlice fs = fslice<MODE>(c.nt, c.nk, tri, nq_ao);
        c.total = fs.total;
        c.wide = fs.wide;
        return;
      }
      ++c.i;
      open_tile(c);
    };
    double v[kFK];
    unsigned ok = 0;  // mu of the stage that are not padding
    bool nu_ok = false;
    auto load_idx = [&](const Cur& c, int& mu, int& nu) {
      const int32_t* am = tb.aomap + (int64_t)c.t * tb.Kcap;
      mu = am[c.kb * kFK + lane];
      nu = am[c.nt * kFN + ptid];  // -1 beyond ktrue (padded to 64)
    };
    // loads without a condition (clamped index; the value is dropped later): a
    // condition on each makes the compiler wait for one before the next
    auto gather = [&](int mu, int nu) {
      ok = __ballot_sync(0xffffffffu, mu >= 0);
      nu_ok = nu >= 0;
      const int m = max(mu, 0);
      const double* d = args.D + max(nu, 0);
#pragma unroll
      for (int k = 0; k < kFK; ++k) v[k] = __ldg(d + (int64_t)__shfl_sync(0xffffffffu, m, k) * args.Mpad);
    };
    Cur cur{};
    open_tile(cur);
    if (pair) advance(cur);
    if (cur.t >= 0) {
      int mu, nu;
      load_idx(cur, mu, nu);
      gather(mu, nu);
    }
    for (int it = pair; cur.t >= 0; it += 2) {
      Cur nxt = cur;
      advance(nxt);
      advance(nxt);
      int mu = -1, nu = -1;
      if (nxt.t >= 0) load_idx(nxt, mu, nu);
      const int s = it % kFStages;
      if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], ((it / kFStages) & 1) ^ 1, args.wait_cycles))) {
        s_abort = 1;
        break;
      }
      double* a = sA + s * kFAStage;
      double* b = sB + s * kFBStage;
      {
        const double* A = tb.ao + (int64_t)cur.t * nq_ao * ldq + (int64_t)cur.kb * kFK * PTS;
        const bool wide = !NARROW_ONLY && cur.kb < cur.wide;
        constexpr int NRUN = MODE == kFLocal4 ? 4 : (FORCE2 ? 2 : 1);  // quantities of a wide stage
        const int runs = wide ? NRUN : 1;
        if (lane == 0) {
          s_issued[s][khalf] = it;
          mbar_arrive_expect_tx(&tma_bar[s], 16 * runs * PTS * 8);
        }
        __syncwarp();
        for (int x = lane; x < 16 * runs; x += 32) {
          const int kk = 16 * khalf + x / runs, r = x % runs;
          const int q = FORCE2 ? 10 * r : r;
          bulk_copy(a + kk * kFALd + r * PTS, A + q * ldq + (int64_t)kk * PTS, PTS * 8, &tma_bar[s]);
        }
      }
#pragma unroll
      for (int k = 0; k < kFK; ++k) b[k * kFBLd + ptid] = (nu_ok && ((ok >> k) & 1u)) ? v[k] : 0.0;
      mbar_arrive(&full_bar[s]);
      if (nxt.t >= 0) gather(mu, nu);
      cur = nxt;
    }
  } else if (warp >= 8) {
    // ---------------- matrix warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kFMatrixRegs));
    const int w = warp - 8, wm = w & 3, wn = w >> 2;  // wide: 32 x 32 block (wm, wn) of 128 x 64
    const int fk = lane & 3, fr = lane >> 2;
    int it = 0, gs = 0, ga = 0;  // stages, slices, slices with both wide and narrow sums
    bool stop = false;
    for (int i = 0; !stop; ++i) {
      const int t = fturn(tb, i);
      if (t < 0) break;
      const int nk = (tb.ktrue[t] + kFK - 1) / kFK;
      const int nn = (nk * kFK + kFN - 1) / kFN;
      for (int nt = 0; nt < nn && !stop; ++nt, ++gs) {
        const FSlice fs = fslice<MODE>(nt, nk, tri, nq_ao);
        const int ncol = min(kFN, nk * kFK - nt * kFN);  // 32 or 64
        const bool on_w = wn * 32 < ncol && wm * 32 < ROWS, on_n = w * 8 < ncol;
        double c[4][4][2];  // wide accumulators
        double d[4][2];     // narrow: rows 0..31, columns w * 8 ..
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          d[a][0] = d[a][1] = 0.0;
#pragma unroll
          for (int b = 0; b < 4; ++b) c[a][b][0] = c[a][b][1] = 0.0;
        }
        for (int kb = 0; kb < fs.total; ++kb, ++it) {
          const int s = it % kFStages;
          const uint32_t ph = (it / kFStages) & 1;
          const bool ready = mbar_wait(&full_bar[s], ph, args.wait_cycles) && mbar_wait(&tma_bar[s], ph, args.wait_cycles);
          if (!__all_sync(0xffffffffu, ready)) {
            s_abort = 1;
            stop = true;
            break;
          }
          const double* a = sA + s * kFAStage + fk * kFALd + fr;
          const double* b = sB + s * kFBStage + fk * kFBLd + fr;
          if (kb == fs.twice) {
            // rows that use the symmetry (kFLocal4: the derivative rows only)
            if (!NARROW_ONLY && (MODE != kFLocal4 || wm > 0)) {
#pragma unroll
              for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                  c[x][y][0] *= 2.0;
                  c[x][y][1] *= 2.0;
                }
            }
            if (NARROW_ONLY) {
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                d[x][0] *= 2.0;
                d[x][1] *= 2.0;
              }
            }
          }
          if (!NARROW_ONLY && kb < fs.wide) {
            if (on_w) {
#pragma unroll
              for (int ks = 0; ks < kFK; ks += 4) {
                double af[4], bf[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) af[x] = a[ks * kFALd + wm * 32 + x * 8];
#pragma unroll
                for (int y = 0; y < 4; ++y) bf[y] = b[ks * kFBLd + wn * 32 + y * 8];
#pragma unroll
                for (int x = 0; x < 4; ++x)
#pragma unroll
                  for (int y = 0; y < 4; ++y) dmma(c[x][y][0], c[x][y][1], af[x], bf[y]);
              }
            }
          } else if (HAS_NARROW && on_n) {
#pragma unroll
            for (int ks = 0; ks < kFK; ks += 4) {
              const double bf = b[ks * kFBLd + w * 8];
#pragma unroll
              for (int x = 0; x < 4; ++x) dmma(d[x][0], d[x][1], a[ks * kFALd + x * 8], bf);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty_bar[s]);
        }
        if (stop) break;
        // the epilogue has released the previous slice of G
        if (!__all_sync(0xffffffffu, mbar_wait(&gempty_bar, (gs & 1) ^ 1, args.wait_cycles))) {
          s_abort = 1;
          stop = true;
          break;
        }
        // C fragment: row lane / 4, columns 2 (lane % 4), + 1
        if (!NARROW_ONLY && on_w) {
#pragma unroll
          for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) {
              double* g = sG + (wn * 32 + y * 8 + 2 * fk) * kFGLd + wm * 32 + x * 8 + fr;
              g[0] = c[x][y][0];
              g[kFGLd] = c[x][y][1];
            }
        }
        if (HAS_NARROW) {
          const bool add = !NARROW_ONLY && fs.wide < fs.total;
          if (add) {  // the wide sums of every matrix warp are in shared memory
            __syncwarp();
            if (lane == 0) mbar_arrive(&gwide_bar);
            if (!__all_sync(0xffffffffu, mbar_wait(&gwide_bar, ga++ & 1, args.wait_cycles))) {
              s_abort = 1;
              stop = true;
              break;
            }
          }
          if ((NARROW_ONLY || add) && on_n) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              double* g = sG + (w * 8 + 2 * fk) * kFGLd + x * 8 + fr;
              g[0] = d[x][0] + (NARROW_ONLY ? 0.0 : g[0]);
              g[kFGLd] = d[x][1] + (NARROW_ONLY ? 0.0 : g[kFGLd]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&gfull_bar);
      }
    }
  } else {
    // ---------------- epilogue warps
    const int role = warp - 4;
    const int etid = role * 32 + lane;
    int gs = 0;
    bool stop = false;  // per warp; the four warps meet only in the bounded barriers below
    for (int i = 0;; ++i) {
      const int t = fturn(tb, i);
      if (t < 0) break;
      const int nk = (tb.ktrue[t] + kFK - 1) / kFK;
      const int nn = (nk * kFK + kFN - 1) / kFN;
      const int32_t* am = tb.aomap + (int64_t)t * tb.Kcap;
      const double* A = tb.ao + (int64_t)t * nq_ao * ldq;
      double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      // forces: weights of this lane's points, running sums of one atom
      constexpr int NP = FORCE ? PTS / 32 : 1;
      double vr[NP], vg[NP][3], fsum[3] = {0.0, 0.0, 0.0};
      bool live[NP];  // points without weight are left out, whatever their AO values
      int fatom = -1;
      if constexpr (FORCE) {
#pragma unroll
        for (int h = 0; h < NP; ++h) {
          const int64_t p = (int64_t)t * PTS + h * 32 + lane;
          const int64_t oi = tb.out[p];
          const bool ok = oi >= 0;
          vr[h] = ok ? args.v_rho[oi] : 0.0;
          for (int k = 0; k < 3; ++k) vg[h][k] = ok && FORCE2 ? args.v_grad[3 * oi + k] : 0.0;
          live[h] = !(vr[h] == 0.0 && vg[h][0] == 0.0 && vg[h][1] == 0.0 && vg[h][2] == 0.0);
        }
      }
      auto flush_atom = [&]() {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          double v = fsum[j];
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0 && fatom >= 0 && v != 0.0) atomicAdd(&args.dLdR[3 * fatom + j], v);
          fsum[j] = 0.0;
        }
      };
      for (int nt = 0; nt < nn; ++nt, ++gs) {
        const int ncol = min(kFN, nk * kFK - nt * kFN);
        if (!__all_sync(0xffffffffu, mbar_wait(&gfull_bar, gs & 1, args.wait_cycles))) {
          s_abort = 1;
          stop = true;
          break;
        }
        const double* ao = A + (int64_t)nt * kFN * PTS;
        if constexpr (MODE == kFLocal4) {
          switch (role) {
            case 0: fcontract4<0>(ao + lane, ldq, sG, lane, nq_ao, ncol, acc); break;
            case 1: fcontract4<1>(ao + lane, ldq, sG, lane, nq_ao, ncol, acc); break;
            case 2: fcontract4<2>(ao + lane, ldq, sG, lane, nq_ao, ncol, acc); break;
            default: fcontract4<3>(ao + lane, ldq, sG, lane, nq_ao, ncol, acc); break;
          }
        } else if constexpr (MODE == kFLocal1) {
          if (nq_ao == 1) fcontract1<1, PTS>(ao + etid, ldq, sG, etid, 0, ncol, acc);
          else fcontract1<4, PTS>(ao + etid, ldq, sG, etid, 0, ncol, acc);
        } else if constexpr (MODE == kFSmall1) {
          const int part = ncol / 4;  // columns of this warp (8 or 16)
          if (nq_ao == 1) fcontract1<1, PTS>(ao + lane, ldq, sG, lane, role * part, (role + 1) * part, acc);
          else fcontract1<4, PTS>(ao + lane, ldq, sG, lane, role * part, (role + 1) * part, acc);
        } else {
          // dL/dR_A,j = -2 sum over points, nu on atom A of
          //   d_j phi (v_rho G0 + sum_k v_k G_k) + G0 sum_k v_k d_j d_k phi,
          // v_rho G0 + sum_k v_k G_k = (w D)_nu with w = v_rho phi + sum_k v_k d_k phi
          constexpr int hidx[3][3] = {{4, 5, 6}, {5, 7, 8}, {6, 8, 9}};
          const int part = ncol / 4;
          for (int v = role * part; v < (role + 1) * part; ++v) {
            const int nu = am[nt * kFN + v];
            const int atom = nu >= 0 ? args.ao_atom[nu] : -1;  // uniform over the warp
            if (atom != fatom) {
              if (fatom >= 0) flush_atom();
              fatom = atom;
            }
            if (atom < 0) continue;
#pragma unroll
            for (int h = 0; h < NP; ++h) {
              if (!live[h]) continue;
              const int p = h * 32 + lane;
              const double* ap = ao + (int64_t)v * PTS + p;
              const double G0 = sG[v * kFGLd + p];
              const double Y = FORCE2 ? sG[v * kFGLd + (PTS % kFRows) + p] : vr[h] * G0;
              if constexpr (FORCE2) {
                double H[6];
#pragma unroll
                for (int x = 0; x < 6; ++x) H[x] = __ldg(ap + (4 + x) * ldq);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                  const double q = vg[h][0] * H[hidx[j][0] - 4] + vg[h][1] * H[hidx[j][1] - 4] + vg[h][2] * H[hidx[j][2] - 4];
                  fsum[j] -= 2.0 * (__ldg(ap + (1 + j) * ldq) * Y + q * G0);
                }
              } else {
#pragma unroll
                for (int j = 0; j < 3; ++j) fsum[j] -= 2.0 * __ldg(ap + (1 + j) * ldq) * Y;
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&gempty_bar);
      }
      if constexpr (FORCE) {
        if (__any_sync(0xffffffffu, stop || s_abort != 0)) break;
        if (fatom >= 0) flush_atom();
      } else {
        // the four warps' sums of a point meet in shared memory
        const int64_t p0 = (int64_t)t * PTS;
        if constexpr (MODE == kFLocal1) {
          if (__any_sync(0xffffffffu, stop || s_abort != 0)) break;
          const int64_t oidx = tb.out[p0 + etid];
          if (oidx >= 0) {
            double s16[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) s16[q] = q < 4 ? acc[q] : 0.0;
            if (finite_point(tb.xyz + 3 * (p0 + etid))) finalize_point(s16, 1, nq_ao, args.out, oidx, args.prm);
            else nan_point(args.out, oidx);
          }
        } else {
          if constexpr (MODE == kFLocal4) {
            switch (role) {
              case 0: fstore4<0>(s_sums, lane, acc); break;
              case 1: fstore4<1>(s_sums, lane, acc); break;
              case 2: fstore4<2>(s_sums, lane, acc); break;
              default: fstore4<3>(s_sums, lane, acc); break;
            }
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) s_sums[lane][role * 4 + q] = acc[q];
          }
          // every epilogue warp takes part, stopped or not, and all four take the
          // same decision from one thread's reading, so none is left waiting
          if (etid == 0) s_epi_abort = s_abort;
          asm volatile("bar.sync 1, 128;\n" ::: "memory");
          const bool bad = s_epi_abort != 0;
          const int64_t oidx = tb.out[p0 + lane];
          if (role == 0 && !bad && oidx >= 0) {
            double s16[16];
            if constexpr (MODE == kFLocal4) {
#pragma unroll
              for (int q = 0; q < 16; ++q) s16[q] = s_sums[lane][q];
              if (tri) {
                s16[11] = 0.5 * (s16[11] + s_sums[lane][16]);
                s16[12] = 0.5 * (s16[12] + s_sums[lane][17]);
                s16[14] = 0.5 * (s16[14] + s_sums[lane][18]);
              }
            } else {
#pragma unroll
              for (int q = 0; q < 16; ++q)
                s16[q] = q < 4 ? (s_sums[lane][q] + s_sums[lane][4 + q]) + (s_sums[lane][8 + q] + s_sums[lane][12 + q]) : 0.0;
            }
            if (finite_point(tb.xyz + 3 * (p0 + lane))) finalize_point(s16, MODE == kFLocal4 ? 4 : 1, nq_ao, args.out, oidx, args.prm);
            else nan_point(args.out, oidx);
          }
          asm volatile("bar.sync 1, 128;\n" ::: "memory");  // s_sums may be written again
          if (bad) break;
        }
      }
    }
  }
  __syncthreads();
  // No copy may land after the CTA has left.  After a normal end the matrix warps
  // have waited for every one.  After a timeout in any role -- every warp is here,
  // so s_abort is final and nothing is issued any more -- copies may be on their
  // way, also those of producers that ended normally.  A slot's last stage is
  // waited for with the full limit; where one of its two warps has not issued its
  // half, the phase cannot end and kLandCycles gives the other half time to land.
  if (s_abort && threadIdx.x == 0) {
    for (int s = 0; s < kFStages; ++s) {
      const int x = s_issued[s][0], y = s_issued[s][1], last = max(x, y);
      if (last >= 0) mbar_wait(&tma_bar[s], (last / kFStages) & 1, x == y ? kWaitCycles : kLandCycles);
    }
    atomicExch(args.status, kStatusFp64Timeout);
  }
}

// Launches one chunk; args holds what the mode needs beyond the tiles.
template <int MODE>
int launch_fp64(ctc_molecule* mol, const TileBatch& tb, Fp64Args args, cudaStream_t st) {
  if (int rc = ensure_smem_attr((const void*)fp64_tile_kernel<MODE>, (int)kFSmem); rc != CTC_OK) return rc;
  int nsm = 0;
  if (int rc = device_sm_count(&nsm); rc != CTC_OK) return rc;
  args.tb = tb;
  args.D = mol->d_D;
  args.Mpad = mol->Mpad;
  args.sym = mol->d_sym;
  args.status = mol->d_status;
  args.wait_cycles = mol->wait_cycles > 0 ? (long long)mol->wait_cycles : kWaitCycles;
  fp64_tile_kernel<MODE><<<tb.C < nsm ? tb.C : nsm, kFThreads, kFSmem, st>>>(args);
  CTC_CUDA_TRY(cudaGetLastError());
  return CTC_OK;
}

}  // namespace
}  // namespace ctc
