// ctc_ao.cu -- contracted Gaussian AOs and their first/second derivatives on points.
//
// Restates the reference's AO evaluation (src/evaluate_density.cu:25-393,
// src/evaluate_gradient.cu:18-1127, src/evaluate_hessian.cu:17-1835) in one
// generic form.  Every AO component of a segment is
//     phi_j(r) = sum_t c_t x^a y^b z^c * R0(r^2),   R0 = sum_k coef_k exp(-alpha_k r^2)
// (x, y, z relative to the shell centre; c_t from gen_terms.py).  With
// R1 = sum_k alpha_k coef_k exp(..) and R2 = sum_k alpha_k^2 coef_k exp(..) the
// derivatives follow from those of the angular polynomial (gen_ao_poly.py), so
// one exponential per primitive serves every component and derivative.
//
// A warp evaluates one segment at 32 points, so it runs one code path.  A
// segment whose centre is farther than its screening radius from the point
// (every value and derivative below 1e-18) writes zeros without evaluating
// exponentials.  Arithmetic is FP64 throughout.
#include <algorithm>

#include "ctc_internal.h"
#include "ctc_split.cuh"

namespace ctc {

namespace {

constexpr int kAoThreads = 128;

// High 32 bits of |x| (sign cleared): ordered like |x|, and bits 20..30 hold
// the biased exponent.
__device__ __forceinline__ unsigned abs_hi(double x) {
  return (unsigned)__double2hiint(x) & 0x7fffffffu;
}

#include "ctc_ao_poly.inc"

// Evaluation of one segment at one point: the polynomial code of every
// component has literal exponents (ctc_ao_poly.inc), so the powers stay in
// registers.  Entry (quantity q, component j) goes to o[q * ld_q + j * ldc];
// outside the screening radius every entry is zero.
template <int DERIV, int TYPE, int TRACK>
__device__ __forceinline__ void eval_typed(const DevSeg& sg, const double* __restrict__ alpha,
                                           const double* __restrict__ coef, double px, double py,
                                           double pz, double* __restrict__ o, int64_t ld_q,
                                           int64_t ldc, int nq_out, unsigned* mx, const double* wv) {
  constexpr int L = TYPE == 0 ? 0 : (TYPE == 1 ? 1 : (TYPE <= 3 ? 2 : (TYPE <= 5 ? 3 : 4)));
  constexpr int NC = TYPE == 0 ? 1 : TYPE == 1 ? 3 : TYPE == 2 ? 6 : TYPE == 3 ? 5
                     : TYPE == 4 ? 10 : TYPE == 5 ? 7 : TYPE == 6 ? 15 : 9;
  constexpr int NP = L + 2;  // powers x^i for i < NP
  const double x = px - sg.cx, y = py - sg.cy, z = pz - sg.cz;
  const double r2 = x * x + y * y + z * z;
  if (r2 > sg.rcut2) {
    for (int q = 0; q < nq_out; ++q)
#pragma unroll
      for (int j = 0; j < NC; ++j) o[q * ld_q + j * ldc] = 0.0;
    return;
  }
  double R0 = 0.0, R1 = 0.0, R2 = 0.0;
  for (int k = 0; k < sg.nprim; ++k) {
    const double a = alpha[sg.prim0 + k];
    const double e = coef[sg.prim0 + k] * exp(-a * r2);
    R0 += e;
    if (DERIV >= 1) R1 += a * e;
    if (DERIV >= 2) R2 += a * a * e;
  }
  double X[NP], Y[NP], Z[NP];
  X[0] = Y[0] = Z[0] = 1.0;
#pragma unroll
  for (int i = 1; i < NP; ++i) {
    X[i] = X[i - 1] * x;
    Y[i] = Y[i - 1] * y;
    Z[i] = Z[i - 1] * z;
  }
  if constexpr (TYPE == 0) ao_poly_0<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 1) ao_poly_1<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 2) ao_poly_2<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 3) ao_poly_3<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 4) ao_poly_4<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 5) ao_poly_5<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else if constexpr (TYPE == 6) ao_poly_6<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
  else ao_poly_7<DERIV, TRACK>(X, Y, Z, R0, R1, R2, o, ld_q, ldc, nq_out, mx, wv);
}

template <int DERIV, int TRACK>
__device__ __forceinline__ void eval_dispatch(const DevSeg& sg, const double* __restrict__ alpha,
                                              const double* __restrict__ coef, double px, double py,
                                              double pz, double* __restrict__ o, int64_t ld_q,
                                              int64_t ldc, int nq_out, unsigned* mx, const double* wv) {
  switch (sg.type) {
    case 0: eval_typed<DERIV, 0, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 1: eval_typed<DERIV, 1, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 2: eval_typed<DERIV, 2, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 3: eval_typed<DERIV, 3, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 4: eval_typed<DERIV, 4, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 5: eval_typed<DERIV, 5, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    case 6: eval_typed<DERIV, 6, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
    default: eval_typed<DERIV, 7, TRACK>(sg, alpha, coef, px, py, pz, o, ld_q, ldc, nq_out, mx, wv); break;
  }
}

// AO values in the public layout out[q][point][AO] (AO in the caller's order,
// fastest).  Bound: the writes, 8 nq M bytes per point.  A CTA takes 32 points
// and a chunk of whole segments with at most ao_chunk(DERIV) consecutive AOs:
// its warps evaluate a segment at a time, lane = point, into a padded block in
// shared memory (conflict-free both ways), from which every (quantity, point)
// row of the chunk is written as one run of consecutive addresses.  (One thread
// per segment and point, stores M doubles apart and the terms read from
// constant memory, took 990 us for values and gradients of 820 functions at
// 30 000 points, 0.8 TB/s; this form 328 us, 420 with 32
// AOs per chunk.)
constexpr int kAoPubThreads = 256;
__host__ __device__ constexpr int ao_chunk(int deriv) { return deriv == 2 ? 32 : 64; }
__host__ __device__ constexpr size_t ao_pub_smem(int deriv) {
  return sizeof(double) * (deriv == 0 ? 1 : (deriv == 1 ? 4 : 10)) * 32 * (ao_chunk(deriv) + 1);
}
template <int DERIV>
__global__ void __launch_bounds__(kAoPubThreads)
    ao_public_kernel(const DevSeg* __restrict__ segs, const int32_t* __restrict__ order,
                     const int2* __restrict__ chunks, int nchunk, int nseg, const double* __restrict__ alpha,
                     const double* __restrict__ coef, const double* __restrict__ pts, int64_t n, int M,
                     double* __restrict__ out) {
  constexpr int NQ = DERIV == 0 ? 1 : (DERIV == 1 ? 4 : 10);
  constexpr int LD = ao_chunk(DERIV) + 1;  // row of one (quantity, point)
  extern __shared__ __align__(16) double s_ao[];  // [NQ][32][LD]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t items = (n + 31) / 32 * nchunk;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int64_t p0 = it / nchunk * 32;
    const int2 ck = chunks[it % nchunk];  // segments [ck.x, ck.y) of the order
    const int np = (int)min((int64_t)32, n - p0);
    const double* x = pts + 3 * (p0 + min(lane, np - 1));
    const double px = x[0], py = x[1], pz = x[2];
    const int c0 = segs[order[ck.x]].orig_ao0;
    for (int i = ck.x + warp; i < ck.y; i += kAoPubThreads / 32) {
      const DevSeg sg = segs[order[i]];
      eval_dispatch<DERIV, 0>(sg, alpha, coef, px, py, pz, s_ao + lane * LD + (sg.orig_ao0 - c0), 32 * LD, 1, NQ,
                              nullptr, nullptr);
    }
    __syncthreads();
    const int nc = (ck.y < nseg ? segs[order[ck.y]].orig_ao0 : M) - c0;
    for (int r = warp; r < NQ * 32; r += kAoPubThreads / 32) {
      const int q = r >> 5, p = r & 31;
      if (p >= np) continue;
      double* row = out + ((int64_t)q * n + p0 + p) * M + c0;
      for (int c = lane; c < nc; c += 32) row[c] = s_ao[r * LD + c];
    }
    __syncthreads();
  }
}

// One CTA per tile; each warp takes one significant segment at a time and
// its lanes take the tile's points, so a warp always runs one segment type
// and its stores of one (quantity, AO) cover consecutive points.  Layout of
// the tile block: A[q][k][point] (point fastest).  Padding columns
// [ktrue, kt) are zeroed.
//
// SLICE = 4 or 1 also produces the row exponents of the tensor-core split
// operands of the tile (ctc_split.cuh): the rows are the tile's points x {phi,
// d_x, d_y, d_z phi} (SLICE = 4, blocks of 32 points x 4 quantities, TP = 32)
// or its points x phi (SLICE = 1, TP <= 256).  Every lane keeps the running
// maximum of its values while it evaluates, so the exponents cost no second
// pass over the block; slice_rows_kernel then writes the digit planes.
//
// With SLICE = 0 a tile's segments may be dealt out to gridDim.y CTAs.
//
// SLICE = -1 or -2 is the adjoint's form: from the weights of the tile's points
// (dL/drho, dL/dgrad rho at their original index) it also writes the row
// w = v_rho phi + v_grad . grad phi, as quantity 10 behind the ten AO quantities
// (-1) or as the only one besides phi (-2, dL/dD alone).  The contraction for
// dL/dR then needs two rows per point instead of four, and dL/dD reads two
// quantities instead of four.
template <int DERIV, int SLICE>
__global__ void __launch_bounds__(kAoThreads, 3)
    ao_tile_kernel(const DevSeg* __restrict__ segs, int nseg, const double* __restrict__ alpha,
                   const double* __restrict__ coef, TileBatch tb, int32_t* __restrict__ eexp,
                   const int32_t* __restrict__ order, const double* __restrict__ v_rho,
                   const double* __restrict__ v_grad) {
  // per-warp maxima of the high word of |value| per row, [warp][row]
  constexpr int kMaxRows = 256;
  __shared__ unsigned s_mx[SLICE > 0 ? kAoThreads / 32 : 1][SLICE > 0 ? kMaxRows : 1];
  const int t = order ? order[blockIdx.x] : blockIdx.x;
  const int ns = tb.nsig[t], TP = tb.TP;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int32_t* sl = tb.segs + (int64_t)t * nseg;
  const int32_t* k0 = tb.k0 + (int64_t)t * nseg;
  const double* xyz = tb.xyz + (int64_t)t * TP * 3;
  double* A = tb.ao + (int64_t)t * tb.nq * TP * tb.Kcap;
  const int64_t ld_q = (int64_t)TP * tb.Kcap;
  for (int pg = 0; pg < TP; pg += 32) {
    const int j = pg + lane;
    const double px = xyz[3 * j], py = xyz[3 * j + 1], pz = xyz[3 * j + 2];
    unsigned mx[4] = {0u, 0u, 0u, 0u};
    double wv[4] = {0.0, 0.0, 0.0, 0.0};
    if (SLICE < 0) {
      const int64_t oi = tb.out[(int64_t)t * TP + j];
      if (oi >= 0) {
        wv[0] = v_rho[oi];
        for (int k = 0; k < 3; ++k) wv[1 + k] = v_grad[3 * oi + k];
      }
    }
    for (int i = warp + blockIdx.y * (kAoThreads / 32); i < ns; i += gridDim.y * (kAoThreads / 32)) {
      const DevSeg sg = segs[sl[i]];
      eval_dispatch<DERIV, SLICE>(sg, alpha, coef, px, py, pz, A + (int64_t)k0[i] * TP + j, ld_q, TP,
                                  tb.nq, mx, wv);
    }
    if (SLICE == 4) {
#pragma unroll
      for (int q = 0; q < 4; ++q) s_mx[SLICE > 0 ? warp : 0][SLICE > 0 ? (pg / 32) * 128 + q * 32 + lane : 0] = mx[q];
    } else if (SLICE == 1) {
      s_mx[SLICE > 0 ? warp : 0][SLICE > 0 ? j : 0] = mx[0];
    }
  }
  const int kt_true = tb.ktrue[t], kt = tb.kt[t];
  const int npad = (kt - kt_true) * TP;
  for (int idx = threadIdx.x; idx < tb.nq * npad && blockIdx.y == 0; idx += kAoThreads) {
    const int q = idx / npad, r = idx % npad;
    A[q * ld_q + (int64_t)kt_true * TP + r] = 0.0;
  }
  if (SLICE > 0) {
    __syncthreads();  // row maxima of every warp are in shared memory
    const int rows = split_tile_rows(TP, SLICE);
    for (int r = threadIdx.x; r < rows; r += kAoThreads) {
      unsigned m = 0u;
#pragma unroll
      for (int w = 0; w < kAoThreads / 32; ++w) m = max(m, s_mx[SLICE > 0 ? w : 0][SLICE > 0 ? r : 0]);
      // |x| = 1.f 2^(E - 1023) < 2^(E - 1022) for the biased exponent E of the
      // largest |x| (frexp's exponent); a row of zeros gets 0
      const int E = (int)(m >> 20);
      const int e = m == 0u ? 0 : E - 1022;
      eexp[(int64_t)t * rows + r] = e < kMinScaleExponent ? kMinScaleExponent : e;
    }
  }
}

// Digit planes of the tile rows (ctc_split.cuh) with the exponents found by
// ao_tile_kernel, columns in the order of the tile's quads of AOs (TileBatch::ksrc;
// places without a compact AO get zeros).  One block per tile, the tiles taken in the chunk's order
// (largest compact K first) when one is given.  Work items are (32-row
// group, 32-column chunk); the block's warps take them in turn: a warp reads
// one 256-byte line per column (32 consecutive rows = points of one
// quantity), all 32 lines before any conversion so that they are in flight
// together, and each lane writes 32 bytes per plane of its own row.
constexpr int kSliceThreads = 256;

__global__ void __launch_bounds__(kSliceThreads, 2)
    slice_rows_kernel(TileBatch tb, int nqa, const int32_t* __restrict__ eexp,
                      int8_t* __restrict__ planes, const int32_t* __restrict__ order) {
  const int t = order ? order[blockIdx.x] : blockIdx.x;
  const int kp = tb.kp[t];
  const int TP = tb.TP;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t ld_q = (int64_t)TP * tb.Kcap;
  const double* A = tb.ao + (int64_t)t * tb.nq * ld_q;
  const int32_t* ksrc = tb.ksrc + (int64_t)t * tb.Kpcap;
  const int rows = split_tile_rows(TP, nqa);
  int8_t* P = planes + (int64_t)t * kSplitPlanesA * rows * tb.Kpcap;
  const int nitem = (rows / 32) * (kp / 32);  // warp-sized items
  for (int it = warp; it < nitem; it += kSliceThreads / 32) {
    const int rg = it % (rows / 32), c = it / (rows / 32);
    const int r = rg * 32 + lane;             // tile row
    const int blk = r / kSplitRows;           // 128-row block of the row
    const int q = nqa == 4 ? rg % 4 : 0;      // quantity
    const int p = nqa == 4 ? blk * 32 + lane : r;  // point
    const double f = split_row_factor(eexp[(int64_t)t * rows + r], kFixedBitsA);
    const double* col = A + q * ld_q + p;
    const int src = ksrc[c * 32 + lane];
    const unsigned used = __ballot_sync(0xffffffffu, src >= 0);
    double v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __ldg(col + (int64_t)max(__shfl_sync(0xffffffffu, src, i), 0) * TP);
    write_row_digits32([&](int i) { return (used >> i) & 1u ? v[i] : 0.0; }, f,
                       P + (int64_t)blk * kSplitPlanesA * kSplitRows * tb.Kpcap, r % kSplitRows,
                       tb.Kpcap, c * 32);
  }
}

}  // namespace

int launch_ao_tiles(const ctc_molecule* mol, const TileBatch& tb, int deriv, cudaStream_t st) {
  if (tb.C <= 0) return CTC_OK;
  const auto* sg = mol->d_segs;
  const double *al = mol->d_alpha, *co = mol->d_coef;
  // few tiles: their segments on more CTAs, up to twelve for every SM, of which
  // three or more run at a time, so that the last round is a small part (values of
  // 62 segments at 200 points, seven tiles: 18 us on one CTA each, 5.5 on eight)
  int nsm = 0;
  if (int rc = device_sm_count(&nsm); rc != CTC_OK) return rc;
  const dim3 grid((unsigned)tb.C, (unsigned)std::max(1, std::min(8, (12 * nsm + tb.C - 1) / tb.C)));
  switch (deriv) {
    case 0: ao_tile_kernel<0, 0><<<grid, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, nullptr, nullptr, nullptr, nullptr); break;
    case 1: ao_tile_kernel<1, 0><<<grid, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, nullptr, nullptr, nullptr, nullptr); break;
    default: ao_tile_kernel<2, 0><<<grid, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, nullptr, nullptr, nullptr, nullptr);
  }
  CTC_CUDA_TRY(cudaGetLastError());
  return CTC_OK;
}

int launch_ao_tiles_weighted(const ctc_molecule* mol, const TileBatch& tb, const double* v_rho,
                             const double* v_grad, cudaStream_t st) {
  if (tb.C <= 0) return CTC_OK;
  const auto* sg = mol->d_segs;
  const double *al = mol->d_alpha, *co = mol->d_coef;
  if (tb.nq == 11) ao_tile_kernel<2, -1><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, nullptr, nullptr, v_rho, v_grad);
  else if (tb.nq == 2) ao_tile_kernel<1, -2><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, nullptr, nullptr, v_rho, v_grad);
  else return fail(CTC_ERR_INVALID, "weighted AO tiles: unsupported quantity count");
  CTC_CUDA_TRY(cudaGetLastError());
  return CTC_OK;
}

int launch_ao_tiles_sliced(const ctc_molecule* mol, const TileBatch& tb, int deriv, int nqa,
                           int8_t* planes, int32_t* eexp, const int32_t* order, cudaStream_t st) {
  if (tb.C <= 0) return CTC_OK;
  // (second derivatives come with four rows per point: plan_local)
  if (!(nqa == 4 && tb.TP == 32 && deriv >= 1) && !(nqa == 1 && tb.TP == 128 && deriv <= 1))
    return fail(CTC_ERR_INVALID, "sliced AO tiles: unsupported row layout");
  if (planes == nullptr || eexp == nullptr)
    return fail(CTC_ERR_INVALID, "sliced AO tiles: null workspace");
  const auto* sg = mol->d_segs;
  const double *al = mol->d_alpha, *co = mol->d_coef;
  if (nqa == 4) {
    if (deriv == 1) ao_tile_kernel<1, 4><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, eexp, order, nullptr, nullptr);
    else ao_tile_kernel<2, 4><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, eexp, order, nullptr, nullptr);
  } else {
    if (deriv == 0) ao_tile_kernel<0, 1><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, eexp, order, nullptr, nullptr);
    else ao_tile_kernel<1, 1><<<tb.C, kAoThreads, 0, st>>>(sg, mol->nseg, al, co, tb, eexp, order, nullptr, nullptr);
  }
  CTC_CUDA_TRY(cudaGetLastError());
  slice_rows_kernel<<<tb.C, kSliceThreads, 0, st>>>(tb, nqa, eexp, planes, order);
  CTC_CUDA_TRY(cudaGetLastError());
  return CTC_OK;
}

// Public layout (nq, n, M).
template <int DERIV>
static int launch_ao_pub(const ctc_molecule* mol, const double* pts, int64_t n, double* out, cudaStream_t st) {
  if (int rc = ensure_smem_attr((const void*)ao_public_kernel<DERIV>, (int)ao_pub_smem(DERIV)); rc != CTC_OK) return rc;
  int nsm = 0;
  if (int rc = device_sm_count(&nsm); rc != CTC_OK) return rc;
  // few points: the narrower chunks, on more CTAs (values at one or two points of 60
  // to 200 atoms: 12.2 us, 10.4 with them)
  const int64_t groups = (n + 31) / 32;
  const int k = DERIV == 2 || groups * mol->n_aochunk[0] < nsm ? 1 : 0;
  const int64_t items = groups * mol->n_aochunk[k];
  ao_public_kernel<DERIV><<<(unsigned)std::min<int64_t>(items, INT32_MAX), kAoPubThreads, ao_pub_smem(DERIV), st>>>(
      mol->d_segs, mol->d_order, mol->d_aochunk[k], mol->n_aochunk[k], mol->nseg, mol->d_alpha, mol->d_coef, pts, n,
      mol->M, out);
  CTC_CUDA_TRY(cudaGetLastError());
  return CTC_OK;
}
int launch_ao_public(const ctc_molecule* mol, const double* pts, int64_t n, int deriv, double* out, cudaStream_t st) {
  if (n <= 0) return CTC_OK;
  return deriv == 0 ? launch_ao_pub<0>(mol, pts, n, out, st)
       : deriv == 1 ? launch_ao_pub<1>(mol, pts, n, out, st) : launch_ao_pub<2>(mol, pts, n, out, st);
}

}  // namespace ctc
