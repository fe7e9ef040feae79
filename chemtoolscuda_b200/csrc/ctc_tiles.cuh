// ctc_tiles.cuh -- the screened point-tile pipeline shared by the local
// descriptors (ctc_local.cu) and the adjoint (ctc_adjoint.cu).
//
// Points are grouped into spatially compact tiles (3-D blocks of a cubic grid,
// or sort-tile-recursive runs of explicit points); every tile lists the segments whose
// screening sphere (every AO value and derivative below 1e-18 outside it)
// meets the tile's bounding sphere, and works on that compacted AO set only.
// Per chunk of tiles: tile points -> screen -> AO block (compact) -> a
// contraction kernel supplied by the caller.
#pragma once

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <functional>

#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include "ctc_chunk.h"
#include "ctc_internal.h"
#include "ctc_finalize.cuh"

namespace ctc {

namespace {

__device__ __forceinline__ int ncomp_of_type_dev(int type) {
  switch (type) {
    case 0: return 1;
    case 1: return 3;
    case 2: return 6;
    case 3: return 5;
    case 4: return 10;
    case 5: return 7;
    case 6: return 15;
    default: return 9;
  }
}

// ------------------------------------------------------------------ tiles
constexpr int kTileThreads = 256;
constexpr int kSortCap = 2048;  // segment lists up to this length are ordered by type

__device__ __forceinline__ uint32_t spread10(uint32_t v) {
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

// Morton key of each point, `bits` bits per axis (the single-sort order of small
// calls and of the fixed-scratch entry point, ctc_noalloc.cu; morton_axis_bits).
// A point with a non-finite coordinate gets the last key, so the sort puts such
// points behind the others (but for points in the box's last cell).
__global__ void morton_kernel(const double* __restrict__ pts, int64_t n, double lox, double loy,
                              double loz, double inv_cell, int bits, uint32_t* keys, int32_t* vals) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double last = (double)((1 << bits) - 1);
  auto q = [&](double v, double lo) {
    double c = (v - lo) * inv_cell;
    c = c < 0.0 ? 0.0 : (c > last ? last : c);
    return (uint32_t)c;
  };
  const double x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
  keys[i] = finite_point(pts + 3 * i)
                ? spread10(q(x, lox)) | (spread10(q(y, loy)) << 1) | (spread10(q(z, loz)) << 2)
                : (1u << 3 * bits) - 1u;
  vals[i] = (int32_t)i;
}

// Corner and edge of the cube the Morton keys cover: the molecule's box padded
// by 12 bohr.
inline void morton_box(const ctc_molecule* mol, double* lo, double* ext) {
  *ext = 24.0;
  for (int d = 0; d < 3; ++d) {
    double a = mol->natom ? 1e300 : -1.0, b = mol->natom ? -1e300 : 1.0;
    for (int i = 0; i < mol->natom; ++i) {
      a = std::min(a, mol->atom_xyz[3 * i + d]);
      b = std::max(b, mol->atom_xyz[3 * i + d]);
    }
    lo[d] = a - 12.0;
    *ext = std::max(*ext, b - a + 24.0);
  }
}

// Sort-tile-recursive packing of explicit points (Leutenegger, Lopez and
// Edgington, "STR: a simple and efficient algorithm for R-tree packing",
// ICDE 1997): sort by x and cut into sx slabs of whole tiles; sort each slab
// by y and cut it into sy columns; sort each column by z; tiles are then runs
// of TP consecutive points.  sx and sy follow the points' bounding box
// (edge a = (volume / P)^(1/3) for P tiles, sx ~ Lx / a, sy ~ Ly / a), so the
// tiles are close to cubes also for slab-shaped point sets such as a
// few-plane slice of a grid.  The box and the cut counts are formed on the
// device (every thread of the key kernel derives the same counts), so the
// host never waits.  Three radix sorts of 64-bit keys (group id << 32 |
// coordinate key); a point with a non-finite coordinate gets the largest
// coordinate key on every axis, so it sorts after every finite point and
// shares tiles only with its kind (and at most one tile's finite points).
__device__ __forceinline__ unsigned long long ordered_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double ordered_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}
// box[0..2] = ordered keys of the minima, box[3..5] of the maxima (start at
// all-ones and zero); finite points only
__global__ void point_box_kernel(const double* __restrict__ pts, int64_t n, unsigned long long* box) {
  unsigned long long mn[3] = {~0ull, ~0ull, ~0ull}, mx[3] = {0ull, 0ull, 0ull};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* x = pts + 3 * i;
    if (!finite_point(x)) continue;
    for (int d = 0; d < 3; ++d) {
      const unsigned long long k = ordered_key(x[d]);
      mn[d] = k < mn[d] ? k : mn[d];
      mx[d] = k > mx[d] ? k : mx[d];
    }
  }
  for (int d = 0; d < 3; ++d)
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long a = __shfl_xor_sync(0xffffffffu, mn[d], o), b = __shfl_xor_sync(0xffffffffu, mx[d], o);
      mn[d] = a < mn[d] ? a : mn[d];
      mx[d] = b > mx[d] ? b : mx[d];
    }
  if ((threadIdx.x & 31) == 0)
    for (int d = 0; d < 3; ++d) {
      atomicMin(&box[d], mn[d]);
      atomicMax(&box[3 + d], mx[d]);
    }
}
struct StrShape {
  double lo[3], scale[3];  // coordinate key = (x - lo) * scale, clamped
  int64_t Sx, Scol, c;     // points per slab, points per column, columns per slab
};
__device__ StrShape str_shape(const unsigned long long* __restrict__ box, int64_t P, int TP) {
  StrShape sh;
  double L[3];
  bool any = box[0] <= box[3];
  double Lmax = 0.0;
  for (int d = 0; d < 3; ++d) {
    sh.lo[d] = any ? ordered_value(box[d]) : 0.0;
    L[d] = any ? ordered_value(box[3 + d]) - sh.lo[d] : 0.0;
    Lmax = fmax(Lmax, L[d]);
  }
  if (!(Lmax > 0.0)) Lmax = 1.0;
  for (int d = 0; d < 3; ++d) {
    L[d] = fmax(L[d], 1e-3 * Lmax);  // planar or linear sets: keep the volume positive
    sh.scale[d] = 4294967040.0 / L[d];
  }
  const double a = cbrt(L[0] * L[1] * L[2] / (double)P);
  int64_t sx = (int64_t)fmin(fmax(rint(L[0] / a), 1.0), (double)P);
  const int64_t Tsl = (P + sx - 1) / sx;
  int64_t sy = (int64_t)fmin(fmax(rint(L[1] / a), 1.0), (double)Tsl);
  const int64_t Tcol = (Tsl + sy - 1) / sy;
  sy = (Tsl + Tcol - 1) / Tcol;
  sh.Sx = Tsl * TP;
  sh.Scol = Tcol * TP;
  sh.c = sy;
  return sh;
}
__device__ __forceinline__ uint32_t axis_key(double v, double lo, double scale) {
  double c = (v - lo) * scale;
  c = c < 0.0 ? 0.0 : (c > 4294967040.0 ? 4294967040.0 : c);
  return (uint32_t)c;
}
__global__ void str_key_kernel(const double* __restrict__ pts, const int32_t* __restrict__ perm,
                               int64_t n, int pass, const unsigned long long* __restrict__ box,
                               int64_t P, int TP, uint64_t* __restrict__ keys, int32_t* __restrict__ vals) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const StrShape sh = str_shape(box, P, TP);
  const int64_t p = perm ? perm[i] : i;
  const double* x = pts + 3 * p;
  uint64_t g = 0;
  if (pass == 1) g = (uint64_t)(i / sh.Sx);
  if (pass == 2) g = (uint64_t)(i / sh.Sx) * (uint64_t)sh.c + (uint64_t)((i % sh.Sx) / sh.Scol);
  const uint32_t k = finite_point(x) ? axis_key(x[pass], sh.lo[pass], sh.scale[pass]) : 0xFFFFFFFFu;
  keys[i] = (g << 32) | k;
  vals[i] = (int32_t)p;
}

// Tiles of TP consecutive sorted points; padding slots repeat the tile's first point.
__global__ void tile_gather_kernel(const double* __restrict__ pts, const int32_t* __restrict__ perm,
                                   int64_t n, int64_t t0, TileBatch tb) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)tb.C * tb.TP) return;
  const int64_t t = gid / tb.TP;
  const int j = (int)(gid % tb.TP);
  const int64_t g = (t0 + t) * tb.TP + j;
  const bool v = g < n;
  const int64_t i = v ? g : (t0 + t) * tb.TP;
  const int64_t p = perm ? perm[i] : i;
  tb.xyz[3 * gid] = pts[3 * p];
  tb.xyz[3 * gid + 1] = pts[3 * p + 1];
  tb.xyz[3 * gid + 2] = pts[3 * p + 2];
  tb.out[gid] = v ? p : -1;
}

// Cubic grid: tile = TX x TY x TZ block of grid points (z fastest).
__global__ void tile_cubic_kernel(PointSrc src, int nx, int TX, int TY, int TZ, int nby, int nbz,
                                  int64_t t0, TileBatch tb) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)tb.C * tb.TP) return;
  const int64_t t = t0 + gid / tb.TP;
  const int j = (int)(gid % tb.TP);
  const int64_t bz = t % nbz, by = (t / nbz) % nby, bx = t / ((int64_t)nbz * nby);
  const int iz = j % TZ, iy = (j / TZ) % TY, ix = j / (TZ * TY);
  int64_t i = bx * TX + ix, k = by * TY + iy, l = bz * TZ + iz;
  const bool v = i < nx && k < src.ny && l < src.nz;
  if (!v) { i = bx * TX; k = by * TY; l = bz * TZ; }
  const double fi = (double)i, fj = (double)k, fk = (double)l;
  tb.xyz[3 * gid] = src.o[0] + fi * src.ax[0] + fj * src.ax[3] + fk * src.ax[6];
  tb.xyz[3 * gid + 1] = src.o[1] + fi * src.ax[1] + fj * src.ax[4] + fk * src.ax[7];
  tb.xyz[3 * gid + 2] = src.o[2] + fi * src.ax[2] + fj * src.ax[5] + fk * src.ax[8];
  tb.out[gid] = v ? (i * src.ny + k) * (int64_t)src.nz + l : -1;
}

// Bounding sphere of one tile's points, computed by a whole block of
// kTileThreads threads: centre = mean of the finite points (padding repeats a
// real point; a point with a non-finite coordinate gets NaN outputs and must
// not move the sphere of its tile mates), radius = largest distance from it,
// widened by a relative 1e-12 plus 1e-9 bohr; -1e300 when no point is finite.
// The screening kernel and the capacity pre-pass both use this code, so they
// see the same sphere to the last bit.
__device__ void tile_sphere(const double* __restrict__ xyz, int TP, double* sctr, double* srad) {
  __shared__ double red[3][kTileThreads / 32];
  __shared__ int s_nfin;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_nfin = 0;
  __syncthreads();
  double c[3] = {0, 0, 0};
  int nfin = 0;
  for (int j = threadIdx.x; j < TP; j += kTileThreads)
    if (finite_point(xyz + 3 * j)) {
      ++nfin;
      for (int d = 0; d < 3; ++d) c[d] += xyz[3 * j + d];
    }
  for (int o = 16; o > 0; o >>= 1) nfin += __shfl_xor_sync(0xffffffffu, nfin, o);
  if (lane == 0 && nfin) atomicAdd(&s_nfin, nfin);
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) c[d] += __shfl_xor_sync(0xffffffffu, c[d], o);
    if (lane == 0) red[d][warp] = c[d];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double acc = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) acc += red[threadIdx.x][w];
    sctr[threadIdx.x] = s_nfin ? acc / s_nfin : 0.0;
  }
  __syncthreads();
  double r2 = 0.0;
  for (int j = threadIdx.x; j < TP; j += kTileThreads) {
    if (!finite_point(xyz + 3 * j)) continue;
    const double dx = xyz[3 * j] - sctr[0], dy = xyz[3 * j + 1] - sctr[1], dz = xyz[3 * j + 2] - sctr[2];
    r2 = fmax(r2, dx * dx + dy * dy + dz * dz);
  }
  for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if (lane == 0) red[0][warp] = r2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) m = fmax(m, red[0][w]);
    // a tile without a finite point keeps no segment
    *srad = s_nfin ? sqrt(m) * (1.0 + 1e-12) + 1e-9 : -1e300;
  }
  __syncthreads();
}

// Is segment sg significant on the tile sphere (ctr, rad)?  Every AO value and
// derivative of the segment is below 1e-18 beyond sqrt(rcut2) of its centre.
__device__ __forceinline__ bool seg_significant(const DevSeg& sg, const double* ctr, double rad) {
  const double dx = sg.cx - ctr[0], dy = sg.cy - ctr[1], dz = sg.cz - ctr[2];
  const double d = sqrt(dx * dx + dy * dy + dz * dz);
  return d <= sqrt(sg.rcut2) + rad;
}

// Status code of a tile whose compact AO set exceeds the batch's capacity
// (cannot happen when the capacity comes from tile_capacity_kernel).
constexpr int32_t kStatusCapacity = 0x7201;

// Capacity pre-pass: the largest padded compact AO count of a batch of tiles
// (atomicMax into kmax[0]) and a bound of the AOs in their quads (kmax[1]: each
// run of consecutive AOs adds at most three at either end).  One block per tile.
__global__ void __launch_bounds__(kTileThreads)
    tile_capacity_kernel(const DevSeg* __restrict__ segs, int nseg, TileBatch tb, int* kmax) {
  __shared__ double sctr[3], srad;
  __shared__ int part[2][kTileThreads / 32];
  const int t = blockIdx.x;
  tile_sphere(tb.xyz + (int64_t)t * tb.TP * 3, tb.TP, sctr, &srad);
  int cnt = 0, runs = 0;
  for (int s = threadIdx.x; s < nseg; s += kTileThreads) {
    const DevSeg sg = segs[s];
    if (seg_significant(sg, sctr, srad)) {
      cnt += ncomp_of_type_dev(sg.type);
      runs += s == 0 || !seg_significant(segs[s - 1], sctr, srad);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    runs += __shfl_xor_sync(0xffffffffu, runs, o);
  }
  if ((threadIdx.x & 31) == 0) {
    part[0][threadIdx.x >> 5] = cnt;
    part[1][threadIdx.x >> 5] = runs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0, nr = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) {
      tot += part[0][w];
      nr += part[1][w];
    }
    atomicMax(kmax, (tot + kKtAlign - 1) / kKtAlign * kKtAlign);
    atomicMax(kmax + 1, (tot + 6 * nr + kKtAlign - 1) / kKtAlign * kKtAlign);
  }
}

// One CTA per tile: bounding sphere of the tile's points, then the ordered
// list of segments whose screening sphere meets it.
__global__ void __launch_bounds__(kTileThreads)
    screen_kernel(const DevSeg* __restrict__ segs, int nseg, TileBatch tb, int rows,
                  double* __restrict__ stats, int32_t* __restrict__ status) {
  using Scan = cub::BlockScan<int, kTileThreads>;
  __shared__ typename Scan::TempStorage scan_tmp;
  __shared__ int s_sl[kSortCap], s_k0[kSortCap], s_cnt[8];
  __shared__ double sctr[3], srad;
  __shared__ int base_s, base_k;
  __shared__ int s_over_s, s_over_k;  // first segment beyond the capacity
  const int t = blockIdx.x, TP = tb.TP;
  tile_sphere(tb.xyz + (int64_t)t * TP * 3, TP, sctr, &srad);
  if (threadIdx.x == 0) {
    base_s = 0;
    base_k = 0;
    s_over_s = INT_MAX;
    s_over_k = INT_MAX;
  }
  __syncthreads();
  const double rad = srad;
  int32_t* sl = tb.segs + (int64_t)t * nseg;
  int32_t* k0 = tb.k0 + (int64_t)t * nseg;
  int32_t* am = tb.aomap + (int64_t)t * tb.Kcap;
  for (int s0 = 0; s0 < nseg; s0 += kTileThreads) {
    const int s = s0 + threadIdx.x;
    int sig = 0, nc = 0;
    DevSeg sg;
    if (s < nseg) {
      sg = segs[s];
      if (seg_significant(sg, sctr, rad)) {
        sig = 1;
        nc = ncomp_of_type_dev(sg.type);
      }
    }
    // pack (segment count, AO count) into one int: both sums stay below 2^16
    int packed, ptot;
    Scan(scan_tmp).ExclusiveSum((sig << 16) | nc, packed, ptot);
    const int2 pos = make_int2(packed >> 16, packed & 0xffff);
    const int2 tot = make_int2(ptot >> 16, ptot & 0xffff);
    if (sig) {
      const int ks = base_k + pos.y;
      sl[base_s + pos.x] = s;
      k0[base_s + pos.x] = ks;
      if (ks + nc <= tb.Kcap) {
        for (int q = 0; q < nc; ++q) am[ks + q] = sg.ao0 + q;
      } else {
        // never with a capacity from the pre-pass or Kcap = Mpad: the tile is
        // cut at this segment and the call reports kStatusCapacity
        atomicMin(&s_over_s, base_s + pos.x);
        atomicMin(&s_over_k, ks);
        atomicExch(status, kStatusCapacity);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      base_s += tot.x;
      base_k += tot.y;
    }
    __syncthreads();
  }
  // Visit order for the AO kernel: the significant segments grouped by type
  // (counting sort; compact positions k0 keep the AO order), so that the
  // warps of a CTA run one type's evaluation code at a time instead of
  // alternating between the types' large unrolled bodies.
  const int ns = min(base_s, s_over_s);
  if (ns <= kSortCap) {
    if (threadIdx.x < 8) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < ns; i += kTileThreads) {
      const int sg = sl[i];
      s_sl[i] = sg;
      s_k0[i] = k0[i];
      atomicAdd(&s_cnt[segs[sg].type & 7], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int acc = 0;
      for (int ty = 0; ty < 8; ++ty) {
        const int c = s_cnt[ty];
        s_cnt[ty] = acc;
        acc += c;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ns; i += kTileThreads) {
      const int sg = s_sl[i];
      const int pos = atomicAdd(&s_cnt[segs[sg].type & 7], 1);
      sl[pos] = sg;
      k0[pos] = s_k0[i];
    }
  }
  const int kt_true = min(base_k, s_over_k);
  const int kt = min((kt_true + kKtAlign - 1) / kKtAlign * kKtAlign, tb.Kcap);
  for (int k = kt_true + threadIdx.x; k < kt; k += kTileThreads) am[k] = -1;
  if (tb.Kpcap > 0) {
    // quads of the compact AOs (ascending, as the AOs are) and the compact index
    // of every place in them
    int32_t* kq = tb.kq + (int64_t)t * (tb.Kpcap / 4);
    int4* ks = reinterpret_cast<int4*>(tb.ksrc + (int64_t)t * tb.Kpcap);
    const int qcap = tb.Kpcap / 4;
    __syncthreads();
    int nq = 0;
    for (int k0 = 0; k0 < kt_true; k0 += kTileThreads) {
      const int k = k0 + threadIdx.x;
      const int ao = k < kt_true ? am[k] : 0;
      const int first = k < kt_true && (k == 0 || (am[k - 1] >> 2) != (ao >> 2));
      int before, total;
      Scan(scan_tmp).ExclusiveSum(first, before, total);
      const int q = nq + before + first - 1;
      if (first && q < qcap) {
        kq[q] = ao >> 2;
        ks[q] = make_int4(-1, -1, -1, -1);
      }
      __syncthreads();
      if (k < kt_true) {
        if (q < qcap) tb.ksrc[(int64_t)t * tb.Kpcap + 4 * q + (ao & 3)] = k;
        else atomicExch(status, kStatusCapacity);  // never, as above
      }
      nq += total;
    }
    nq = min(nq, qcap);
    const int kp = (4 * nq + kKtAlign - 1) / kKtAlign * kKtAlign;
    for (int q = nq + threadIdx.x; q < kp / 4; q += kTileThreads) {
      kq[q] = 0;
      ks[q] = make_int4(-1, -1, -1, -1);
    }
    if (threadIdx.x == 0) tb.kp[t] = kp;
  }
  if (threadIdx.x == 0) {
    tb.nsig[t] = ns;
    tb.ktrue[t] = kt_true;
    tb.kt[t] = kt;
    int npts = 0;
    for (int j = 0; j < TP; ++j) npts += tb.out[(int64_t)t * TP + j] >= 0;
    atomicAdd(&stats[0], 1.0);
    atomicAdd(&stats[1], (double)npts);
    atomicAdd(&stats[2], (double)kt_true);
    atomicAdd(&stats[3], (double)rows * (double)kt * (double)kt);
  }
}

// The chunk's tiles, largest compact set first (counting sort by kt / 64; the
// order within a bin is free), the chunk's tile counter set to zero, and the
// work items per tile of the tensor-core contraction.  The FP64 contraction and
// the tensor-core path's AO kernel take the tiles in this order, so the last
// tiles of a launch are the cheapest.  One block: ~4 us at 2 000 tiles, where a
// radix sort of the counts took ~8 us and two launches.
//
// A tile's digit planes (640 bytes per function) are read once for every 64
// functions and D by every tile, so the contraction wants the planes of the
// tiles in flight and D in L2: with `parts` items per tile the SMs work on 1 /
// parts as many tiles.  parts is the smallest power of two for which the planes
// and D (8 M^2 bytes, or what the tiles use of it) stay below kL2Bytes, and at
// least what gives every SM four items.  (One item per tile: contraction of the
// 530 000-point cube of 200 atoms 67.7 ms, with parts 56.6; 640-atom sparse cube
// 153 and 136; 300 000 host points 16.2 and 14.5.)
constexpr int kOrderThreads = 1024;
constexpr double kL2Bytes = 96e6;
__global__ void __launch_bounds__(kOrderThreads) tile_order_kernel(TileBatch tb, int sms, double d_bytes) {
  using Scan = cub::BlockScan<int, kOrderThreads>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ int s_bin[kOrderThreads];
  __shared__ unsigned long long s_kt;
  s_bin[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    *tb.counter = 0;
    s_kt = 0;
  }
  __syncthreads();
  auto bin = [&](int t) { return kOrderThreads - 1 - min(tb.kt[t] / kKtAlign, kOrderThreads - 1); };
  unsigned long long kt = 0;
  for (int t = threadIdx.x; t < tb.C; t += kOrderThreads) {
    atomicAdd(&s_bin[bin(t)], 1);
    kt += tb.kt[t];
  }
  for (int o = 16; o > 0; o >>= 1) kt += __shfl_xor_sync(0xffffffffu, kt, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_kt, kt);
  __syncthreads();
  if (threadIdx.x == 0) {
    const double mean = (double)s_kt / tb.C, d = fmin(d_bytes, 0.6 * kL2Bytes);
    int parts = 1;
    while (parts < kMaxParts && ((double)min(sms, tb.C * parts) / parts * 640.0 * mean + d > kL2Bytes ||
                                 (int64_t)tb.C * parts < 4 * sms))
      parts *= 2;
    *tb.parts = parts;
  }
  int first;
  Scan(tmp).ExclusiveSum(s_bin[threadIdx.x], first);
  __syncthreads();
  s_bin[threadIdx.x] = first;
  __syncthreads();
  for (int t = threadIdx.x; t < tb.C; t += kOrderThreads) tb.order[atomicAdd(&s_bin[bin(t)], 1)] = t;
}

// ------------------------------------------------------------------ chunk scratch

struct Carve {
  char* p;
  size_t off = 0;
  template <class T>
  T* take(size_t count) {
    off = (off + 255) / 256 * 256;
    T* r = (T*)(p + off);
    off += sizeof(T) * count;
    return r;
  }
};

size_t tile_bytes(const ctc_molecule* mol, int C, int TP, int Kcap_, int Kpcap = 0) {
  const size_t Kcap = Kcap_;
  size_t b = 0;
  auto add = [&](size_t x) { b = (b + 255) / 256 * 256 + x; };
  add(sizeof(double) * C * TP * 3);
  add(sizeof(int64_t) * C * TP);
  add(sizeof(int32_t) * C);
  add(sizeof(int32_t) * C);
  add(sizeof(int32_t) * C);
  add(sizeof(int32_t) * (size_t)C * mol->nseg);
  add(sizeof(int32_t) * (size_t)C * mol->nseg);
  add(sizeof(int32_t) * (size_t)C * Kcap);
  add(sizeof(int32_t) * C);
  add(2 * sizeof(int32_t));
  add(sizeof(int32_t) * C);
  add(sizeof(int32_t) * (size_t)C * (Kpcap / 4));
  add(sizeof(int32_t) * (size_t)C * Kpcap);
  return b + 256;
}


// Tile builder + chunk loop.  For every chunk: tile points, screen, AO block
// (derivative order deriv, nq quantities; ao_launch replaces the plain AO
// kernel launch when given), then compute(tb).  quads: the tensor-core
// contraction's K side is formed too.
inline int run_tiles(ctc_molecule* mol, const PointSrc& src, int64_t n, int TP, int nq, int deriv,
                     cudaStream_t st, const std::function<int(const TileBatch&)>& compute,
                     const std::function<int(const TileBatch&)>* ao_launch = nullptr,
                     int rows = 128, bool quads = false) {
  if (n <= 0) return CTC_OK;  // (no zero-sized grids below)
  // cubic-grid tiles: blocks of 2x4x4 or 4x4x8 grid points
  int TX = 2, TY = 4, TZ = 4;
  if (TP == 128) { TX = 4; TY = 4; TZ = 8; }
  int64_t ntiles, nbx = 0, nby = 0, nbz = 0;
  int nx = 0;
  if (src.cubic) {
    nx = (int)(n / ((int64_t)src.ny * src.nz));
    nbx = (nx + TX - 1) / TX;
    nby = (src.ny + TY - 1) / TY;
    nbz = (src.nz + TZ - 1) / TZ;
    ntiles = nbx * nby * nbz;
  } else {
    ntiles = (n + TP - 1) / TP;
  }
  int rc;
  // explicit points: sort-tile-recursive order over the points' own box for
  // calls of kStrMinPoints points or more; below that, one sort of Morton keys
  // over the molecule's box padded by 12 bohr (three sorts cost ~0.4 ms, as much
  // as a whole 1e5-point density call of a small molecule, while the tiles' shape
  // matters little there), or none (sort_points)
  constexpr int64_t kStrMinPoints = (int64_t)1 << 18;
  int32_t* perm = nullptr;
  double lo[3], ext = 0;
  if (!src.cubic) morton_box(mol, lo, &ext);
  if (!src.cubic && sort_points(n, mol->Mpad, ext)) {
    const bool str = n >= kStrMinPoints;
    const int bits = morton_axis_bits(ext);
    size_t tmp_bytes = 0, tmp32 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                    (int32_t*)nullptr, (int32_t*)nullptr, (int)n, 0, 64, st);
    cub::DeviceRadixSort::SortPairs(nullptr, tmp32, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                    (int32_t*)nullptr, (int32_t*)nullptr, (int)n, 0, 3 * bits, st);
    tmp_bytes = std::max(tmp_bytes, tmp32);
    const size_t need = 2 * sizeof(uint64_t) * (size_t)n + 2 * sizeof(int32_t) * (size_t)n + tmp_bytes + 4096;
    if ((rc = mol->ws_part.ensure(need, st)) != CTC_OK) return rc;
    Carve cv{(char*)mol->ws_part.p};
    unsigned long long* box = cv.take<unsigned long long>(6);
    uint64_t* k_in = cv.take<uint64_t>(n);
    uint64_t* k_out = cv.take<uint64_t>(n);
    int32_t* v_in = cv.take<int32_t>(n);
    perm = cv.take<int32_t>(n);
    void* tmp = cv.take<char>(tmp_bytes);
    if (str) {
      CTC_CUDA_TRY(cudaMemsetAsync(box, 0xFF, 3 * sizeof(unsigned long long), st));
      CTC_CUDA_TRY(cudaMemsetAsync(box + 3, 0, 3 * sizeof(unsigned long long), st));
      point_box_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 4 * 148), 256, 0, st>>>(src.pts, n, box);
      CTC_CUDA_TRY(cudaGetLastError());
      // group ids of passes 2 and 3 are below sx * sy <= sx * ceil(P / sx) < P + sx <= 2 P
      const int gbits = 64 - __builtin_clzll((unsigned long long)(2 * ntiles));
      const unsigned g = (unsigned)((n + 255) / 256);
      for (int pass = 0; pass < 3; ++pass) {
        str_key_kernel<<<g, 256, 0, st>>>(src.pts, pass ? perm : nullptr, n, pass, box, ntiles, TP, k_in, v_in);
        CTC_CUDA_TRY(cudaGetLastError());
        CTC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k_in, k_out, v_in, perm, (int)n, 0,
                                                     32 + (pass ? gbits : 0), st));
      }
      mol->host_launches += 7;
    } else {
      uint32_t* k32_in = (uint32_t*)k_in;
      uint32_t* k32_out = (uint32_t*)k_out;
      morton_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(src.pts, n, lo[0], lo[1], lo[2], (1 << bits) / ext,
                                                                  bits, k32_in, v_in);
      CTC_CUDA_TRY(cudaGetLastError());
      CTC_CUDA_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k32_in, k32_out, v_in, perm, (int)n, 0,
                                                   3 * bits, st));
      mol->host_launches += 2;
    }
  }
  // tile points of tiles [t0, t0 + tb.C)
  auto tile_points = [&](const TileBatch& tb, int64_t t0) -> int {
    const int64_t npts = (int64_t)tb.C * TP;
    const unsigned g = (unsigned)((npts + 255) / 256);
    if (src.cubic)
      tile_cubic_kernel<<<g, 256, 0, st>>>(src, nx, TX, TY, TZ, (int)nby, (int)nbz, t0, tb);
    else
      tile_gather_kernel<<<g, 256, 0, st>>>(src.pts, perm, n, t0, tb);
    CTC_CUDA_TRY(cudaGetLastError());
    return CTC_OK;
  };
  // chunk of tiles: AO block (nq x TP x Kcap doubles per tile) within
  // min(12 GiB, a quarter of the free device memory) (CTC_CHUNK_BYTES
  // overrides), at least one tile per SM (ctc_chunk.h).  Larger chunks
  // amortise the per-chunk launches and tails: on the 215^3 benchmark cube
  // 6 GiB gave 20.95 M points/s, 12 GiB 21.46 M, 24 GiB 21.60 M.
  int nsm = 148;
  if ((rc = device_sm_count(&nsm)) != CTC_OK) return rc;
  const size_t held = mol->ws_ao.bytes, tile_most = sizeof(double) * (size_t)nq * TP * mol->Mpad;
  size_t budget = kMostAo;
  bool asked = false;
  auto ask = [&]() {
    size_t free_b = 0, total_b = 0;
    asked = true;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) budget = std::max(held, std::min(kMostAo, free_b / 4));
    else cudaGetLastError();  // clear the error; keep the default
  };
  if (const char* env = std::getenv("CTC_CHUNK_BYTES")) {
    const long long v = std::atoll(env);
    if (v > 0) {
      budget = (size_t)v;
      asked = true;
    }
  }
  // Capacity of a tile's compact AO set: Mpad always suffices.  When a chunk
  // sized for Mpad columns would hold fewer than four waves of tiles (large
  // bases: the 1 000-atom molecule keeps ~350 of 16 128 functions per tile), a
  // count-only screening pass over every tile of the call finds the largest
  // compact set and the workspace is sized for that instead.  It waits for
  // the stream once (to read the count back); smaller bases skip it.
  int Kcap = mol->Mpad, Kpcap = quads ? mol->Mpad : 0;
  auto few_tiles = [&]() { return (int64_t)(budget / tile_most) < 4 * nsm && ntiles > nsm; };
  if (!asked && !few_tiles() && ask_free_memory(tile_most * chunk_tiles(budget, tile_most, ntiles, nsm), held)) ask();
  if (few_tiles()) {
    const int64_t PB = std::min<int64_t>(ntiles, 16384);
    const size_t pb_bytes = sizeof(double) * (size_t)PB * TP * 3 + sizeof(int64_t) * (size_t)PB * TP + 1024;
    if ((rc = mol->ws_cap.ensure(pb_bytes, st)) != CTC_OK) return rc;
    TileBatch pb;
    pb.TP = TP;
    Carve cv{(char*)mol->ws_cap.p};
    int* d_kmax = cv.take<int>(2);
    pb.xyz = cv.take<double>((size_t)PB * TP * 3);
    pb.out = cv.take<int64_t>((size_t)PB * TP);
    CTC_CUDA_TRY(cudaMemsetAsync(d_kmax, 0, 2 * sizeof(int), st));
    for (int64_t t0 = 0; t0 < ntiles; t0 += PB) {
      pb.C = (int)std::min<int64_t>(PB, ntiles - t0);
      if ((rc = tile_points(pb, t0)) != CTC_OK) return rc;
      tile_capacity_kernel<<<pb.C, kTileThreads, 0, st>>>(mol->d_segs, mol->nseg, pb, d_kmax);
      CTC_CUDA_TRY(cudaGetLastError());
      mol->host_launches += 2;
    }
    CTC_CUDA_TRY(cudaMemcpyAsync(mol->h_status + 1, d_kmax, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    CTC_CUDA_TRY(cudaStreamSynchronize(st));
    Kcap = std::min(mol->Mpad, std::max(kKtAlign, (int)mol->h_status[1]));
    if (quads) Kpcap = std::min(mol->Mpad, std::max(kKtAlign, (int)mol->h_status[2]));
  }
  const size_t ao_per_tile = sizeof(double) * (size_t)nq * TP * Kcap;
  int64_t C = chunk_tiles(budget, ao_per_tile, ntiles, nsm);
  if (!asked && ask_free_memory(ao_per_tile * C, held)) {
    ask();
    C = chunk_tiles(budget, ao_per_tile, ntiles, nsm);
  }
  rc = mol->ws_ao.ensure(ao_per_tile * C, st);
  if (rc == CTC_ERR_NOMEM && !asked) {
    ask();  // a small block did not fit: the chunk that the free memory allows
    C = chunk_tiles(budget, ao_per_tile, ntiles, nsm);
    rc = mol->ws_ao.ensure(ao_per_tile * C, st);
  }
  if (rc != CTC_OK) return rc;
  if ((rc = mol->ws_misc.ensure(tile_bytes(mol, (int)C, TP, Kcap, Kpcap), st)) != CTC_OK) return rc;
  TileBatch tb;
  tb.TP = TP;
  tb.Kcap = Kcap;
  tb.nq = nq;
  tb.ao = (double*)mol->ws_ao.p;
  {
    Carve cv{(char*)mol->ws_misc.p};
    tb.xyz = cv.take<double>((size_t)C * TP * 3);
    tb.out = cv.take<int64_t>((size_t)C * TP);
    tb.nsig = cv.take<int32_t>(C);
    tb.ktrue = cv.take<int32_t>(C);
    tb.kt = cv.take<int32_t>(C);
    tb.segs = cv.take<int32_t>((size_t)C * mol->nseg);
    tb.k0 = cv.take<int32_t>((size_t)C * mol->nseg);
    tb.aomap = cv.take<int32_t>((size_t)C * tb.Kcap);
    tb.order = cv.take<int32_t>(C);
    tb.counter = cv.take<int32_t>(2);
    tb.parts = tb.counter + 1;
    tb.kp = cv.take<int32_t>(C);
    tb.kq = cv.take<int32_t>((size_t)C * (Kpcap / 4));
    tb.ksrc = cv.take<int32_t>((size_t)C * Kpcap);
    tb.Kpcap = Kpcap;
  }
  for (int64_t t0 = 0; t0 < ntiles; t0 += C) {
    tb.C = (int)std::min<int64_t>(C, ntiles - t0);
    if ((rc = tile_points(tb, t0)) != CTC_OK) return rc;
    screen_kernel<<<tb.C, kTileThreads, 0, st>>>(mol->d_segs, mol->nseg, tb, rows, mol->d_stats,
                                                 mol->d_status);
    CTC_CUDA_TRY(cudaGetLastError());
    tile_order_kernel<<<1, kOrderThreads, 0, st>>>(tb, nsm, 8.0 * mol->M * mol->M);
    CTC_CUDA_TRY(cudaGetLastError());
    {
      ProfScope ps(mol, 1, st);
      rc = ao_launch ? (*ao_launch)(tb) : launch_ao_tiles(mol, tb, deriv, st);
      if (rc != CTC_OK) return rc;
    }
    mol->host_launches += 4;
    mol->host_chunks += 1;
    if ((rc = compute(tb)) != CTC_OK) return rc;
  }
  return CTC_OK;
}

}  // namespace
}  // namespace ctc
