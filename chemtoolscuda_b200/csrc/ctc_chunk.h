// ctc_chunk.h -- host-side rules of the tile pipeline (arithmetic only): how many
// tiles a chunk takes and when the driver is asked for the free memory first;
// whether and how finely points are sorted along a Morton curve.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace ctc {

// Largest AO block of a chunk (a quarter of the free device memory, if that is
// less), and the block that is taken without asking how much is free.
constexpr size_t kMostAo = (size_t)12 << 30, kSmallAo = (size_t)64 << 20;

// Tiles of a chunk: what the budget holds and at least one per SM.  A call of
// several chunks takes whole rounds of one tile per SM where that drops at most a
// twentieth of the chunk (1 787 -> 1 776 tiles, FP64 contraction of the 90 945-point
// cube of 200 atoms: call 33.5 -> 33.2 ms; the tensor-core form, which deals out
// items, 78.0 either way; 714 -> 592 would make eleven chunks of nine).
inline int64_t chunk_tiles(size_t budget, size_t tile_bytes, int64_t ntiles, int sms) {
  const int64_t C = std::min<int64_t>(std::max<int64_t>(sms, (int64_t)(budget / tile_bytes)), ntiles);
  return C < ntiles && C % sms <= C / 20 ? C - C % sms : C;
}

// The free memory matters only to a block that has still to be allocated: not to
// one that fits what the molecule holds already.  (The question takes 0.1 to 6 ms
// on a shared host, as long as a whole call of 1e5 points.)
inline bool ask_free_memory(size_t block, size_t held) { return block > std::max(held, kSmallAo); }

// Bits per axis of the Morton keys of points over a box of edge ext (bohr).  Cells
// of 1/256 of the box are well below a tile's size for most molecules (0.14 bohr
// for 12 atoms), and 24 bits take three passes of the radix sort instead of four
// (30 000 points of 12 to 60 atoms: 1 to 8% of the call).  Beyond 512 bohr such a
// cell is wider than 2 bohr and holds whole tiles' worth of unordered points: on a
// chain of 500 bohr 24 and 30 bits take the same time (200 000 points on
// tensor cores: 1.00 and, all at one end, 1.02 of the 30-bit time), on one of 1 500
// bohr 24 bits cost 5 to 11% more.
inline int morton_axis_bits(double ext) { return ext <= 512.0 ? 8 : 10; }

// Are explicit points sorted at all?  A basis of up to 256 functions at up to
// 2 048 points is not, unless its atoms lie far apart (box beyond 64 bohr, 24 of
// them padding): its tiles keep most functions in any order, and the sort's two
// launches take as long as the rest (a call of 100 to 2 048 points unsorted, of its
// time sorted: 6 to 20 atoms 0.68 to 0.96, chain of 40 bohr 0.81 to 1.04, of 70 bohr
// 0.78 to 1.21, of 170 bohr 0.94 to 1.42).
inline bool sort_points(int64_t n, int mpad, double ext) { return n > 2048 || mpad > 256 || !(ext <= 64.0); }

}  // namespace ctc
