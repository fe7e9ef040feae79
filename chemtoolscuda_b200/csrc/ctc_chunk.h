// ctc_chunk.h -- how many tiles a chunk of the tile pipeline takes, and when the
// driver is asked for the free memory first (host arithmetic only).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace ctc {

// Largest AO block of a chunk (a quarter of the free device memory, if that is
// less), and the block that is taken without asking how much is free.
constexpr size_t kMostAo = (size_t)12 << 30, kSmallAo = (size_t)64 << 20;

// Tiles of a chunk: what the budget holds and at least one per SM; a call of
// several chunks takes whole rounds of one tile per SM.
inline int64_t chunk_tiles(size_t budget, size_t tile_bytes, int64_t ntiles, int sms) {
  const int64_t C = std::min<int64_t>(std::max<int64_t>(sms, (int64_t)(budget / tile_bytes)), ntiles);
  return C < ntiles ? C - C % sms : C;
}

// The free memory matters only to a block that has still to be allocated: not to
// one that fits what the molecule holds already.  (The question takes 0.1 to 6 ms
// on a shared host, as long as a whole call of 1e5 points.)
inline bool ask_free_memory(size_t block, size_t held) { return block > std::max(held, kSmallAo); }

}  // namespace ctc
