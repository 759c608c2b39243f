// Grid of the CTA path's global-bitmap mode (host arithmetic only).
#pragma once

#include <algorithm>
#include <cstddef>

namespace msbfs {

// Blocks for a call of num_sources sources, when `resident` blocks may run at
// once (the caller's share of the device) and the bitmaps of `in_l2` are the
// most that are kept in the L2. Every edge is an atomic on a bitmap, and more
// blocks than that slow each other down. Road 1448x1448 (262 KB bitmaps), S=512 /
// 2,048, ms with 152, 228, 304, 456 blocks: 62 / 222, 52 / 175, 42 / 158, 54 / 167.
// About as many sources per block each: the nearest whole number of rounds that
// the resident blocks can do. (The share has to be known here: cut to 85%
// afterwards, the blocks of one round took two: S=160 15.6 ms, 27.5 so.)
inline size_t global_bitmap_grid(size_t resident, size_t in_l2, size_t num_sources) {
  const size_t most = std::max<size_t>(std::min(resident, in_l2), 1);
  const size_t rounds = std::max({(num_sources + most / 2) / most,
                                  (num_sources + resident - 1) / resident, size_t(1)});
  return std::max<size_t>((num_sources + rounds - 1) / rounds, 1);
}

}  // namespace msbfs
