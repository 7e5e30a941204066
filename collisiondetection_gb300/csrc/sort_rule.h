// Which form a key sort takes (radix_sort.cu).
#pragma once

#include <stdint.h>

namespace ccd {

constexpr int kGridThreads = 512;
constexpr int64_t kGridPer = 2048;                  // keys per block at least
constexpr int64_t kGridMaxKeys = (int64_t)1 << 22;
constexpr int kGridMaxBlocks = 256;

// Blocks of the one-launch sort that a device runs at once, at most one per SM
// (per_sm: blocks that one SM holds); 0 where it cannot run it.
inline int grid_sort_limit(bool cooperative, int sms, int per_sm) {
  if (!cooperative || per_sm < 1 || sms < 1) return 0;
  return sms < kGridMaxBlocks ? sms : kGridMaxBlocks;
}

// Blocks of the one-launch sort of n keys, or 0 where the passes are launched
// one by one: beyond kGridMaxKeys, and on a device without room (limit 0).
inline int grid_sort_blocks(int64_t n, int limit) {
  if (n <= 0 || n > kGridMaxKeys) return 0;
  const int64_t want = (n + kGridPer - 1) / kGridPer;
  return want < limit ? (int)want : limit;
}

}  // namespace ccd
