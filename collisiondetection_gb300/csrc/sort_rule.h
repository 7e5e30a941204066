// Which form a key sort takes (radix_sort.cu).
#pragma once

#include <stdint.h>

namespace ccd {

constexpr int kGridThreads = 512;
constexpr int64_t kGridPer = 2048;                  // keys per block at least
constexpr int64_t kGridMaxKeys = (int64_t)1 << 22;
constexpr int kGridMaxBlocks = 256;

// Blocks of the one-launch sort of n keys, at most one per SM, or 0 where the
// passes are launched one by one: beyond kGridMaxKeys, and on a device that
// cannot hold the blocks all at once (per_sm: blocks that one SM holds).
inline int grid_sort_blocks(int64_t n, bool cooperative, int sms, int per_sm) {
  if (n <= 0 || n > kGridMaxKeys || !cooperative || per_sm < 1 || sms < 1) return 0;
  const int most = sms < kGridMaxBlocks ? sms : kGridMaxBlocks;
  const int64_t want = (n + kGridPer - 1) / kGridPer;
  return want < most ? (int)want : most;
}

}  // namespace ccd
