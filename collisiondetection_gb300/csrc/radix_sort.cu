// Stable LSD radix sort and exclusive scan (radix_sort.cuh).
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "radix_sort.cuh"
#include "sort_rule.h"

namespace ccd {

namespace {

constexpr int kThreads = 256;
constexpr int kItems = 16;
constexpr int kTile = kThreads * kItems;  // keys per block
constexpr int kWarps = kThreads / 32;
constexpr int kRun = kTile / kWarps;      // keys per warp run (contiguous)

size_t align_up(size_t x) { return (x + 255) / 256 * 256; }

// ------------------------------------------------------------------ scan
// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t &total) {
  __shared__ uint32_t warp_sums[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < kWarps ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kWarps) warp_sums[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  total = warp_sums[kWarps - 1];
  const uint32_t before = warp > 0 ? warp_sums[warp - 1] : 0;
  __syncthreads();
  return before + x - v;
}

__global__ void __launch_bounds__(kThreads) scan_tiles(const uint32_t *in, uint32_t *out, int64_t n,
                                                       uint32_t *tile_sums) {
  const int64_t base = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
  uint32_t v[kItems];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    v[i] = (base + i < n) ? in[base + i] : 0u;
    sum += v[i];
  }
  uint32_t total;
  uint32_t run = block_exclusive(sum, total);
#pragma unroll
  for (int i = 0; i < kItems; i++) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kThreads) add_offsets(uint32_t *out, int64_t n, const uint32_t *tile_offs) {
  const int64_t base = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
  const uint32_t add = tile_offs[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kItems; i++)
    if (base + i < n) out[base + i] += add;
}

__global__ void write_total(const uint32_t *scanned, const uint32_t *in, int64_t n, uint32_t *total) {
  *total = n > 0 ? scanned[n - 1] + in[n - 1] : 0u;
}

// ------------------------------------------------------------------ radix sort
__global__ void __launch_bounds__(kThreads) digit_histogram(const uint64_t *keys, int64_t n, int shift,
                                                            uint32_t *counts, int nblocks) {
  __shared__ uint32_t hist[256];
  hist[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kTile;
  for (int i = threadIdx.x; i < kTile; i += kThreads) {
    const int64_t k = base + i;
    if (k < n) atomicAdd(&hist[(keys[k] >> shift) & 255u], 1u);
  }
  __syncthreads();
  counts[(int64_t)threadIdx.x * nblocks + blockIdx.x] = hist[threadIdx.x];
}

__global__ void __launch_bounds__(kThreads) digit_scatter(const uint64_t *keys, const uint32_t *vals, uint64_t *okeys,
                                                          uint32_t *ovals, int64_t n, int shift,
                                                          const uint32_t *offsets, int nblocks) {
  __shared__ uint32_t warp_hist[kWarps][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < kWarps * 256; i += kThreads) (&warp_hist[0][0])[i] = 0;
  __syncthreads();
  const int64_t run0 = (int64_t)blockIdx.x * kTile + (int64_t)warp * kRun;
  // Digit counts of this warp's run.
  for (int c = 0; c < kRun; c += 32) {
    const int64_t k = run0 + c + lane;
    if (k < n) atomicAdd(&warp_hist[warp][(keys[k] >> shift) & 255u], 1u);
  }
  __syncthreads();
  // Per digit: offsets of the warp runs inside the block, then the block's
  // global offset.
  {
    const int d = threadIdx.x;
    uint32_t run = offsets[(int64_t)d * nblocks + blockIdx.x];
    for (int w = 0; w < kWarps; w++) {
      const uint32_t c = warp_hist[w][d];
      warp_hist[w][d] = run;
      run += c;
    }
  }
  __syncthreads();
  // Stable scatter: runs in order, chunks of 32 in order, lanes in order.
  for (int c = 0; c < kRun; c += 32) {
    const int64_t k = run0 + c + lane;
    const bool valid = k < n;
    uint64_t key = valid ? keys[k] : 0;
    const unsigned d = valid ? (unsigned)((key >> shift) & 255u) : 256u + lane;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t pos = 0;
    if (valid) pos = warp_hist[warp][d] + __popc(peers & lt);
    __syncwarp();
    if (valid && (peers & lt) == 0) warp_hist[warp][d] += __popc(peers);
    __syncwarp();
    if (valid) {
      okeys[pos] = key;
      if (vals) ovals[pos] = vals[k];
    }
  }
}

// The whole sort in one cooperative launch, for the sizes at which the passes'
// launches and not their traffic set the time: a pass of the kernels above is
// three or more launches of some 7 us each whatever their size, and a mesh
// step sorts two lists of 10^4 to 10^5 keys in five passes each: the sorts of
// a 211,970-face step took 365 us, now 77.  Every block keeps one contiguous
// range; per pass it counts its digits, the grid meets, thread d adds up the
// other blocks' counts of digit d, and the block scatters.  Both forms on keys
// of 38 bits: 2^12 keys 111 and 40 us, 2^16 136 and 45, 2^20 210 and 108, 2^22
// 339 and 258, 2^23 693 and 768 (one block per SM no longer keeps enough of its
// range in flight), so the line lies at 2^22.
constexpr int kGridWarps = kGridThreads / 32;

__global__ void __launch_bounds__(kGridThreads) sort_grid(uint64_t *keys, uint64_t *keys_alt, int64_t n, int begin_bit,
                                                          int end_bit, uint32_t *counts) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  __shared__ uint32_t warp_hist[kGridWarps][256];
  __shared__ uint32_t warp_sums[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nblocks = (int)gridDim.x;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t run = ((n + nblocks - 1) / nblocks + kGridThreads - 1) / kGridThreads * 32;
  const int64_t run0 = ((int64_t)blockIdx.x * kGridWarps + warp) * run;
  const int64_t run1 = run0 + run < n ? run0 + run : n;
  uint64_t *src = keys, *dst = keys_alt;
  int pass = 0;
  for (int shift = begin_bit; shift < end_bit; shift += 8, pass++) {
    for (int i = tid; i < kGridWarps * 256; i += kGridThreads) (&warp_hist[0][0])[i] = 0;
    __syncthreads();
    for (int64_t k = run0 + lane; k < run1; k += 32) atomicAdd(&warp_hist[warp][(src[k] >> shift) & 255u], 1u);
    __syncthreads();
    if (tid < 256) {
      uint32_t c = 0;
#pragma unroll
      for (int w = 0; w < kGridWarps; w++) c += warp_hist[w][tid];
      counts[(size_t)blockIdx.x * 256 + tid] = c;
    }
    grid.sync();
    uint32_t before = 0, total = 0, x = 0;
    if (tid < 256) {
#pragma unroll 8
      for (int b = 0; b < nblocks; b++) {
        const uint32_t c = __ldcg(counts + (size_t)b * 256 + tid);
        total += c;
        if (b < (int)blockIdx.x) before += c;
      }
      x = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) warp_sums[warp] = x;
    }
    __syncthreads();
    if (tid < 256) {
      uint32_t at = before + x - total;
      for (int w = 0; w < warp; w++) at += warp_sums[w];
#pragma unroll
      for (int w = 0; w < kGridWarps; w++) {
        const uint32_t c = warp_hist[w][tid];
        warp_hist[w][tid] = at;
        at += c;
      }
    }
    __syncthreads();
    // Stable scatter: runs in order, chunks of 32 in order, lanes in order.
    // (212,000 Morton keys 60 us unrolled by two, 69 rolled, 90 by four.)
#pragma unroll 2
    for (int64_t k0 = run0; k0 < run1; k0 += 32) {
      const int64_t k = k0 + lane;
      const bool valid = k < run1;
      const uint64_t key = valid ? src[k] : 0;
      const unsigned d = valid ? (unsigned)((key >> shift) & 255u) : 256u + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      uint32_t pos = 0;
      if (valid) pos = warp_hist[warp][d] + __popc(peers & lt);
      __syncwarp();
      if (valid && (peers & lt) == 0) warp_hist[warp][d] += __popc(peers);
      __syncwarp();
      if (valid) dst[pos] = key;
    }
    grid.sync();
    uint64_t *t = src;
    src = dst;
    dst = t;
  }
  if (pass & 1) {
    for (int64_t k = (int64_t)blockIdx.x * kGridThreads + tid; k < n; k += (int64_t)nblocks * kGridThreads)
      keys[k] = src[k];
  }
}

// Blocks of sort_grid that the current device runs at once, at most one per SM;
// asked once per device (the occupancy query takes longer than a launch).
cudaError_t resident_blocks(int *most) {
  constexpr int kDevices = 64;
  static std::atomic<int> known[kDevices];  // blocks + 1; 0: not asked yet
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kDevices && known[dev].load() > 0) {
    *most = known[dev].load() - 1;
    return cudaSuccess;
  }
  int sms = 0, cooperative = 0, per_sm = 0;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sort_grid, kGridThreads, 0);
  if (e != cudaSuccess) return e;
  *most = grid_sort_limit(cooperative != 0, sms, per_sm);
  if (dev >= 0 && dev < kDevices) known[dev].store(*most + 1);
  return cudaSuccess;
}

}  // namespace

size_t scan_temp_bytes(int64_t n) {
  size_t bytes = 0;
  int64_t m = n;
  while (true) {
    const int64_t tiles = (m + kTile - 1) / kTile;
    bytes += 2 * align_up((size_t)tiles * sizeof(uint32_t));
    if (tiles <= 1) break;
    m = tiles;
  }
  return bytes + 256;
}

static cudaError_t scan_rec(const uint32_t *in, uint32_t *out, int64_t n, char *temp, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t tiles = (n + kTile - 1) / kTile;
  uint32_t *sums = (uint32_t *)temp;
  uint32_t *offs = (uint32_t *)(temp + align_up((size_t)tiles * sizeof(uint32_t)));
  char *next = temp + 2 * align_up((size_t)tiles * sizeof(uint32_t));
  scan_tiles<<<(unsigned)tiles, kThreads, 0, s>>>(in, out, n, sums);
  if (tiles > 1) {
    cudaError_t e = scan_rec(sums, offs, tiles, next, s);
    if (e != cudaSuccess) return e;
    add_offsets<<<(unsigned)tiles, kThreads, 0, s>>>(out, n, offs);
  }
  return cudaGetLastError();
}

cudaError_t exclusive_scan_u32(const uint32_t *in, uint32_t *out, int64_t n, uint32_t *total, void *temp,
                               size_t temp_bytes, cudaStream_t s) {
  if (temp_bytes < scan_temp_bytes(n)) return cudaErrorInvalidValue;
  if (total && n > 0 && in == out) return cudaErrorInvalidValue;  // the total needs the input
  cudaError_t e = scan_rec(in, out, n, (char *)temp, s);
  if (e != cudaSuccess) return e;
  if (total) {
    if (n > 0)
      write_total<<<1, 1, 0, s>>>(out, in, n, total);
    else
      e = cudaMemsetAsync(total, 0, sizeof(uint32_t), s);
  }
  return e != cudaSuccess ? e : cudaGetLastError();
}

size_t radix_sort_temp_bytes(int64_t n) {
  const int64_t nblocks = (n + kTile - 1) / kTile;
  const int64_t m = std::max<int64_t>(256 * nblocks, 256 * kGridMaxBlocks);  // sort_grid: 256 counts per block
  return 2 * align_up((size_t)m * sizeof(uint32_t)) + scan_temp_bytes(m);
}

cudaError_t radix_sort_u64(uint64_t *keys, uint64_t *keys_alt, uint32_t *vals, uint32_t *vals_alt, int64_t n,
                           int begin_bit, int end_bit, void *temp, size_t temp_bytes, cudaStream_t s) {
  if (n <= 1) return cudaSuccess;
  if (n >= (int64_t)1 << 31 || temp_bytes < radix_sort_temp_bytes(n)) return cudaErrorInvalidValue;
  const int64_t nblocks = (n + kTile - 1) / kTile;
  const int64_t m = 256 * nblocks;
  if (!vals && n <= kGridMaxKeys) {
    int most = 0;
    cudaError_t e = resident_blocks(&most);
    if (e != cudaSuccess) return e;
    const int grid = grid_sort_blocks(n, most);
    if (grid > 0) {
      uint32_t *counts = (uint32_t *)temp;
      void *args[] = {&keys, &keys_alt, &n, &begin_bit, &end_bit, &counts};
      e = cudaLaunchCooperativeKernel((const void *)sort_grid, dim3(grid), dim3(kGridThreads), args, 0, s);
      // a context that may use part of the SMs only refuses what it cannot
      // hold at once: the passes then follow one by one
      if (e != cudaErrorCooperativeLaunchTooLarge) return e;
      cudaGetLastError();
    }
  }
  uint32_t *counts = (uint32_t *)temp;
  uint32_t *offsets = (uint32_t *)((char *)temp + align_up((size_t)m * sizeof(uint32_t)));
  char *scan_tmp = (char *)temp + 2 * align_up((size_t)m * sizeof(uint32_t));
  uint64_t *src = keys, *dst = keys_alt;
  uint32_t *vsrc = vals, *vdst = vals_alt;
  int passes = 0;
  for (int shift = begin_bit; shift < end_bit; shift += 8, passes++) {
    digit_histogram<<<(unsigned)nblocks, kThreads, 0, s>>>(src, n, shift, counts, (int)nblocks);
    cudaError_t e = scan_rec(counts, offsets, m, scan_tmp, s);
    if (e != cudaSuccess) return e;
    digit_scatter<<<(unsigned)nblocks, kThreads, 0, s>>>(src, vsrc, dst, vdst, n, shift, offsets, (int)nblocks);
    uint64_t *t = src;
    src = dst;
    dst = t;
    uint32_t *tv = vsrc;
    vsrc = vdst;
    vdst = tv;
  }
  if (passes & 1) {
    cudaError_t e = cudaMemcpyAsync(keys, src, (size_t)n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    if (vals) {
      e = cudaMemcpyAsync(vals, vsrc, (size_t)n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
      if (e != cudaSuccess) return e;
    }
  }
  return cudaGetLastError();
}

}  // namespace ccd
