// Stable least-significant-digit radix sort of (64-bit key, 32-bit value) pairs, 8 bits per pass.
// Used to put GPU-side events in order of their start timestamp before sizes are scanned, so the
// emit pass still writes every event straight to its final offset.  Per pass: per-tile digit
// histograms, one exclusive scan over the digit-major histogram, and a stable scatter.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace k2j {

constexpr int kSortThreads = 256;
// Rounds of kSortThreads keys a block (a tile) takes.  The scatter's rounds are a serial chain of barriers, so a sort too
// short to fill the chip with tiles of eight rounds takes fewer, up to one tile for every block that can be resident
// (8 an SM, 1184 with 148 SMs): 500 k keys fill 245 blocks at eight rounds and 977 at two.  Size pass and sort of 500 k
// events: 263 -> 252 us.
constexpr uint64_t kSortBlocks = 8;
constexpr uint32_t kSortMaxRounds = 8;
inline uint32_t sort_rounds(uint64_t n, uint32_t sms) {
  const uint64_t round = sms * kSortBlocks * kSortThreads, r = (n + round - 1) / round;
  return r < 1 ? 1u : r > kSortMaxRounds ? kSortMaxRounds : (uint32_t)r;
}
inline uint32_t sort_tiles(uint64_t n, uint32_t sms) {
  const uint64_t tile = (uint64_t)sort_rounds(n, sms) * kSortThreads;
  return (uint32_t)((n + tile - 1) / tile);
}

// hist[digit * n_tiles + tile] = number of keys of the tile with that digit
__global__ void __launch_bounds__(kSortThreads) k_rs_hist(const uint64_t* keys, uint64_t n, uint32_t rounds, int shift, uint32_t* hist, uint32_t n_tiles) {
  __shared__ uint32_t s_h[256];
  let_next_start();
  wait_for_previous();
  s_h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = (uint64_t)blockIdx.x * rounds * kSortThreads;
  for (uint32_t r = 0; r < rounds; r++) {
    const uint64_t i = base + (uint64_t)r * kSortThreads + threadIdx.x;
    if (i < n) atomicAdd(&s_h[(uint32_t)(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * n_tiles + blockIdx.x] = s_h[threadIdx.x];
}

// base[digit * n_tiles + tile] = global position of the tile's first key with that digit
__global__ void __launch_bounds__(kSortThreads) k_rs_scatter(const uint64_t* keys, const uint32_t* vals, uint64_t n, uint32_t rounds, int shift,
                                                             const uint64_t* base, uint32_t n_tiles, uint64_t* keys_out,
                                                             uint32_t* vals_out) {
  __shared__ uint32_t s_cnt[kSortThreads / 32][256];  // per warp and digit: count, then offset within the round
  __shared__ uint32_t s_run[256];                      // keys of each digit placed by earlier rounds
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  let_next_start();
  wait_for_previous();
  s_run[threadIdx.x] = 0;
  const uint64_t tile0 = (uint64_t)blockIdx.x * rounds * kSortThreads;
  for (uint32_t r = 0; r < rounds; r++) {
    for (int i = threadIdx.x; i < (kSortThreads / 32) * 256; i += kSortThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const uint64_t i = tile0 + (uint64_t)r * kSortThreads + threadIdx.x;
    const bool in = i < n;
    const uint64_t key = in ? keys[i] : 0;
    const uint32_t val = in ? vals[i] : 0;
    const uint32_t dg = (uint32_t)(key >> shift) & 255u;
    // lanes of this warp with the same digit (out-of-range lanes form their own group)
    const uint32_t peers = __match_any_sync(0xffffffffu, in ? dg : 256u + 0u);
    const uint32_t rank_in_warp = __popc(peers & ((1u << lane) - 1u));
    if (in && rank_in_warp == 0) s_cnt[w][dg] = __popc(peers);
    __syncthreads();
    {  // thread d: exclusive prefix over warps of digit d, on top of what earlier rounds placed
      const uint32_t d = threadIdx.x;
      uint32_t acc = s_run[d];
#pragma unroll
      for (int ww = 0; ww < kSortThreads / 32; ww++) { const uint32_t t = s_cnt[ww][d]; s_cnt[ww][d] = acc; acc += t; }
      s_run[d] = acc;
    }
    __syncthreads();
    if (in) {
      const uint64_t pos = base[(uint64_t)dg * n_tiles + blockIdx.x] + s_cnt[w][dg] + rank_in_warp;
      keys_out[pos] = key;
      vals_out[pos] = val;
    }
    __syncthreads();
  }
}

// rank[vals_sorted[pos]] = pos
__global__ void k_rs_invert(const uint32_t* vals_sorted, uint64_t n, uint32_t* rank) {
  let_next_start();
  wait_for_previous();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) rank[vals_sorted[i]] = (uint32_t)i;
}

}  // namespace k2j
