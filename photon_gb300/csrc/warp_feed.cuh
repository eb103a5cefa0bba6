// How the warps of the persistent kernels take their work: shared by the
// wavefront kernels and the ray back-end's.
#pragma once

#include <cstdint>

namespace phc {

constexpr uint32_t WARP_FULL = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Next `k`-item batch of a warp; uniform across the warp.  Every lane of
// the warp calls it.  The __syncwarp makes the reconvergence explicit: a
// lane that ran long divergent work (a tracking loop, a shading call) must
// be back before the warp votes, or the lanes' views of the batch differ.
__device__ __forceinline__ uint32_t warp_fetch(uint32_t *ctr, uint32_t k = 32u)
{
  __syncwarp();
  uint32_t base = 0;
  if (lane_id() == 0)
    base = atomicAdd(ctr, k);
  return __shfl_sync(WARP_FULL, base, 0);
}

// Rays that a warp of a persistent traversal or tracking kernel works on at a
// time, for a queue of n rays and a grid of `warps`: 32, or the power of two
// that still gives half of the grid's warps work when n is too short for
// full ones.  Such a queue is bound by latency: a step of a full warp takes
// as long as its slowest lane (on the 500K-triangle scene a lone ray's step
// takes 0.42 us and each triangle test 0.34 us, and a full warp makes 2.7-3.7
// tests in a row per step where a lane makes 0.4), and the idle schedulers
// cost nothing.  Measured on a 640 x 360, 1-spp frame of that scene: closest
// hits 0.89 -> 0.71 ms, shadow rays 0.52 -> 0.41 ms; an adaptive 811 x 613
// frame through a volume (one sample of every pixel per wave) 139 -> 122 ms.
// All of the grid's warps, or a quarter of them, instead of half measured 1%
// and 2% slower there.  Shading kernels gain nothing from it (their warps
// wait for instructions, which more warps fetch more often).
__device__ __forceinline__ uint32_t spread_lanes(uint32_t n)
{
  const uint32_t warps = max(gridDim.x * (blockDim.x / 32u) / 2u, 1u);
  uint32_t k = 1u;
  while (k < 32u && k * warps < n)
    k <<= 1;
  return k;
}

constexpr uint32_t FEED_CHUNK = 64;

// A persistent warp's supply of queue items [0, n): chunks of consecutive
// items from the launch's work counter, handed out to the warp's lanes as they
// become idle.  One atomic per chunk, and lanes that refill at different times
// still work on neighbouring rays.  Closest-hit traversal of the 500K workload
// (1024 x 1024, 128 spp) with one atomic per refill / chunks of 32 / 64 / 128 /
// 512 rays: 84.3 / 82.1 / 81.6 / 81.5 / 83.1 ms, shadow rays 13.4 / 13.3 / 12.4 /
// 12.6 / 13.1 ms (time_kernels).  The shading kernels (5.42 -> 5.57 ms in the
// box room) and the volume tracking gain nothing from it.
struct WarpFeed {
  uint32_t cur{0}, end{0}, chunk;
  bool last{false}; // the counter has run past n
  // per_warp: items the warp works on at a time (spread_lanes).  A chunk is at
  // most an eighth of a warp's share, so that the launch's end stays even.
  __device__ __forceinline__ WarpFeed(uint32_t n, uint32_t per_warp)
  {
    const uint32_t share = n / (gridDim.x * (blockDim.x / 32u) * 8u);
    chunk = per_warp < 32u ? per_warp : min(max(share & ~31u, 32u), FEED_CHUNK);
  }
  __device__ __forceinline__ bool empty() const { return last && cur == end; }
  // Up to k items: the first one; k becomes their number.  Uniform across the
  // warp, called by all of its lanes.
  __device__ __forceinline__ uint32_t take(uint32_t *ctr, uint32_t n, uint32_t &k)
  {
    if (cur == end) {
      cur = warp_fetch(ctr, chunk);
      last = cur + chunk >= n;
      end = min(cur + chunk, n);
      cur = min(cur, n);
    }
    const uint32_t base = cur;
    k = min(k, end - cur);
    cur += k;
    return base;
  }
};

// Blocks that work in step.  Shading code is far larger than the instruction
// caches, and warps that run through it each at its own place wait for
// instructions more than for anything else; the warps of one block, started
// together on a batch of blockDim.x consecutive items, fetch it once for all.
// Every thread of the block calls these.

// Items a block takes at a time: all its threads', or whole warps' fewer when
// the queue is too short to give every block of the grid that many.
__device__ __forceinline__ uint32_t block_share(uint32_t n)
{
  const uint32_t even = ((n + gridDim.x - 1u) / gridDim.x + 31u) & ~31u;
  return min(max(even, 32u), blockDim.x);
}
__device__ __forceinline__ uint32_t block_fetch(uint32_t *ctr, uint32_t k)
{
  __shared__ uint32_t base;
  __syncthreads();
  if (threadIdx.x == 0)
    base = atomicAdd(ctr, k);
  __syncthreads();
  return base;
}

} // namespace phc
