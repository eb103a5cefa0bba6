// How the warps of the persistent kernels take their work: shared by the
// wavefront kernels and the ray back-end's.
#pragma once

#include <cstdint>

#include "warp_rules.h"

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

// lanes_for this grid.
__device__ __forceinline__ uint32_t spread_lanes(uint32_t n)
{
  return lanes_for(n, gridDim.x * (blockDim.x / 32u));
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
  // per_warp: items the warp works on at a time (spread_lanes).  A full warp's
  // chunk is an eighth of its share, so that the launch's end stays even, but
  // at least 32 and at most FEED_CHUNK items.
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
