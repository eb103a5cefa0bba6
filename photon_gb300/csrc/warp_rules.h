// The rules by which the warps of a persistent kernel size their work,
// __host__ __device__ so that host tests run the very code the kernels run.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#ifndef PHC_HD
#define PHC_HD __host__ __device__ __forceinline__
#endif

namespace phc {

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
PHC_HD uint32_t lanes_for(uint32_t n, uint32_t warps)
{
  const uint32_t half = warps / 2u > 1u ? warps / 2u : 1u;
  uint32_t k = 1u;
  while (k < 32u && k * half < n)
    k <<= 1;
  return k;
}

// Rays per warp of a ray back-end call that gives every warp its rays by its
// place in the grid; 0 for longer calls, whose warps take batches from a
// counter.  All rays of such a call must be in flight at once (half of the
// grid's warps are resident): beyond, a block's place is only free again when
// its last warp is done, and 160K-311K rays took 3-15% longer than from the
// counter (200K random rays, 50K triangles: 206 and 226 us).  16 rays a
// warp cost the issue slots of full warps and save little waiting: 45K-77K camera
// rays on 6K triangles 80-91 us from the counter, 83-103 with 16, 72-81 with 32.
// With 8, 30K rays on 500K triangles: camera rays 76 -> 61 us, any hit 53 -> 41
// and 37 -> 35, incoherent closest hits 58 -> 60 (6K triangles: 79 -> 81, 74 -> 67,
// 88 -> 89); with fewer, all calls gain (1,000 rays on 6K triangles 79 -> 51 us).
PHC_HD uint32_t brief_lanes(uint32_t n, uint32_t warps)
{
  const uint32_t half = warps / 2u > 1u ? warps / 2u : 1u;
  if (n > half * 32u)
    return 0u;
  const uint32_t k = lanes_for(n, warps);
  return k <= 8u ? k : 32u;
}

// Idle lanes at which a warp that works on per_warp rays at a time takes new
// ones: what the caller asked for (1..32; 32: only when all are idle), but no
// more than half of the rays of a warp that has fewer than 32.
PHC_HD uint32_t refill_lanes(uint32_t refill, uint32_t per_warp)
{
  const uint32_t most = per_warp >= 32u ? 32u : (per_warp + 1u) >> 1;
  return refill < most ? refill : most;
}

} // namespace phc
