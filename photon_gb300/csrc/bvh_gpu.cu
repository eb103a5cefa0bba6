// GPU construction of the BVH8 of bvh8.h (same node and triangle-record
// layout, so the traversal kernels read either build).
//
// The reference builds its BVH on the host (src/photon/pt/bvh/bvh.cpp:77-125,
// median split); so does this renderer's default builder (binned SAH,
// bvh8.cpp).  For scene upload latency (many scenes per second in the batched
// mode) this file builds on the GPU instead:
//
//   1. primitive boxes and centroids, scene bounds;
//   2. 30-bit Morton codes of the centroids, sorted with a stable LSD radix
//      sort (4 passes of 8 bits: block histograms, one scan, ranked scatter);
//   3. a binary tree by parallel locally-ordered clustering (Meister and
//      Bittner, "Parallel Locally-Ordered Clustering for Bounding Volume
//      Hierarchy Construction", IEEE TVCG 2018): every cluster finds, among
//      the `radius` clusters on each side in Morton order (2, 4, 8, 16 or 32;
//      tuning key ploc_radius), the one whose merged
//      box has the least surface area; mutual pairs merge; the survivors are
//      compacted in order; repeat until one cluster is left.  Ties in the
//      area are broken by the pair's indices, so the globally smallest pair
//      is always mutual and every iteration merges;
//   4. the binary tree collapsed into the 8-wide quantised nodes level by
//      level, each node taking the up to eight descendants of largest area
//      (subtrees of more than max_leaf primitives opened first), the octant
//      slot order and the outward-rounded 8-bit child grid of the host
//      builder; a descendant with at most max_leaf primitives (1..3) is one
//      leaf child.  With a triangle cost (tuning key collapse_tri_cost) the
//      descendants are chosen instead by the surface-area cost of the whole
//      wide tree (the dynamic program of Ylitie, Karras and Laine,
//      "Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
//      BVHs", HPG 2017): bottom-up, the cheapest way to cover every
//      binary subtree with 1..8 slots, then the collapse follows those
//      choices from the root down.
//
// The result is deterministic except for where nodes and leaf records land
// in memory (atomic allocation order), which changes no traversal result.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "bvh_collapse.cuh"
#include "bvh_gpu.h"

namespace phc {
namespace {

constexpr int SORT_BLOCK = 256;
constexpr int TILE = 256;    // clusters per block of the neighbour search

__device__ __forceinline__ float area(const float *lo, const float *hi)
{
  const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
  return 2.f * (dx * dy + dy * dz + dz * dx);
}

// ---------------------------------------------------------------- stage 1
// Primitive boxes (6 floats) and the scene's centroid bounds through ordered
// integer atomics on the float bits.
__device__ __forceinline__ uint32_t ord(float f)
{
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord(uint32_t u)
{
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__global__ void k_prim_boxes(const float4 *__restrict__ pos, const uint4 *__restrict__ vidx, uint32_t n,
    float *__restrict__ boxes, uint32_t *cbounds)
{
  float clo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, chi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 v = vidx[i];
    const float4 a = pos[v.x], b = pos[v.y], c = pos[v.z];
    float *bx = boxes + 6 * size_t(i);
    bx[0] = fminf(fminf(a.x, b.x), c.x);
    bx[1] = fminf(fminf(a.y, b.y), c.y);
    bx[2] = fminf(fminf(a.z, b.z), c.z);
    bx[3] = fmaxf(fmaxf(a.x, b.x), c.x);
    bx[4] = fmaxf(fmaxf(a.y, b.y), c.y);
    bx[5] = fmaxf(fmaxf(a.z, b.z), c.z);
    for (int k = 0; k < 3; ++k) {
      const float cc = 0.5f * (bx[k] + bx[3 + k]);
      clo[k] = fminf(clo[k], cc);
      chi[k] = fmaxf(chi[k], cc);
    }
  }
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      clo[k] = fminf(clo[k], __shfl_xor_sync(0xffffffffu, clo[k], o));
      chi[k] = fmaxf(chi[k], __shfl_xor_sync(0xffffffffu, chi[k], o));
    }
  }
  if ((threadIdx.x & 31u) == 0)
    for (int k = 0; k < 3; ++k) {
      atomicMin(&cbounds[k], ord(clo[k]));
      atomicMax(&cbounds[3 + k], ord(chi[k]));
    }
}

__device__ __forceinline__ uint32_t spread10(uint32_t x)
{
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__global__ void k_morton(const float *__restrict__ boxes, uint32_t n, const uint32_t *cbounds,
    uint32_t *__restrict__ keys, uint32_t *__restrict__ vals)
{
  float lo[3], sc[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = unord(cbounds[k]);
    const float ext = unord(cbounds[3 + k]) - lo[k];
    sc[k] = ext > 0.f ? 1023.99f / ext : 0.f;
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float *bx = boxes + 6 * size_t(i);
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
      const float c = 0.5f * (bx[k] + bx[3 + k]);
      const float f = (c - lo[k]) * sc[k];
      q[k] = uint32_t(fminf(fmaxf(f, 0.f), 1023.f));
    }
    keys[i] = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
    vals[i] = i;
  }
}

// ---------------------------------------------------------------- stage 2
// Stable LSD radix sort, one element per thread: per-block digit counts,
// one exclusive scan over (digit, block), then each element's rank among the
// equal digits before it in its block (lanes through match_any, warps
// through shared counts).
__global__ void __launch_bounds__(SORT_BLOCK) k_digit_hist(const uint32_t *__restrict__ keys, uint32_t n, int shift,
    uint32_t *__restrict__ hist, uint32_t nblocks)
{
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t i = blockIdx.x * SORT_BLOCK + threadIdx.x;
  if (i < n)
    atomicAdd(&h[(keys[i] >> shift) & 0xffu], 1u);
  __syncthreads();
  hist[size_t(threadIdx.x) * nblocks + blockIdx.x] = h[threadIdx.x]; // digit-major
}

// Exclusive scan of `count` words in place by one block (sequential chunks,
// in order, so the result is independent of the block size): the scan of
// the tile sums below.
__global__ void __launch_bounds__(1024) k_scan_inplace(uint32_t *__restrict__ v, uint32_t count, uint32_t *total)
{
  __shared__ uint32_t part[1024];
  const uint32_t per = (count + 1023u) / 1024u;
  const uint32_t b = threadIdx.x * per, e = min(count, b + per);
  uint32_t s = 0;
  for (uint32_t i = b; i < e; ++i)
    s += v[i];
  part[threadIdx.x] = s;
  __syncthreads();
  for (uint32_t off = 1; off < 1024u; off <<= 1) {
    const uint32_t x = threadIdx.x >= off ? part[threadIdx.x - off] : 0u;
    __syncthreads();
    part[threadIdx.x] += x;
    __syncthreads();
  }
  uint32_t run = threadIdx.x ? part[threadIdx.x - 1] : 0u;
  for (uint32_t i = b; i < e; ++i) {
    const uint32_t x = v[i];
    v[i] = run;
    run += x;
  }
  if (threadIdx.x == 1023 && total)
    *total = part[1023];
}

// Multi-block exclusive scan: tiles of SCAN_TILE words, one block each;
// the tile sums, their scan by one block, then each tile's scan from its
// offset.  Integer sums, so the result is exact whatever the tiling.
constexpr int SCAN_T = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_T * SCAN_ITEMS;

__device__ __forceinline__ uint32_t block_exclusive(uint32_t x, uint32_t &block_total)
{
  __shared__ uint32_t warp_sum[SCAN_T / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t inc = x;
  for (uint32_t off = 1; off < 32u; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off)
      inc += y;
  }
  if (lane == 31u)
    warp_sum[warp] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (uint32_t w = 0; w < SCAN_T / 32; ++w) {
    const uint32_t v = warp_sum[w];
    before += w < warp ? v : 0u;
    all += v;
  }
  __syncthreads(); // warp_sum is reused by the next call
  block_total = all;
  return before + inc - x;
}

__global__ void __launch_bounds__(SCAN_T) k_tile_sums(const uint32_t *__restrict__ in, uint32_t n,
    uint32_t *__restrict__ sums)
{
  const size_t base = size_t(blockIdx.x) * SCAN_TILE;
  uint32_t s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const size_t i = base + size_t(k) * SCAN_T + threadIdx.x;
    if (i < n)
      s += in[i];
  }
  uint32_t total;
  block_exclusive(s, total);
  if (threadIdx.x == 0)
    sums[blockIdx.x] = total;
}

// Padded shared index: thread t's SCAN_ITEMS consecutive words fall in
// different banks.
__device__ __forceinline__ uint32_t scan_pad(uint32_t i) { return i + (i >> 5); }

__global__ void __launch_bounds__(SCAN_T) k_tile_scan(const uint32_t *in, uint32_t n,
    const uint32_t *__restrict__ offsets, uint32_t *out)
{
  __shared__ uint32_t tile[SCAN_TILE + SCAN_TILE / 32];
  const size_t base = size_t(blockIdx.x) * SCAN_TILE;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const uint32_t j = uint32_t(k) * SCAN_T + threadIdx.x;
    tile[scan_pad(j)] = base + j < n ? in[base + j] : 0u;
  }
  __syncthreads();
  uint32_t v[SCAN_ITEMS], local = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    v[k] = tile[scan_pad(threadIdx.x * SCAN_ITEMS + k)];
    local += v[k];
  }
  uint32_t total;
  uint32_t run = offsets[blockIdx.x] + block_exclusive(local, total);
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    tile[scan_pad(threadIdx.x * SCAN_ITEMS + k)] = run;
    run += v[k];
  }
  __syncthreads();
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    const uint32_t j = uint32_t(k) * SCAN_T + threadIdx.x;
    if (base + j < n)
      out[base + j] = tile[scan_pad(j)];
  }
}

__global__ void __launch_bounds__(SORT_BLOCK) k_digit_scatter(const uint32_t *__restrict__ kin,
    const uint32_t *__restrict__ vin, uint32_t n, int shift, const uint32_t *__restrict__ hist, uint32_t nblocks,
    uint32_t *__restrict__ kout, uint32_t *__restrict__ vout)
{
  __shared__ uint32_t wcount[SORT_BLOCK / 32][256];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t k = threadIdx.x; k < (SORT_BLOCK / 32) * 256; k += SORT_BLOCK)
    (&wcount[0][0])[k] = 0u;
  __syncthreads();
  const uint32_t i = blockIdx.x * SORT_BLOCK + threadIdx.x;
  const bool live = i < n;
  const uint32_t key = live ? kin[i] : 0u;
  const uint32_t dg = live ? (key >> shift) & 0xffu : 256u + lane; // dead lanes get private digits
  const uint32_t peers = __match_any_sync(0xffffffffu, dg);
  const uint32_t before = __popc(peers & ((1u << lane) - 1u));
  if (live && before == 0)
    wcount[warp][dg] = __popc(peers);
  __syncthreads();
  if (live) {
    uint32_t rank = before;
    for (uint32_t w = 0; w < warp; ++w)
      rank += wcount[w][dg];
    const uint32_t dst = hist[size_t(dg) * nblocks + blockIdx.x] + rank;
    kout[dst] = key;
    vout[dst] = vin[i];
  }
}

// ---------------------------------------------------------------- stage 3
// BVH2 nodes: n leaves (0..n-1, leaf j = the j-th primitive in Morton order)
// then n-1 internal nodes.  child.x = left (-1 for a leaf), child.y = right
// (the primitive id for a leaf).
__global__ void k_leaves(const float *__restrict__ boxes, const uint32_t *__restrict__ sorted_prim, uint32_t n,
    float *__restrict__ nbox, int2 *__restrict__ nchild, uint32_t *__restrict__ cid, float *__restrict__ cbox)
{
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const uint32_t p = sorted_prim[j];
    for (int k = 0; k < 6; ++k) {
      const float b = boxes[6 * size_t(p) + k];
      nbox[6 * size_t(j) + k] = b;
      cbox[6 * size_t(j) + k] = b;
    }
    nchild[j] = make_int2(-1, int(p));
    cid[j] = j;
  }
}

// The whole clustering in one cooperative launch: 45-58 iterations of mostly a
// few hundred clusters each, which as launches of their own (ten, and a read of
// two counters) take 2.4 ms for 50K triangles, in whole builds of 4.6 and 1.5 ms.  An
// iteration is three phases between grid barriers (neighbours; merges and
// survivors counted per block; ranks and output), and once the clusters fit
// one block (PLOC_ALONE), it goes on alone with them in shared memory.  The
// surface-area program of the nodes an iteration made runs with the next
// one's neighbour search (their children are older, so their entries are
// final).  Measured whole builds (968 / 63,368 triangles): blocks of 256, 512 and
// 1024 threads within 5% of one another, 512 with two per SM the fastest.  Ranks
// are exact integer prefix sums in cluster order, so the tree and its numbering
// do not depend on the grid.
constexpr int PLOC_BLOCK = 512;
constexpr int PLOC_BLOCKS_PER_SM = 2;
constexpr uint32_t PLOC_ALONE = PLOC_BLOCK;

struct PlocJob {
  uint32_t n;
  uint32_t *cid[2];        // clusters in Morton order: binary node
  float *cbox[2];          // and box
  uint32_t *nn;            // nearest neighbour of each cluster
  unsigned long long *sums; // per block: survivors << 32 | merges of its clusters
  float *nbox;
  int2 *nchild;
  CollapseDp dp;           // dp.cost null: no surface-area program
  float tri_cost;
  int max_leaf;
  uint32_t *result;        // [0] 1: no progress, [1] root, [2] inner nodes made
};

// Exclusive prefix sum of x over the block in thread order; total = the sum.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long x, unsigned long long &total)
{
  __shared__ unsigned long long warp_sum[PLOC_BLOCK / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned long long inc = x;
  for (uint32_t off = 1; off < 32u; off <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= off)
      inc += y;
  }
  if (lane == 31u)
    warp_sum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    unsigned long long w = lane < PLOC_BLOCK / 32 ? warp_sum[lane] : 0ull;
    for (uint32_t off = 1; off < 32u; off <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off)
        w += y;
    }
    if (lane < PLOC_BLOCK / 32)
      warp_sum[lane] = w;
  }
  __syncthreads();
  total = warp_sum[PLOC_BLOCK / 32 - 1];
  const unsigned long long before = warp ? warp_sum[warp - 1] : 0ull;
  __syncthreads(); // warp_sum is reused by the next call
  return before + inc - x;
}

// Survivors << 32 | merges of cluster i: it merges when it and its neighbour
// chose one another and it is the smaller index, and survives unless it is the
// larger one of such a pair.
__device__ __forceinline__ unsigned long long ploc_flags(const uint32_t *nn, uint32_t i, uint32_t &j)
{
  j = nn[i];
  const bool mutual = j != i && nn[j] == i;
  return (mutual && i < j ? 1ull : 0ull) | (mutual && i > j ? 0ull : 1ull << 32);
}

// The nearest neighbour of cluster i of `count`, whose box is me[0] and its
// neighbours' boxes lie around it; the pair order is (merged area, smaller
// index, larger index): scanning j upward, a strict < keeps the smaller partner
// index on ties, and the other keys are i's own.
template <int RADIUS>
__device__ __forceinline__ uint32_t ploc_nearest(const float (*me)[6], int i, int count)
{
  float best = 3.4e38f;
  int bj = i;
  const int j0 = max(0, i - RADIUS), j1 = min(count - 1, i + RADIUS);
  for (int j = j0; j <= j1; ++j) {
    if (j == i)
      continue;
    const float *m = me[0], *o = me[j - i];
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
      lo[k] = fminf(m[k], o[k]);
      hi[k] = fmaxf(m[3 + k], o[3 + k]);
    }
    const float a = area(lo, hi);
    if (a < best) {
      best = a;
      bj = j;
    }
  }
  return uint32_t(bj);
}

template <int RADIUS>
__global__ void __launch_bounds__(PLOC_BLOCK) k_ploc(PlocJob job)
{
  __shared__ float sb[PLOC_BLOCK + 2 * RADIUS][6];
  __shared__ uint32_t s_nn[PLOC_BLOCK], s_id[PLOC_BLOCK];
  const uint32_t blocks = gridDim.x, blk = blockIdx.x, tid = threadIdx.x;
  auto barrier = [] { cooperative_groups::this_grid().sync(); };
  uint32_t count = job.n, made = job.n, program_lo = job.n; // inner nodes so far end at `made`
  int c = 0;
  // the surface-area program of the nodes made since the last call, by this
  // block's threads from the last one down (the first ones have clusters)
  auto program = [&](uint32_t b, uint32_t of) {
    if (job.dp.cost)
      for (uint32_t v = program_lo + b * PLOC_BLOCK + (PLOC_BLOCK - 1 - tid); v < made; v += of * PLOC_BLOCK)
        collapse_dp_node(job.dp, job.nbox, job.nchild, job.n, v, job.tri_cost, job.max_leaf);
    program_lo = made;
  };
  while (count > PLOC_ALONE) { // the same count in every block
    program(blk, blocks);
    const float *cbox = job.cbox[c];
    for (uint32_t base = blk * PLOC_BLOCK; base < count; base += blocks * PLOC_BLOCK) {
      for (int t = tid; t < PLOC_BLOCK + 2 * RADIUS; t += PLOC_BLOCK) {
        const int g = int(base) - RADIUS + t;
        for (int k = 0; k < 6; ++k)
          sb[t][k] = (g >= 0 && g < int(count)) ? cbox[6 * size_t(g) + k] : 0.f;
      }
      __syncthreads();
      if (base + tid < count)
        job.nn[base + tid] = ploc_nearest<RADIUS>(&sb[tid + RADIUS], int(base + tid), int(count));
      __syncthreads();
    }
    barrier();
    // each block's consecutive clusters: how many merge and how many survive
    const uint32_t tiles = (count + PLOC_BLOCK - 1) / PLOC_BLOCK;
    const uint32_t seg = (tiles + blocks - 1) / blocks * PLOC_BLOCK;
    const uint32_t lo = min(count, blk * seg), hi = min(count, lo + seg);
    unsigned long long sum = 0, total;
    uint32_t j;
    for (uint32_t i = lo + tid; i < hi; i += PLOC_BLOCK)
      sum += ploc_flags(job.nn, i, j);
    block_scan(sum, total);
    if (tid == 0)
      job.sums[blk] = total;
    barrier();
    unsigned long long before = 0, all = 0;
    for (uint32_t b = tid; b < blocks; b += PLOC_BLOCK) {
      const unsigned long long x = job.sums[b];
      all += x;
      before += b < blk ? x : 0ull;
    }
    unsigned long long base_rank, t2;
    block_scan(before, base_rank);
    block_scan(all, t2);
    all = t2;
    const uint32_t merges = uint32_t(all), kept = uint32_t(all >> 32);
    if (merges == 0 || kept >= count) { // the same sums in every block
      if (blk == 0 && tid == 0)
        job.result[0] = 1u;
      return;
    }
    // survivors in order, merged pairs as new nodes
    for (uint32_t i0 = lo; i0 < hi; i0 += PLOC_BLOCK) {
      const uint32_t i = i0 + tid;
      const unsigned long long f = i < hi ? ploc_flags(job.nn, i, j) : 0ull;
      const unsigned long long rank = base_rank + block_scan(f, t2);
      base_rank += t2;
      if (f >> 32) {
        const uint32_t dst = uint32_t(rank >> 32);
        const float *bi = job.cbox[c] + 6 * size_t(i);
        float *bo = job.cbox[c ^ 1] + 6 * size_t(dst);
        if (uint32_t(f)) {
          const uint32_t node = made + uint32_t(rank);
          const float *bj = job.cbox[c] + 6 * size_t(j);
          float *bn = job.nbox + 6 * size_t(node);
          for (int k = 0; k < 3; ++k) {
            bn[k] = bo[k] = fminf(bi[k], bj[k]);
            bn[3 + k] = bo[3 + k] = fmaxf(bi[3 + k], bj[3 + k]);
          }
          job.nchild[node] = make_int2(int(job.cid[c][i]), int(job.cid[c][j]));
          job.cid[c ^ 1][dst] = node;
        } else {
          for (int k = 0; k < 6; ++k)
            bo[k] = bi[k];
          job.cid[c ^ 1][dst] = job.cid[c][i];
        }
      }
    }
    made += merges;
    count = kept;
    c ^= 1;
    barrier();
  }
  if (blk != 0)
    return;
  // the rest in one block: thread i's cluster in sb[RADIUS + i], s_id[i]
  if (tid < count) {
    s_id[tid] = job.cid[c][tid];
    for (int k = 0; k < 6; ++k)
      sb[RADIUS + tid][k] = job.cbox[c][6 * size_t(tid) + k];
  }
  __syncthreads();
  while (count > 1) {
    program(0u, 1u);
    if (tid < count)
      s_nn[tid] = ploc_nearest<RADIUS>(&sb[tid + RADIUS], int(tid), int(count));
    __syncthreads();
    uint32_t j = 0;
    unsigned long long f = 0, total;
    float box[6];
    uint32_t id = 0, id2 = 0;
    if (tid < count) {
      f = ploc_flags(s_nn, tid, j);
      id = s_id[tid];
      for (int k = 0; k < 6; ++k)
        box[k] = sb[RADIUS + tid][k];
      if (uint32_t(f)) {
        id2 = s_id[j];
        for (int k = 0; k < 3; ++k) {
          box[k] = fminf(box[k], sb[RADIUS + j][k]);
          box[3 + k] = fmaxf(box[3 + k], sb[RADIUS + j][3 + k]);
        }
      }
    }
    const unsigned long long rank = block_scan(f, total); // (a barrier: every box is read)
    const uint32_t merges = uint32_t(total), kept = uint32_t(total >> 32);
    if (merges == 0 || kept >= count) {
      if (tid == 0)
        job.result[0] = 1u;
      return;
    }
    if (f >> 32) {
      const uint32_t dst = uint32_t(rank >> 32);
      if (uint32_t(f)) {
        const uint32_t node = made + uint32_t(rank);
        for (int k = 0; k < 6; ++k)
          job.nbox[6 * size_t(node) + k] = box[k];
        job.nchild[node] = make_int2(int(id), int(id2));
        id = node;
      }
      s_id[dst] = id;
      for (int k = 0; k < 6; ++k)
        sb[RADIUS + dst][k] = box[k];
    }
    made += merges;
    count = kept;
    __syncthreads();
  }
  program(0u, 1u);
  if (tid == 0) {
    job.result[1] = s_id[0];
    job.result[2] = made - job.n;
  }
}

// ---------------------------------------------------------------- stage 4
struct Collapse {
  const float *nbox;   // BVH2 boxes
  const int2 *nchild;  // BVH2 children
  const float4 *pos;
  const uint4 *vidx;
  uint32_t *nodes;     // 20 words per BVH8 node
  float4 *tris;        // 3 per triangle record
  uint32_t *counters;  // [0] nodes, [1] triangle records, [2] next queue length, [3] overflow
  uint32_t node_cap;
  int max_leaf;        // triangles per leaf child (1..3)
};

// The primitives of BVH2 subtree v when it has at most `limit` leaves (at
// most 3): their count, with the primitives in `prims` in left-to-right
// order; limit + 1 when it has more.
__device__ int subtree_prims(const int2 *__restrict__ nchild, int v, int limit, int *prims)
{
  int stack[4], sp = 0, n = 0;
  stack[sp++] = v;
  while (sp > 0) {
    const int u = stack[--sp];
    const int2 c = nchild[u];
    if (c.x < 0) {
      if (n == limit)
        return limit + 1;
      prims[n++] = c.y;
    } else {
      if (sp + 2 > 4)
        return limit + 1;
      stack[sp++] = c.y;
      stack[sp++] = c.x;
    }
  }
  return n;
}

__device__ __forceinline__ float node_area(const float *nbox, int v)
{
  const float *b = nbox + 6 * size_t(v);
  return area(b, b + 3);
}

// One BVH8 node per thread: queue entries (BVH8 node index, BVH2 root).
__global__ void __launch_bounds__(128) k_collapse(Collapse c, const uint2 *__restrict__ qin, uint32_t nq,
    uint2 *__restrict__ qout)
{
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq)
    return;
  const uint32_t ni = qin[t].x;
  const int root = int(qin[t].y);
  // candidates: child v, whether it is internal, its area, and whether it
  // has at most max_leaf primitives (it becomes one leaf child unless a free
  // slot opens it), each found once when the candidate is added
  int ch[8];
  bool inner[8], sm[8];
  float ar[8];
  int prims[3];
  int k = 0;
  auto add = [&](int slot, int v) {
    ch[slot] = v;
    inner[slot] = c.nchild[v].x >= 0;
    ar[slot] = inner[slot] ? node_area(c.nbox, v) : 0.f;
    sm[slot] = inner[slot] && c.max_leaf > 1 && subtree_prims(c.nchild, v, c.max_leaf, prims) <= c.max_leaf;
  };
  if (c.nchild[root].x < 0) {
    add(k++, root); // a leaf root: one leaf child
  } else {
    add(k++, c.nchild[root].x);
    add(k++, c.nchild[root].y);
  }
  while (k < 8) { // open the internal child of largest area, larger subtrees first
    int best = -1;
    for (int i = 0; i < k; ++i)
      if (inner[i] && (best < 0 || (sm[best] && !sm[i]) || (sm[i] == sm[best] && ar[i] > ar[best])))
        best = i;
    if (best < 0)
      break;
    const int2 cc = c.nchild[ch[best]];
    add(best, cc.x);
    add(k++, cc.y);
  }
  float nlo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, nhi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
  for (int i = 0; i < k; ++i)
    for (int a = 0; a < 3; ++a) {
      nlo[a] = fminf(nlo[a], c.nbox[6 * size_t(ch[i]) + a]);
      nhi[a] = fmaxf(nhi[a], c.nbox[6 * size_t(ch[i]) + 3 + a]);
    }
  // octant slots, greedily by the smallest cost (the host builder's rule)
  float pc[3];
  for (int a = 0; a < 3; ++a)
    pc[a] = 0.5f * (nlo[a] + nhi[a]);
  float cost[8][8];
  for (int i = 0; i < k; ++i) {
    float cc[3];
    for (int a = 0; a < 3; ++a)
      cc[a] = 0.5f * (c.nbox[6 * size_t(ch[i]) + a] + c.nbox[6 * size_t(ch[i]) + 3 + a]) - pc[a];
    for (int s = 0; s < 8; ++s) {
      const float dx = (s & 4) ? -1.f : 1.f, dy = (s & 2) ? -1.f : 1.f, dz = (s & 1) ? -1.f : 1.f;
      cost[i][s] = cc[0] * dx + cc[1] * dy + cc[2] * dz;
    }
  }
  int child_at[8];
  for (int s = 0; s < 8; ++s)
    child_at[s] = -1;
  uint32_t used_c = 0u, used_s = 0u;
  for (int it = 0; it < k; ++it) {
    float best = 3.4e38f;
    int bc = -1, bs = -1;
    for (int i = 0; i < k; ++i) {
      if (used_c & (1u << i))
        continue;
      for (int s = 0; s < 8; ++s) {
        if (used_s & (1u << s))
          continue;
        if (cost[i][s] < best || bc < 0) {
          best = cost[i][s];
          bc = i;
          bs = s;
        }
      }
    }
    used_c |= 1u << bc;
    used_s |= 1u << bs;
    child_at[bs] = ch[bc];
  }
  // quantisation grid (double, exact powers of two: outward rounding)
  uint8_t e[3];
  double scale[3];
  for (int a = 0; a < 3; ++a) {
    const double ext = double(nhi[a]) - double(nlo[a]);
    int ex = -127;
    if (ext > 0.0) {
      ex = int(ceil(log2(ext / 255.0)));
      while (ldexp(255.0, ex) < ext)
        ++ex;
      while (ex > -127 && ldexp(255.0, ex - 1) >= ext)
        --ex;
    }
    ex = min(max(ex, -127), 127);
    e[a] = uint8_t(ex + 127);
    scale[a] = ex == -127 ? 0.0 : ldexp(1.0, ex);
  }
  // leaf children: single primitives, and internal children of at most
  // max_leaf primitives (lcount[s] primitives each)
  uint32_t internal = 0, leaves = 0;
  uint8_t imask = 0;
  int lcount[8];
  for (int s = 0; s < 8; ++s) {
    lcount[s] = 0;
    if (child_at[s] < 0)
      continue;
    const int v = child_at[s];
    if (c.nchild[v].x < 0)
      lcount[s] = 1;
    else if (c.max_leaf > 1) {
      const int m = subtree_prims(c.nchild, v, c.max_leaf, prims);
      lcount[s] = m <= c.max_leaf ? m : 0;
    }
    if (lcount[s] == 0) {
      imask |= uint8_t(1u << s);
      ++internal;
    } else {
      leaves += uint32_t(lcount[s]);
    }
  }
  uint32_t child_base = 0, tri_base = 0;
  if (internal)
    child_base = atomicAdd(&c.counters[0], internal);
  if (leaves)
    tri_base = atomicAdd(&c.counters[1], leaves);
  if (child_base + internal > c.node_cap) {
    atomicExch(&c.counters[3], 1u);
    return;
  }
  uint32_t q_out_base = 0;
  if (internal)
    q_out_base = atomicAdd(&c.counters[2], internal);
  uint8_t meta[8] = {}, q[6][8] = {};
  uint32_t next_child = child_base, tri_off = 0, qo = q_out_base;
  for (int s = 0; s < 8; ++s) {
    const int v = child_at[s];
    if (v < 0)
      continue;
    const float *b = c.nbox + 6 * size_t(v);
    for (int a = 0; a < 3; ++a) {
      double lo = 0.0, hi = 0.0;
      if (scale[a] > 0.0) {
        lo = floor((double(b[a]) - double(nlo[a])) / scale[a]);
        hi = ceil((double(b[3 + a]) - double(nlo[a])) / scale[a]);
      }
      q[a][s] = uint8_t(fmin(fmax(lo, 0.0), 255.0));
      q[3 + a][s] = uint8_t(fmin(fmax(hi, 0.0), 255.0));
    }
    if (lcount[s] == 0) {
      meta[s] = 0x80;
      qout[qo++] = make_uint2(next_child++, uint32_t(v));
    } else {
      meta[s] = uint8_t((uint32_t(lcount[s]) << 5) | tri_off);
      if (c.nchild[v].x < 0)
        prims[0] = c.nchild[v].y;
      else
        subtree_prims(c.nchild, v, c.max_leaf, prims);
      for (int j = 0; j < lcount[s]; ++j) {
        const uint32_t prim = uint32_t(prims[j]);
        const uint4 vi = c.vidx[prim];
        const float4 v0 = c.pos[vi.x], v1 = c.pos[vi.y], v2 = c.pos[vi.z];
        float4 *r = c.tris + 3 * size_t(tri_base + tri_off);
        r[0] = make_float4(v0.x, v0.y, v0.z, __uint_as_float(prim));
        r[1] = make_float4(v1.x - v0.x, v1.y - v0.y, v1.z - v0.z, 0.f);
        r[2] = make_float4(v2.x - v0.x, v2.y - v0.y, v2.z - v0.z, 0.f);
        ++tri_off;
      }
    }
  }
  uint32_t *w = c.nodes + size_t(ni) * 20;
  w[0] = __float_as_uint(nlo[0]);
  w[1] = __float_as_uint(nlo[1]);
  w[2] = __float_as_uint(nlo[2]);
  w[3] = uint32_t(e[0]) | (uint32_t(e[1]) << 8) | (uint32_t(e[2]) << 16) | (uint32_t(imask) << 24);
  w[4] = child_base;
  w[5] = tri_base;
  w[6] = uint32_t(meta[0]) | (uint32_t(meta[1]) << 8) | (uint32_t(meta[2]) << 16) | (uint32_t(meta[3]) << 24);
  w[7] = uint32_t(meta[4]) | (uint32_t(meta[5]) << 8) | (uint32_t(meta[6]) << 16) | (uint32_t(meta[7]) << 24);
  for (int r = 0; r < 6; ++r) {
    w[8 + 2 * r] = uint32_t(q[r][0]) | (uint32_t(q[r][1]) << 8) | (uint32_t(q[r][2]) << 16) |
        (uint32_t(q[r][3]) << 24);
    w[9 + 2 * r] = uint32_t(q[r][4]) | (uint32_t(q[r][5]) << 8) | (uint32_t(q[r][6]) << 16) |
        (uint32_t(q[r][7]) << 24);
  }
}

// ---------------------------------------------------------------- stage 4a
// The collapse by the surface-area program (bvh_collapse.cuh): every level of
// the wide tree in one cooperative launch, eight lanes per wide node, which
// hold one child, then one slot, each (the octant slots are a greedy choice
// among 64 costs, then come 48 quantised planes).  A level takes about 15 us;
// with one thread per node and a launch and counter read per level it takes
// 60-100 us however few nodes it has.
struct CollapseSah {
  const uint8_t *split; // CollapseDp::split
  const uchar4 *info;   // CollapseDp::info
  uint32_t n;           // primitives (the binary leaves 0..n-1)
  int *leaf_node;       // per triangle record (k_leaf_records)
};
constexpr int COLLAPSE_BLOCK = 128;
constexpr uint32_t COLLAPSE_LEVELS = 1000; // deeper trees are refused

// One wide node over binary node `root` (queue entry (ni, root)) by the 8 lanes
// of a group, as k_collapse's: its children from sah_children, octant slots,
// quantised child boxes, leaf records and the queue entries of its inner
// children.  All lanes of the warp call it; `live`: the group has a node.
// ch, lc: the group's scratch in shared memory.
__device__ void sah_wide_node(const Collapse &c, const CollapseSah &p, bool live, uint32_t ni, int root, int *ch,
    int *lc, uint2 *qout, uint32_t *qlen)
{
  constexpr uint32_t FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, g = lane & 7u, shift = lane & 24u;
  // the children the program chose: an entry (subtree, slots) sits in the lane
  // of its first slot, the root's two subtrees share the 8, and opening one
  // for its slots splits them between its own two subtrees (sah_children's
  // rule; lane order is its order)
  const bool leaf_root = live && uint32_t(root) < p.n; // one leaf child
  int u = -1, slots = 0;
  if (live) {
    int s0 = 8;
    int2 cr = make_int2(root, -1);
    if (!leaf_root) {
      s0 = int(p.info[uint32_t(root) - p.n].x);
      s0 = s0 < 1 ? 1 : (s0 > 7 ? 7 : s0);
      cr = c.nchild[root];
    }
    if (g == 0 || int(g) == s0) {
      u = g == 0 ? cr.x : cr.y;
      slots = g == 0 ? s0 : 8 - s0;
    }
  }
  for (bool more = !leaf_root; __any_sync(FULL, more);) {
    int open = 0, right = -1;
    if (more && u >= 0 && slots >= 2 && uint32_t(u) >= p.n) {
      const int2 cu = c.nchild[u]; // (beside the split, not after it)
      open = int(p.split[8 * size_t(uint32_t(u) - p.n) + size_t(slots - 1)]);
      if (open >= 1 && open < slots) {
        right = cu.y;
        u = cu.x;
      } else {
        open = 0;
      }
    }
    more = open != 0;
    ch[g] = -1;
    __syncwarp();
    if (more) { // the right subtree's entry, in the lane of its first slot
      ch[g + uint32_t(open)] = right;
      lc[g + uint32_t(open)] = slots - open;
      slots = open;
    }
    __syncwarp();
    if (ch[g] >= 0) {
      u = ch[g];
      slots = lc[g];
      more = true;
    }
    __syncwarp();
  }
  const uint32_t have = (__ballot_sync(FULL, u >= 0) >> shift) & 0xffu;
  const int k = __popc(have);
  if (u >= 0) {
    const int i = __popc(have & ((1u << g) - 1u));
    int prim = 1;
    if (uint32_t(u) >= p.n) {
      const uchar4 in = p.info[uint32_t(u) - p.n];
      prim = in.y ? int(in.z) : 0;
    }
    ch[i] = u;
    lc[i] = prim;
  }
  __syncwarp();
  // as child g: its box, the node's bounds
  const bool child = live && int(g) < k;
  float b[6], nlo[3], nhi[3];
  for (int a = 0; a < 3; ++a) {
    b[a] = child ? c.nbox[6 * size_t(ch[g]) + a] : 3.4e38f;
    b[3 + a] = child ? c.nbox[6 * size_t(ch[g]) + 3 + a] : -3.4e38f;
    nlo[a] = b[a];
    nhi[a] = b[3 + a];
    for (int off = 1; off < 8; off <<= 1) {
      nlo[a] = fminf(nlo[a], __shfl_xor_sync(FULL, nlo[a], off));
      nhi[a] = fmaxf(nhi[a], __shfl_xor_sync(FULL, nhi[a], off));
    }
  }
  // octant slots, greedily by the smallest cost, then the smallest child and
  // slot (the host builder's rule)
  float cost[8];
  {
    float cc[3];
    for (int a = 0; a < 3; ++a)
      cc[a] = 0.5f * (b[a] + b[3 + a]) - 0.5f * (nlo[a] + nhi[a]);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const float dx = (s & 4) ? -1.f : 1.f, dy = (s & 2) ? -1.f : 1.f, dz = (s & 1) ? -1.f : 1.f;
      const float x = cc[0] * dx + cc[1] * dy + cc[2] * dz;
      cost[s] = x < 3.4e38f ? x : 3.4e38f; // (and NaN, so that the lanes agree on an order)
    }
  }
  uint32_t used = 0u, at = 0u; // slots taken; per slot its child + 1 (4 bits each)
  bool placed = !child;
  for (int it = 0; it < 8; ++it) {
    float best = 3.4e38f;
    uint32_t key = 64u; // child * 8 + slot of the best pair
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (!placed && !(used & (1u << s)) && (key == 64u || cost[s] < best)) {
        best = cost[s];
        key = g * 8u + uint32_t(s);
      }
    for (int off = 1; off < 8; off <<= 1) {
      const float ob = __shfl_xor_sync(FULL, best, off);
      const uint32_t ok = __shfl_xor_sync(FULL, key, off);
      if (ok != 64u && (key == 64u || ob < best || (ob == best && ok < key))) {
        best = ob;
        key = ok;
      }
    }
    if (key != 64u) {
      used |= 1u << (key & 7u);
      at |= ((key >> 3) + 1u) << (4u * (key & 7u));
      placed = placed || (key >> 3) == g;
    }
  }
  // quantisation grid (double, exact powers of two: outward rounding); lane a
  // finds axis a's exponent
  int ex = -127;
  {
    const float l = g == 0 ? nlo[0] : (g == 1 ? nlo[1] : nlo[2]), h = g == 0 ? nhi[0] : (g == 1 ? nhi[1] : nhi[2]);
    const double ext = double(h) - double(l);
    // the least ex with 255 x 2^ex >= ext = m x 2^e, 1 <= m < 2: e - 7, or one
    // more when m > 255 / 128
    if (g < 3u && live && ext > 0.0) {
      const long long bits = __double_as_longlong(ext);
      ex = int(bits >> 52) - 1023 - 7 + ((bits & 0xfffffffffffffll) > 0xfe00000000000ll ? 1 : 0);
    }
    ex = min(max(ex, -127), 127);
  }
  uint32_t ebits = 0u;
  double per_cell[3]; // 1 / cell, a power of two: the product is the quotient
  for (int a = 0; a < 3; ++a) {
    const int e = __shfl_sync(FULL, ex, a, 8);
    ebits |= uint32_t(e + 127) << (8 * a);
    per_cell[a] = e == -127 ? 0.0 : __longlong_as_double((long long)(1023 - e) << 52);
  }
  // from here on as slot g: the child in it, if any
  const uint32_t cand = (at >> (4u * g)) & 15u;
  const bool filled = live && cand != 0u;
  const int from = filled ? int(cand) - 1 : 0;
  const int v = filled ? ch[from] : 0, leaf = filled ? lc[from] : 0;
  for (int a = 0; a < 6; ++a)
    b[a] = __shfl_sync(FULL, b[a], from, 8);
  const uint32_t imask = (__ballot_sync(FULL, filled && leaf == 0) >> shift) & 0xffu;
  const uint32_t internal = uint32_t(__popc(imask)), rank = uint32_t(__popc(imask & ((1u << g) - 1u)));
  uint32_t tri_end = uint32_t(leaf);
  for (int off = 1; off < 8; off <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, tri_end, off, 8);
    if (int(g) >= off)
      tri_end += y;
  }
  const uint32_t tri_off = tri_end - uint32_t(leaf), leaves = __shfl_sync(FULL, tri_end, 7, 8);
  uint32_t child_base = 0, tri_base = 0, q_base = 0, room = 1u;
  if (live && g == 0) {
    if (internal)
      child_base = atomicAdd(&c.counters[0], internal);
    if (leaves)
      tri_base = atomicAdd(&c.counters[1], leaves);
    if (child_base + internal > c.node_cap) {
      atomicExch(&c.counters[3], 1u);
      room = 0u;
    } else if (internal) {
      q_base = atomicAdd(qlen, internal);
    }
  }
  child_base = __shfl_sync(FULL, child_base, 0, 8);
  tri_base = __shfl_sync(FULL, tri_base, 0, 8);
  q_base = __shfl_sync(FULL, q_base, 0, 8);
  room = __shfl_sync(FULL, room, 0, 8);
  if (!live || !room)
    return;
  uint32_t *w = c.nodes + size_t(ni) * 20;
  if (g < 3u)
    w[g] = __float_as_uint(g == 0 ? nlo[0] : (g == 1 ? nlo[1] : nlo[2]));
  else if (g < 6u)
    w[g] = g == 3u ? (ebits | (imask << 24)) : (g == 4u ? child_base : tri_base);
  // bytes of slot g: its meta byte, then its planes (low x, y, z, high x, y, z)
  uint8_t *bytes = reinterpret_cast<uint8_t *>(w) + 24 + g;
  bytes[0] = filled ? (leaf == 0 ? uint8_t(0x80) : uint8_t((uint32_t(leaf) << 5) | tri_off)) : uint8_t(0);
  for (int a = 0; a < 3; ++a) {
    double lo = 0.0, hi = 0.0;
    if (filled && per_cell[a] > 0.0) {
      lo = floor((double(b[a]) - double(nlo[a])) * per_cell[a]);
      hi = ceil((double(b[3 + a]) - double(nlo[a])) * per_cell[a]);
    }
    bytes[8 * (1 + a)] = uint8_t(fmin(fmax(lo, 0.0), 255.0));
    bytes[8 * (4 + a)] = uint8_t(fmin(fmax(hi, 0.0), 255.0));
  }
  if (!filled)
    return;
  if (leaf == 0) {
    qout[q_base + rank] = make_uint2(child_base + rank, uint32_t(v));
    return;
  }
  // its records are k_leaf_records' work, off the levels' chain
  for (int j = 0; j < leaf; ++j)
    p.leaf_node[tri_base + tri_off + uint32_t(j)] = j == 0 ? v : -1;
}

// The records of the leaf children: leaf_node[r] is the binary node of the leaf
// child whose first record is r, -1 elsewhere.
__global__ void __launch_bounds__(256) k_leaf_records(Collapse c, const int *__restrict__ leaf_node, uint32_t n)
{
  const uint32_t r0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = r0 < n ? leaf_node[r0] : -1;
  if (v < 0)
    return;
  int prims[3];
  int m = 1;
  if (c.nchild[v].x < 0)
    prims[0] = c.nchild[v].y;
  else
    m = subtree_prims(c.nchild, v, c.max_leaf, prims);
  if (m > c.max_leaf || (r0 + uint32_t(m) < n && leaf_node[r0 + uint32_t(m)] < 0) || r0 + uint32_t(m) > n) {
    atomicExch(&c.counters[3], 2u); // cannot happen: the leaf has another size than its slots
    return;
  }
  for (int j = 0; j < m; ++j) {
    const uint32_t prim = uint32_t(prims[j]);
    const uint4 vi = c.vidx[prim];
    const float4 v0 = c.pos[vi.x], v1 = c.pos[vi.y], v2 = c.pos[vi.z];
    float4 *r = c.tris + 3 * size_t(r0 + uint32_t(j));
    r[0] = make_float4(v0.x, v0.y, v0.z, __uint_as_float(prim));
    r[1] = make_float4(v1.x - v0.x, v1.y - v0.y, v1.z - v0.z, 0.f);
    r[2] = make_float4(v2.x - v0.x, v2.y - v0.y, v2.z - v0.z, 0.f);
  }
}

// The triangle records by primitive, for shading (build_prim_records of the
// host build).
__global__ void __launch_bounds__(256) k_prim_records(const float4 *__restrict__ pos, const uint4 *__restrict__ vidx,
    uint32_t n, float4 *__restrict__ geo)
{
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 vi = vidx[i];
    const float4 v0 = pos[vi.x], v1 = pos[vi.y], v2 = pos[vi.z];
    float4 *r = geo + 3 * size_t(i);
    r[0] = make_float4(v0.x, v0.y, v0.z, __uint_as_float(i));
    r[1] = make_float4(v1.x - v0.x, v1.y - v0.y, v1.z - v0.z, 0.f);
    r[2] = make_float4(v2.x - v0.x, v2.y - v0.y, v2.z - v0.z, 0.f);
  }
}

// counters: [0] nodes, [1] triangle records, [3] error, [4..6] lengths of the
// level's, the next and the one after's queue, in turn ([4] starts at 1, the
// root's entry in q0), [7] levels.  Every block reads the same length after a
// barrier; an error only ends the queues, so the blocks leave together.
__global__ void __launch_bounds__(COLLAPSE_BLOCK) k_collapse_sah(Collapse c, CollapseSah p, uint2 *q0, uint2 *q1)
{
  __shared__ int ch[COLLAPSE_BLOCK], lc[COLLAPSE_BLOCK];
  const uint32_t group = threadIdx.x & ~7u;
  const uint32_t warp = (blockIdx.x * COLLAPSE_BLOCK + threadIdx.x) >> 5, warps = gridDim.x * (COLLAPSE_BLOCK / 32);
  uint32_t level = 0;
  for (; level < COLLAPSE_LEVELS; ++level) {
    const uint32_t nq = c.counters[4 + level % 3];
    if (nq == 0)
      break;
    if (blockIdx.x == 0 && threadIdx.x == 0)
      c.counters[4 + (level + 2) % 3] = 0u; // the queue after the next
    const uint2 *qin = level & 1u ? q1 : q0;
    uint2 *qout = level & 1u ? q0 : q1;
    for (uint32_t base = warp * 4u; base < nq; base += warps * 4u) {
      const uint32_t e = base + ((threadIdx.x & 31u) >> 3);
      const uint2 entry = e < nq ? qin[e] : make_uint2(0u, 0u);
      sah_wide_node(c, p, e < nq, entry.x, int(entry.y), ch + group, lc + group, qout,
          &c.counters[4 + (level + 1) % 3]);
      __syncwarp();
    }
    cooperative_groups::this_grid().sync();
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    c.counters[7] = level;
}

struct DevBuf {
  void *p{nullptr};
  ~DevBuf()
  {
    if (p)
      cudaFree(p);
  }
  template <class T> T *as() { return static_cast<T *>(p); }
};

void ck(cudaError_t e, const char *what)
{
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("gpu bvh build: ") + what + ": " + cudaGetErrorString(e));
}

void alloc(DevBuf &b, size_t bytes, const char *what)
{
  ck(cudaMalloc(&b.p, bytes ? bytes : 16), what);
}

uint32_t grid_of(uint32_t n, uint32_t block) { return std::max<uint32_t>(1u, std::min<uint32_t>((n + block - 1) / block, 1u << 20)); }

} // namespace

size_t scan_u32_scratch(uint32_t n) { return (size_t(n) + SCAN_TILE - 1) / SCAN_TILE; }

void scan_u32(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *total, uint32_t *scratch, cudaStream_t s)
{
  if (n == 0)
    return;
  const uint32_t tiles = uint32_t(scan_u32_scratch(n));
  k_tile_sums<<<tiles, SCAN_T, 0, s>>>(in, n, scratch);
  k_scan_inplace<<<1, 1024, 0, s>>>(scratch, tiles, total);
  k_tile_scan<<<tiles, SCAN_T, 0, s>>>(in, n, scratch, out);
}

namespace {

// The device scratch of one build: one allocation, given back at its end.
struct Scratch {
  DevBuf buf;
  size_t used{0};
  std::vector<std::pair<void **, size_t>> parts;
  template <class T> void want(T *&p, size_t count)
  {
    parts.push_back({reinterpret_cast<void **>(&p), used});
    used += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
  }
  void allocate()
  {
    alloc(buf, used, "scratch");
    for (auto &p : parts)
      *p.first = buf.as<char>() + p.second;
  }
};

struct DeviceLimits {
  int sms{0}, ploc_blocks{0}, collapse_blocks{0};
};

// The clustering kernel of a search radius.
const void *ploc_kernel(int radius)
{
  return radius <= 2 ? (const void *)k_ploc<2>
      : radius <= 4  ? (const void *)k_ploc<4>
      : radius <= 8  ? (const void *)k_ploc<8>
      : radius <= 16 ? (const void *)k_ploc<16>
                     : (const void *)k_ploc<32>;
}

// Grid limits of the cooperative kernels on the current device: the clustering
// kernel that will be launched, and the collapse.
DeviceLimits device_limits(const void *ploc)
{
  DeviceLimits d;
  int dev = 0;
  ck(cudaGetDevice(&dev), "device");
  ck(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev), "device");
  ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.ploc_blocks, ploc, PLOC_BLOCK, 0), "occupancy");
  ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.collapse_blocks, k_collapse_sah, COLLAPSE_BLOCK, 0),
      "occupancy");
  return d;
}

} // namespace

GpuBvh8 build_bvh8_gpu(const float4 *positions, const uint4 *prim_vidx, uint32_t n, cudaStream_t s, int max_leaf,
    int radius, float tri_cost)
{
  if (n == 0)
    throw std::runtime_error("gpu bvh build: no triangles");
  if (n > (1u << 30))
    throw std::runtime_error("gpu bvh build: too many triangles");
  const void *ploc = ploc_kernel(radius);
  const DeviceLimits lim = device_limits(ploc);
  const uint32_t nb = (n + SORT_BLOCK - 1) / SORT_BLOCK;
  const uint32_t nodes2 = 2 * n - 1, inner = n - 1;
  const bool program = tri_cost > 0.f && inner > 0;
  const int leaf_max = std::min(std::max(max_leaf, 1), 3);
  const uint32_t ploc_blocks =
      n <= PLOC_ALONE ? 1u
                      : std::min<uint32_t>(uint32_t(lim.sms * std::min(std::max(lim.ploc_blocks, 1), PLOC_BLOCKS_PER_SM)),
                            (n + PLOC_BLOCK - 1) / PLOC_BLOCK);
  Scratch sc;
  float *boxes, *nbox;
  uint32_t *cb, *keys[2], *vals[2], *hist, *scan_tmp, *ctr, *nodes_big;
  int2 *nchild;
  uint2 *q[2];
  int *leaf_node;
  PlocJob job{};
  sc.want(boxes, size_t(n) * 6);
  sc.want(cb, 6);
  for (int k = 0; k < 2; ++k) {
    sc.want(keys[k], n);
    sc.want(vals[k], n);
  }
  sc.want(hist, size_t(nb) * 256);
  sc.want(scan_tmp, std::max(scan_u32_scratch(nb * 256), scan_u32_scratch(n)));
  sc.want(nbox, size_t(nodes2) * 6);
  sc.want(nchild, nodes2);
  for (int k = 0; k < 2; ++k) {
    sc.want(job.cid[k], n);
    sc.want(job.cbox[k], size_t(n) * 6);
    sc.want(q[k], n);
  }
  sc.want(job.nn, n);
  sc.want(job.sums, ploc_blocks);
  sc.want(job.result, 4);
  sc.want(ctr, 8);
  sc.want(leaf_node, n);
  if (program) {
    sc.want(job.dp.cost, size_t(inner) * 8);
    sc.want(job.dp.split, size_t(inner) * 8);
    sc.want(job.dp.info, inner);
  }
  // a BVH8 over n leaves with >= 2 children per inner node has fewer nodes
  sc.want(nodes_big, size_t(n) * 20);
  float4 *tris_big = nullptr; // the greedy collapse writes its records as it goes
  if (!program)
    sc.want(tris_big, size_t(n) * 3);
  sc.allocate();
  // scene centroid bounds start at (+max, -max) in the ordered encoding
  const uint32_t init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
  ck(cudaMemcpyAsync(cb, init, sizeof(init), cudaMemcpyHostToDevice, s), "bounds init");
  k_prim_boxes<<<grid_of(n, 256), 256, 0, s>>>(positions, prim_vidx, n, boxes, cb);
  k_morton<<<grid_of(n, 256), 256, 0, s>>>(boxes, n, cb, keys[0], vals[0]);
  int cur = 0;
  for (int shift = 0; shift < 32; shift += 8) {
    k_digit_hist<<<nb, SORT_BLOCK, 0, s>>>(keys[cur], n, shift, hist, nb);
    scan_u32(hist, hist, nb * 256, nullptr, scan_tmp, s);
    k_digit_scatter<<<nb, SORT_BLOCK, 0, s>>>(keys[cur], vals[cur], n, shift, hist, nb, keys[cur ^ 1],
        vals[cur ^ 1]);
    cur ^= 1;
  }

  // the binary tree, with the surface-area program of its nodes
  k_leaves<<<grid_of(n, 256), 256, 0, s>>>(boxes, vals[cur], n, nbox, nchild, job.cid[0], job.cbox[0]);
  job.n = n;
  job.nbox = nbox;
  job.nchild = nchild;
  job.tri_cost = tri_cost;
  job.max_leaf = leaf_max;
  ck(cudaMemsetAsync(job.result, 0, 16, s), "clustering result");
  {
    void *args[] = {&job};
    ck(cudaLaunchCooperativeKernel(ploc, dim3(ploc_blocks), dim3(PLOC_BLOCK), args, 0, s), "clustering launch");
  }
  uint32_t result[4];
  ck(cudaMemcpyAsync(result, job.result, 16, cudaMemcpyDeviceToHost, s), "read clustering");
  ck(cudaStreamSynchronize(s), "clustering");
  if (result[0] || result[2] != inner)
    throw std::runtime_error("gpu bvh build: clustering made no progress");

  // collapse into BVH8 nodes, level by level
  GpuBvh8 out;
  const uint32_t c0[8] = {1u, 0u, 0u, 0u, 1u, 0u, 0u, 0u};
  ck(cudaMemcpyAsync(ctr, c0, sizeof(c0), cudaMemcpyHostToDevice, s), "collapse counters");
  const uint2 first = make_uint2(0u, result[1]);
  ck(cudaMemcpyAsync(q[0], &first, sizeof(first), cudaMemcpyHostToDevice, s), "first queue entry");
  Collapse col{nbox, nchild, positions, prim_vidx, nodes_big, tris_big, ctr, n, leaf_max};
  uint32_t cc[8];
  auto read_counters = [&](const char *what) {
    ck(cudaMemcpyAsync(cc, ctr, sizeof(cc), cudaMemcpyDeviceToHost, s), "read collapse counters");
    ck(cudaStreamSynchronize(s), what);
    if (cc[3] == 2)
      throw std::runtime_error("gpu bvh build: the collapse's surface-area choices are inconsistent");
    if (cc[3])
      throw std::runtime_error("gpu bvh build: node capacity exceeded");
  };
  if (program) {
    CollapseSah sah{job.dp.split, job.dp.info, n, leaf_node};
    void *args[] = {&col, &sah, &q[0], &q[1]};
    // four blocks per SM: enough groups for the widest levels of a 500K-triangle
    // scene, and a cheaper barrier than with all that fit
    const uint32_t most = uint32_t(lim.sms) * uint32_t(std::min(std::max(lim.collapse_blocks, 1), 4));
    const uint32_t blocks = std::min<uint32_t>(most, (n + COLLAPSE_BLOCK / 8 - 1) / (COLLAPSE_BLOCK / 8));
    ck(cudaLaunchCooperativeKernel((const void *)k_collapse_sah, dim3(blocks), dim3(COLLAPSE_BLOCK), args, 0, s),
        "collapse launch");
    read_counters("collapse");
    if (cc[7] >= COLLAPSE_LEVELS)
      throw std::runtime_error("gpu bvh build: collapse did not end");
    out.max_depth = cc[7];
  } else {
    uint32_t nq = 1;
    int qc = 0;
    while (nq > 0) {
      if (++out.max_depth > COLLAPSE_LEVELS)
        throw std::runtime_error("gpu bvh build: collapse did not end");
      k_collapse<<<(nq + 127) / 128, 128, 0, s>>>(col, q[qc], nq, q[qc ^ 1]);
      ck(cudaGetLastError(), "collapse launch");
      read_counters("collapse level");
      nq = cc[2];
      const uint32_t zero = 0u;
      ck(cudaMemcpyAsync(ctr + 2, &zero, 4, cudaMemcpyHostToDevice, s), "reset queue length");
      qc ^= 1;
    }
  }
  out.node_count = out.node_cap = cc[0];
  out.tri_count = cc[1];
  if (out.tri_count != n)
    throw std::runtime_error("gpu bvh build: leaf records do not cover the triangles");
  // what the scene keeps, in one allocation: the nodes made (out of the
  // worst-case array) and the triangle records in leaf and in primitive order
  DevBuf keep; // owned here until the build succeeds
  const size_t node_bytes = (size_t(out.node_count) * 80 + 255) & ~size_t(255);
  out.bytes = node_bytes + size_t(n) * 96;
  alloc(keep, out.bytes, "bvh8");
  out.nodes = keep.p;
  out.tris = keep.as<char>() + node_bytes;
  out.geo = keep.as<char>() + node_bytes + size_t(n) * 48;
  ck(cudaMemcpyAsync(out.nodes, nodes_big, size_t(out.node_count) * 80, cudaMemcpyDeviceToDevice, s), "nodes");
  if (program) {
    col.tris = static_cast<float4 *>(out.tris);
    k_leaf_records<<<(n + 255) / 256, 256, 0, s>>>(col, leaf_node, n);
    ck(cudaGetLastError(), "leaf records launch");
  } else {
    ck(cudaMemcpyAsync(out.tris, tris_big, size_t(n) * 48, cudaMemcpyDeviceToDevice, s), "triangles");
  }
  k_prim_records<<<grid_of(n, 256), 256, 0, s>>>(positions, prim_vidx, n, static_cast<float4 *>(out.geo));
  ck(cudaGetLastError(), "primitive records launch");
  read_counters("bvh8 build"); // (the leaf records check their sizes)
  keep.p = nullptr; // ownership passes to the caller
  return out;
}

} // namespace phc
