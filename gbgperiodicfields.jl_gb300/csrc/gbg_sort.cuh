// The pieces of the stable counting sort that other kernels take along.
#pragma once

#include "gbg_common.cuh"

namespace gbg {

constexpr int kRsBins = 256;
constexpr int kRunThreads = 512, kRunWarps = kRunThreads / 32, kRunItems = 4, kRunTile = kRunThreads * kRunItems;

// Where a tile's items go when they are placed by digit, in their order within one: base[d] is the next free
// place of digit d, and is moved on.  Items of digit kRsBins go nowhere.  A warp's items are consecutive, 32 at
// a time; every thread of the CTA calls it, and may use wh again after it.
template <int WARPS, int ITEMS>
__device__ __forceinline__ void tile_places(const uint32_t (&digit)[ITEMS], uint32_t (&pos)[ITEMS],
                                            uint32_t (&wh)[WARPS][kRsBins], uint32_t *base) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lower = (1u << lane) - 1u;
  for (int k = threadIdx.x; k < WARPS * kRsBins; k += WARPS * 32) (&wh[0][0])[k] = 0u;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r)
    if (digit[r] < kRsBins) atomicAdd(&wh[warp][digit[r]], 1u);
  __syncthreads();
  if (threadIdx.x < kRsBins) {
    uint32_t run = base[threadIdx.x];
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t x = wh[w][threadIdx.x];
      wh[w][threadIdx.x] = run;
      run += x;
    }
    base[threadIdx.x] = run;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const bool valid = digit[r] < kRsBins;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit[r]);
    pos[r] = 0;
    if (valid) pos[r] = wh[warp][digit[r]] + __popc(peers & lower);
    __syncwarp();
    if (valid && lane == 31 - __clz(peers)) wh[warp][digit[r]] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
}

// The huge runs of a stable counting sort (stable_counting_sort), listed and counted by share but not yet placed;
// shares == 0 where the points are too few for any.
struct HugeRuns {
  const uint32_t *big = nullptr, *huge = nullptr, *keys = nullptr, *starts = nullptr, *id = nullptr;
  uint32_t *perm = nullptr;
  const float4 *rec_user = nullptr;
  float4 *rec = nullptr;
  int64_t n = 0;
  uint32_t limit = 0;
  const uint32_t *counts = nullptr;
  int shares = 0;
};

// The points of one of `shares` shares in the huge runs' placement: even, a whole number of tiles.
__device__ __forceinline__ int64_t huge_share(int64_t n, int64_t shares) {
  return ((n + shares - 1) / shares + kRunTile - 1) / kRunTile * kRunTile;
}
// The place of point p's run in the list of huge runs, or kRsBins.
__device__ __forceinline__ uint32_t huge_digit(const uint32_t *keys, const uint32_t *starts, const uint32_t *huge_id,
                                               int64_t p, uint32_t limit) {
  const uint32_t k = __ldg(keys + p), a = __ldg(starts + k);
  return __ldg(starts + k + 1) - a > limit ? huge_id[a] : (uint32_t)kRsBins;
}

// Places the huge runs, in a launch of kRunThreads threads a block: a block goes through a share of the points in
// their order and places those of huge runs behind the ones that earlier shares counted, all such runs at once
// (there are at most 254, `limit` being at least n / 255).  1e6 points of 1e7 in one cell: the bins built in 1.2
// ms, 7.7 with that cell sorted by one CTA.
__device__ __forceinline__ void place_huge(const HugeRuns &h) {
  if (h.shares == 0) return;
  const uint32_t nhuge = h.big[4];
  if (nhuge == 0u) return;
  __shared__ uint32_t wh[kRunWarps][kRsBins], base[kRsBins];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t size = huge_share(h.n, h.shares);
  for (int share = (int)blockIdx.x; share < h.shares; share += (int)gridDim.x) {
    __syncthreads();  // the previous share is placed
    if (threadIdx.x < nhuge) {
      uint32_t at = h.huge[threadIdx.x];
      for (int b = 0; b < share; ++b) at += h.counts[b * kRsBins + threadIdx.x];
      base[threadIdx.x] = at;
    }
    const int64_t from = share * size, to = min(h.n, from + size);
    for (int64_t t0 = from; t0 < to; t0 += kRunTile) {
      const int64_t seg = t0 + warp * (32 * kRunItems) + lane;
      uint32_t digit[kRunItems], pos[kRunItems];
      bool some = false;
#pragma unroll
      for (int r = 0; r < kRunItems; ++r) {
        digit[r] = seg + 32 * r < to ? huge_digit(h.keys, h.starts, h.id, seg + 32 * r, h.limit) : (uint32_t)kRsBins;
        some |= digit[r] < kRsBins;
      }
      if (!__syncthreads_or(some)) continue;
      tile_places<kRunWarps>(digit, pos, wh, base);
#pragma unroll
      for (int r = 0; r < kRunItems; ++r)
        if (digit[r] < kRsBins) {
          h.perm[pos[r]] = (uint32_t)(seg + 32 * r);
          if (h.rec) h.rec[pos[r]] = h.rec_user[seg + 32 * r];
        }
    }
  }
}

}  // namespace gbg
