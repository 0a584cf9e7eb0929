// Block-level scan helpers for the reduce-then-scan passes.  No kernel ever spins on another CTA: a
// scan over several CTAs is a launch that counts per CTA and one that rescans from the counts before
// its own, which it adds up itself (gather.cu) or finds scanned by a launch of one CTA in between
// (restart.cu, bulk.cu), or by the last CTA of the counting launch to finish (gather.cu's layout).
#pragma once
#include "common.cuh"

namespace b2d {

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= (uint32_t)o) v += t;
  }
  return v;
}

// Exclusive block scan of one u32 per thread; returns the exclusive prefix, *total gets the
// block sum.  `sh` needs blockDim.x/32 + 1 words.  All threads must call it.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = (blockDim.x + 31u) >> 5;
  const uint32_t inc = warp_incl_scan(v);
  if (lane == 31u) sh[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < nw ? sh[lane] : 0u;
    s = warp_incl_scan(s);
    if (lane < nw) sh[lane] = s;   // inclusive per-warp sums
  }
  __syncthreads();
  const uint32_t warp_base = warp == 0 ? 0u : sh[warp - 1];
  const uint32_t tot = sh[nw - 1];
  __syncthreads();
  *total = tot;
  return warp_base + inc - v;
}

__device__ __forceinline__ uint32_t block_reduce_sum(uint32_t v, uint32_t* sh) {
  uint32_t tot;
  block_excl_scan(v, sh, &tot);
  return tot;
}

// warp-parallel lower bound: first index of sorted v[0..cnt) with v[idx] >= key (32-ary search)
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t* v, uint32_t cnt, uint64_t key) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lo = 0, hi = cnt;
  while (hi - lo > 32u) {
    const uint32_t step = (hi - lo + 31u) / 32u;
    const uint32_t probe = lo + lane * step;
    const bool below = probe < hi && v[probe] < key;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, below));
    const uint32_t nlo = c ? lo + (c - 1u) * step + 1u : lo;
    const uint32_t nhi = (c < 32u && lo + c * step < hi) ? lo + c * step : hi;
    lo = nlo;
    hi = nhi;
  }
  const bool below = lo + lane < hi && v[lo + lane] < key;
  return lo + __popc(__ballot_sync(0xffffffffu, below));
}

// contiguous range [beg, end) of `count` items owned by CTA b out of g
__device__ __forceinline__ void cta_range(uint64_t count, uint32_t b, uint32_t g, uint64_t& beg, uint64_t& end) {
  const uint64_t per = (count + g - 1) / g;
  beg = per * b;
  end = beg + per;
  if (beg > count) beg = count;
  if (end > count) end = count;
}

}  // namespace b2d
