// cpt_fetch.h — index arithmetic of the dynamic ray fetch (trace_items_walk, cpt_trace.cuh), which also
// compiles as host C++.
//
// Warps take items 0 .. n - 1 from one counter, up to 32 at a time, each until it has seen the end.  The
// counter therefore ends up to 32 per warp above n, and n may be as large as 2^31 - 2, so counter and
// sums are unsigned: as ints they wrap to negative numbers, which pass for items.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define CPT_HD __host__ __device__ __forceinline__
#else
#define CPT_HD inline
#endif

namespace cpt {

// Lanes of a warp that take items, when n (> 0) items are spread over `warps` warps.  (A signed division:
// with an unsigned one the 8-wide query kernel takes 69 registers instead of 64, 7 blocks an SM instead of
// 8, and 2M rays through 1.31M triangles 376 us instead of 368.)
CPT_HD int spread_lanes(int n, int warps)
{
    const int lanes = (n - 1) / warps + 1;
    return lanes < 32 ? lanes : 32;
}

// Whether a warp that took `count` items from `base` on has seen the end.
CPT_HD bool fetch_ends(uint32_t base, int count, int n) { return base + (uint32_t)count >= (uint32_t)n; }

// Whether number r, counted from a warp's base, is an item.
CPT_HD bool is_item(uint32_t r, int n) { return r < (uint32_t)n; }

}  // namespace cpt
