// Counts of tiles, CTAs and shares over whole ranges of an integer type.
#pragma once

#if defined(__CUDACC__)
#define WFB_COUNT_FN __host__ __device__ constexpr
#else
#define WFB_COUNT_FN constexpr
#endif

namespace wfb {

// ceil(n / d) for n >= 0, d > 0; (n + d - 1) / d overflows for the last d - 1 values of the type.
template <class T>
WFB_COUNT_FN T ceil_div(T n, T d) {
    return n / d + (n % d != 0 ? 1 : 0);
}

// Units that each of `warps` warps holds at first when a launch's units are spread over all of them.
WFB_COUNT_FN unsigned warp_share(unsigned units, unsigned warps) { return ceil_div(units, warps); }

// Traversal goes on with this many lanes: no more than half of what a warp holds at first.
WFB_COUNT_FN int spread_min_active(int min_active, unsigned share) {
    const unsigned half = ceil_div(share, 2u);
    return half < (unsigned)min_active ? (int)half : min_active;
}

// Tiles of a scan or compaction over n elements.
WFB_COUNT_FN int scan_tile_count(int n, int tile) { return ceil_div(n, tile); }

}  // namespace wfb
