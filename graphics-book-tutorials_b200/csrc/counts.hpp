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

// Units that each of `warps` warps holds at first when a launch's units are spread over all of them: for up to kMaxWideUnits
// units and 65,536 warps (148 SMs hold 4,736). The host keeps larger launches from the ordered megakernel; forms that cover
// them in the kernel moved its code and cost small renders of icospheres 1 to 5% (208x160x2: 1.08 -> 1.10 to 1.14 ms).
constexpr unsigned kMaxWideUnits = 0xffff0000u;
WFB_COUNT_FN unsigned warp_share(unsigned units, unsigned warps) { return (units + warps - 1) / warps; }

// Tiles of a scan or compaction over n elements.
WFB_COUNT_FN int scan_tile_count(int n, int tile) { return ceil_div(n, tile); }

}  // namespace wfb
