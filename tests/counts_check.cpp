// Counts at both ends of their ranges (csrc/counts.hpp), against 64-bit arithmetic. Prints "ok <checks>".
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "counts.hpp"

static long long checks = 0;
static void want(long long got, long long expect, const char* what, long long a, long long b) {
    ++checks;
    if (got == expect) return;
    std::printf("%s(%lld, %lld) = %lld, want %lld\n", what, a, b, got, expect);
    std::exit(1);
}

int main() {
    // elements near 0, a tile's edges and the end of the range; the tiles of the scan kernels
    for (int tile : {1024, 4096})
        for (long long mid : {0ll, 1024ll, 4096ll, 1ll << 20, 16000003ll, 0x7fffffffll - 5000, 0x7fffffffll - 4095, 0x7fffffffll})
            for (long long n = mid - 3; n <= mid + 3; ++n)
                if (n >= 1 && n <= 0x7fffffffll)
                    want(wfb::scan_tile_count((int)n, tile), (n + tile - 1) / tile, "scan_tile_count", n, tile);
    // units near 0 and up to the largest launch; warps of one CTA, of small grids, of 148 SMs with 8 CTAs of 4 warps, and the most
    for (long long warps : {4ll, 32ll, 1000ll, 148ll * 8 * 4, 65536ll})
        for (long long mid : {0ll, 5000ll, 1ll << 31, 0xffffffffll - 70000, (long long)wfb::kMaxWideUnits})
            for (long long u = mid - 3; u <= mid; ++u)
                if (u >= 0)
                    want(wfb::warp_share((unsigned)u, (unsigned)warps), (u + warps - 1) / warps, "warp_share", u, warps);
    std::printf("ok %lld\n", checks);
    return 0;
}
