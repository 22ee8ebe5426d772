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
    // units near 0 and the end of the range; warps of one CTA, of small grids, and of 148 SMs with 8 CTAs of 4 warps
    for (long long warps : {4ll, 32ll, 1000ll, 148ll * 8 * 4})
        for (long long mid : {0ll, 5000ll, 1ll << 31, 0xffffffffll - 4736, 0xfffffffell})
            for (long long u = mid - 3; u <= mid + 3; ++u)
                if (u >= 0 && u <= 0xffffffffll) {
                    const long long share = (u + warps - 1) / warps;
                    want(wfb::warp_share((unsigned)u, (unsigned)warps), share, "warp_share", u, warps);
                    for (int least : {1, 4, 8, 16, 32}) {
                        const long long half = (share + 1) / 2;
                        want(wfb::spread_min_active(least, (unsigned)share), half < least ? half : least, "spread_min_active",
                             least, share);
                    }
                }
    std::printf("ok %lld\n", checks);
    return 0;
}
