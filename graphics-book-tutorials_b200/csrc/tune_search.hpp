// The autotuner's search (autotune.cpp measures): which launch configurations of each arm are timed, and which one is taken.
#pragma once
#include <vector>

namespace wfb {

struct TuneResult {
    int mode = 0;  // the faster arm: WFB_MODE_MEGAKERNEL or WFB_MODE_WAVEFRONT
    // Best megakernel knobs.
    int block = 128, occupancy = 0, min_active = 16, leaf_batch = 8;
    // Best wavefront knobs (0: not tried, library defaults).
    int paths_in_flight = 0, wf_min_active = 0, wf_occupancy = -1;
    // kTuneMegakernel, kTuneWavefront: that arm's defaults are as fast as its best knobs above (which are then not applied;
    // paths_in_flight always is).
    int keep_defaults = 0;
    double msamples_s = 0.0;             // the winner's measured rate
    double megakernel_msamples_s = 0.0;  // best megakernel candidate
    double wavefront_msamples_s = 0.0;   // best wavefront candidate (0 if not tried)
    int candidates = 0;
};

enum : int { kTuneMegakernel = 1, kTuneWavefront = 2 };

// Knobs of one probe; all negative: the arm's defaults.
struct MegakernelKnobs {
    int block = -1, occupancy = -1, min_active = -1, leaf_batch = -1;
};
struct WavefrontKnobs {
    int occupancy = -1, min_active = -1;
};

// The ordered traversal's defaults depend on the tree (with_defaults, kWf*) and were measured over longer renders than a probe;
// other knobs replace them only when a probe is faster by more than probes of one configuration differ (2.8% on cornell36
// at 320x180).
constexpr double kTuneMargin = 1.03;

// measure(knobs) -> milliseconds of a probe render. Returns the best time.
//   ordered (the scene has wide nodes): the defaults, then min_active {4, 8, .. 28} x leaf_batch {8, 16, 32}: the kernel has one
//     shape, so block and occupancy stay at 128 and 10, which it does not read
//   else: stage 1, (block, occupancy target) in {(128,10), (128,8), (128,6), (128,0), (64,0), (256,0)} x min_active in {8, 16, 24} at
//     leaf_batch 8; stage 2, the stage-1 winner with leaf_batch in {4, 12, 16, 32}; stage 3, min_active 4 either side of the winner
template <class Measure>
double search_megakernel(bool ordered, Measure&& measure, TuneResult& best) {
    double best_ms = 1e300;
    auto probe = [&](int block, int occupancy, int min_active, int leaf_batch) {
        const double ms = measure(MegakernelKnobs{block, occupancy, min_active, leaf_batch});
        best.candidates++;
        if (!(ms < best_ms)) return;
        best_ms = ms;
        best.block = block;
        best.occupancy = occupancy;
        best.min_active = min_active;
        best.leaf_batch = leaf_batch;
    };
    if (ordered) {
        const double default_ms = measure(MegakernelKnobs{});
        best.candidates++;
        for (int lb : {16, 32, 8})
            for (int ma = 4; ma <= 28; ma += 4) probe(128, 10, ma, lb);
        if (default_ms < best_ms * kTuneMargin) {
            best.keep_defaults |= kTuneMegakernel;
            return default_ms;
        }
        return best_ms;
    }
    const int shapes[][2] = {{128, 10}, {128, 8}, {128, 6}, {128, 0}, {64, 0}, {256, 0}};
    for (const auto& sh : shapes)
        for (int ma : {8, 16, 24}) probe(sh[0], sh[1], ma, 8);
    for (int lb : {4, 12, 16, 32}) probe(best.block, best.occupancy, best.min_active, lb);
    const int ma0 = best.min_active;  // the steps of stage 1 are 8 apart
    for (int ma : {ma0 - 4, ma0 + 4})
        if (ma >= 1 && ma <= 32) probe(best.block, best.occupancy, ma, best.leaf_batch);
    return best_ms;
}

// measure(pool, knobs) -> milliseconds of a probe render's share of probe_spp samples; defaults are measured before any knobs.
//   ordered: every pool at the defaults; then, at the best pool, register cap {8, 10} x min_active {16, 20, 24}
//   else: pool x register cap {10, 8} at min_active 24; then min_active {16, 24} at the best of them
template <class Measure>
double search_wavefront(bool ordered, const std::vector<int>& pools, Measure&& measure, TuneResult& best) {
    double best_ms = 1e300;
    if (ordered) {
        double default_ms = 1e300;
        for (int pool : pools) {
            const double ms = measure(pool, WavefrontKnobs{});
            best.candidates++;
            if (ms < default_ms) {
                default_ms = ms;
                best.paths_in_flight = pool;
            }
        }
        for (int occ : {8, 10})
            for (int ma : {16, 20, 24}) {
                const double ms = measure(best.paths_in_flight, WavefrontKnobs{occ, ma});
                best.candidates++;
                if (ms < best_ms) {
                    best_ms = ms;
                    best.wf_occupancy = occ;
                    best.wf_min_active = ma;
                }
            }
        if (default_ms < best_ms * kTuneMargin) {
            best.keep_defaults |= kTuneWavefront;
            return default_ms;
        }
        return best_ms;
    }
    best.wf_min_active = 24;
    for (int pool : pools)
        for (int occ : {10, 8}) {
            const double ms = measure(pool, WavefrontKnobs{occ, 24});
            best.candidates++;
            if (ms < best_ms) {
                best_ms = ms;
                best.paths_in_flight = pool;
                best.wf_occupancy = occ;
            }
        }
    for (int ma : {16, 24}) {
        const double ms = measure(best.paths_in_flight, WavefrontKnobs{best.wf_occupancy, ma});
        best.candidates++;
        if (ms < best_ms) {
            best_ms = ms;
            best.wf_min_active = ma;
        }
    }
    return best_ms;
}

}  // namespace wfb
