// The autotuner's search (csrc/tune_search.hpp) on made-up probe times. Prints "ok <checks>".
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
#include <tuple>
#include "tune_search.hpp"

static long long checks = 0;
#define CHECK(c)                                                     \
    do {                                                             \
        ++checks;                                                    \
        if (!(c)) {                                                  \
            std::printf("line %d: %s\n", __LINE__, #c);              \
            std::exit(1);                                            \
        }                                                            \
    } while (0)

using namespace wfb;

int main() {
    std::mt19937 rng(7);
    std::uniform_real_distribution<double> ms(0.5, 1.5);
    for (int round = 0; round < 400; ++round) {
        for (const bool ordered : {false, true}) {
            // ---- megakernel ----
            TuneResult t;
            std::map<std::tuple<int, int, int, int>, double> cost;
            int calls = 0;
            // every third round the defaults are the best by far, every other third close to the best
            const double defaults = round % 3 == 0 ? 0.4 : round % 3 == 1 ? 0.5 : ms(rng);
            const double got = search_megakernel(ordered, [&](const MegakernelKnobs& k) {
                const bool def = k.block < 0 && k.occupancy < 0 && k.min_active < 0 && k.leaf_batch < 0;
                CHECK(def == (ordered && calls == 0));  // the defaults first, before a renderer's knobs are set
                ++calls;
                if (def) return defaults;
                return cost.try_emplace({k.block, k.occupancy, k.min_active, k.leaf_batch}, ms(rng)).first->second;
            }, t);
            CHECK(t.candidates == calls && calls == (ordered ? 1 + 7 * 3 : 6 * 3 + 4 + 2));
            const double knobs = cost.at({t.block, t.occupancy, t.min_active, t.leaf_batch});
            for (const auto& [k, v] : cost) CHECK(knobs <= v);
            CHECK((t.keep_defaults & kTuneWavefront) == 0);
            const bool kept = (t.keep_defaults & kTuneMegakernel) != 0;
            CHECK(kept == (ordered && defaults < knobs * kTuneMargin));
            CHECK(got == (kept ? defaults : knobs));
            if (ordered) CHECK(got <= defaults * 1.0000001);  // what is applied is never slower than the defaults
            if (ordered)
                for (const auto& [k, v] : cost) CHECK(std::get<0>(k) == 128 && std::get<1>(k) == 10);

            // ---- wavefront ----
            TuneResult w;
            std::map<std::tuple<int, int, int>, double> wcost;
            std::map<int, double> dcost;
            const std::vector<int> pools = round % 2 ? std::vector<int>{300000, 1 << 21, 1 << 22} : std::vector<int>{2304};
            bool knobs_seen = false;
            const double wgot = search_wavefront(ordered, pools, [&](int pool, const WavefrontKnobs& k) {
                if (k.occupancy < 0 && k.min_active < 0) {
                    CHECK(ordered && !knobs_seen);
                    return dcost[pool] = ms(rng);
                }
                knobs_seen = true;
                CHECK(k.occupancy == 8 || k.occupancy == 10);
                return wcost.try_emplace({pool, k.occupancy, k.min_active}, ms(rng)).first->second;
            }, w);
            CHECK(w.keep_defaults == 0 || w.keep_defaults == kTuneWavefront);
            const double best_knobs = wcost.at({w.paths_in_flight, w.wf_occupancy, w.wf_min_active});
            if (ordered) {
                CHECK(dcost.size() == pools.size());
                for (const auto& [pool, v] : dcost) CHECK(dcost.at(w.paths_in_flight) <= v);
                const double d = dcost.at(w.paths_in_flight);
                CHECK((w.keep_defaults != 0) == (d < best_knobs * kTuneMargin));
                CHECK(wgot == (w.keep_defaults ? d : best_knobs) && wgot <= d * 1.0000001);
            } else {
                CHECK(w.keep_defaults == 0 && wgot == best_knobs);
                for (const auto& [k, v] : wcost)
                    if (std::get<2>(k) == 24) CHECK(best_knobs <= v);
            }
        }
    }
    std::printf("ok %lld\n", checks);
    return 0;
}
