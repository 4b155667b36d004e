// How the molecule sweep launches more systems than the device runs at once
// (host code without CUDA, so that it is tested as it is).
#pragma once
#include <cmath>
#include <cstdint>

namespace fgm {

struct MolTurns {
    int slots;          // systems of one launch
    int64_t quantum;    // trials of each in one launch
};

// n systems with streams of up to maxn trials, in groups of `ahead`; `fit`
// clusters run at once (0: unknown), launches hold at most `chunk` trials of a
// system. A last wave of clusters that is nearly empty costs as much as a full
// one (at 4 CTAs the GPU holds 36 clusters at once: 38 systems ran 2 waves for
// 1.06 waves' work). Where more than a tenth would be lost, the systems take
// turns: launches of exactly `slots` clusters run `quantum` trials of each, in
// rotation, so that all of them are full. Nothing to run: one empty launch set.
// A launch costs some 5 trials, and lasts as long as its unluckiest system, whose
// groups ended early on molecules met twice: 3.5 sqrt(p quantum) trials more, p
// the chance that a group of 16 meets one of `molecules` twice. Measured over 38
// systems of 20-site molecules, milliseconds in waves and by turns: 1000
// molecules 3.04 and 3.18 (64 trials: waves), 12.4 and 9.5 (256: turns); 200
// molecules 1.55 and 1.79, 6.1 and 5.4, 25.4 and 18.2 (1024); 24 molecules 2.46
// and 2.26, 8.9 and 7.8, 34.1 and 25.7.
inline MolTurns mol_turns(int64_t maxn, int n, int fit, int ahead, int molecules, int64_t chunk) {
    MolTurns t{n, chunk};
    if (maxn <= 0 || fit <= 0 || fit >= n) return t;
    const int waves = (n + fit - 1) / fit;
    if (10 * (int64_t)n >= 9 * (int64_t)waves * fit) return t;
    const double late = 3.5 * std::sqrt(1.0 - std::exp(-0.5 * ahead * (ahead - 1) / molecules));
    double best = waves;   // in waves of maxn trials
    for (int q = 2; q <= 16; q++) {   // turns per system; whole groups each
        const int64_t qu = ((maxn + q - 1) / q + ahead - 1) / ahead * ahead;
        const int64_t turns = (maxn + qu - 1) / qu, rounds = (turns * n + fit - 1) / fit;
        const double cost = (double)rounds * ((double)qu + 5.0 + late * std::sqrt((double)qu)) / (double)maxn;
        if (qu <= chunk && cost < best) {
            best = cost;
            t = {fit, qu};
        }
    }
    return t;
}

}  // namespace fgm
