// How the molecule sweep launches more systems than the device runs at once
// (host code without CUDA, so that it is tested as it is).
#pragma once
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
inline MolTurns mol_turns(int64_t maxn, int n, int fit, int ahead, int64_t chunk) {
    MolTurns t{n, chunk};
    if (maxn <= 0 || fit <= 0 || fit >= n) return t;
    const int waves = (n + fit - 1) / fit;
    if (10 * (int64_t)n >= 9 * (int64_t)waves * fit) return t;
    double best = waves;
    for (int q = 2; q <= 16; q++) {   // turns per system; whole groups each
        const int64_t qu = ((maxn + q - 1) / q + ahead - 1) / ahead * ahead;
        const int64_t turns = (maxn + qu - 1) / qu, rounds = (turns * n + fit - 1) / fit;
        // in waves of maxn trials; a launch lasts as long as its unluckiest system, whose
        // groups ended early on a molecule met twice (about 6 trials at 1000 molecules)
        const double cost = (double)rounds * (double)(qu + 6) / (double)maxn;
        if (qu <= chunk && cost < best) {
            best = cost;
            t = {fit, qu};
        }
    }
    return t;
}

}  // namespace fgm
