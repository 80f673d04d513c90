// ident_layout (ident_layout.hpp) over numbers of markers and SMs: blocks that
// the hardware holds; for Gauss-Newton, where a cluster that waits for another
// one or a block that waits for an SM costs a whole call, launches that start at
// once wherever one of the layouts does; and markers whose pixels do not fit in
// shared memory, which read the image through the L1, are given an L1.
#include <cstdio>
#include <initializer_list>

#include "ident_layout.hpp"

using namespace cctagb;

int main()
{
    int bad = 0;
    auto check = [&](bool ok, const char* what, const IdentLaunch& a) {
        if (!ok && ++bad < 20)
            std::printf("%s: n %d sms %d trials %d samples %d gn %d block %d beyond %d half %d\n", what, a.n, a.sms,
                        a.trials, a.samples, a.gn, a.blockLayout, a.beyond, a.beyondHalf);
    };
    for (int sms : {16, 20, 66, 74, 108, 132, 144, 148, 160})
        for (int k = 0; k < 2 * 2 * 2 * 4; ++k)
            for (int n = 1; n <= 8 * sms; ++n)
                for (int share = 0; share < 5; ++share) {
                    IdentLaunch a{n, sms, k & 4 ? 9 : 25, 32 + 31 * (k >> 3), bool(k & 1), bool(k & 2), 0, 0};
                    // all markers fit two blocks on an SM, all one, a few do not, most do not, none fits
                    a.beyond = share < 2 ? 0 : share == 2 ? (n + 9) / 10 : share == 3 ? (4 * n + 4) / 5 : n;
                    a.beyondHalf = share ? n : 0;
                    const IdentLayout r = ident_layout(a);
                    auto want = [&](bool ok, const char* what) { check(ok, what, a); };
                    want(r.cluster == 1 || r.cluster == 2 || r.cluster == 4 || r.cluster == 8, "cluster size");
                    want(!a.blockLayout || r.cluster == 1, "one block per marker asked for");
                    // 72 registers a thread; a quarter of the warps per register partition
                    want((r.perSm * r.warps + 3) / 4 * 32 * 72 <= 16384, "registers");
                    want(r.warps >= 4, "the warps that share out the set-up");
                    if (a.gn) {
                        // clusters share a GPC: not every SM is in a whole cluster
                        want(r.cluster == 1 || n * r.cluster <= sms - sms / (r.cluster > 4 ? 3 : 8),
                             "clusters side by side");
                        want(n > sms || r.cluster > 1 || r.perSm == 1, "a block per SM while there are SMs");
                        want(r.perSm < kGnBlocks || n > 2 * sms + sms / 4, "small blocks for many markers only");
                        continue;
                    }
                    want(r.cluster == 1 || n * r.cluster <= sms + sms / 4, "clusters nearly side by side");
                    want(share == 0 || r.perSm == 1, "blocks that hold their markers' pixels");
                    want(share < 2 || r.pixels != IdentPixels::kAll, "an L1 for markers beyond the shared memory");
                    want(share < 3 || r.pixels == IdentPixels::kNone, "no room where most find none");
                    want(share < 2 || r.cluster > 1 || n > sms || r.pixels == IdentPixels::kNone,
                         "no starved largest marker in a launch of one wave");
                    want(share > 1 || r.pixels == IdentPixels::kAll, "room where it is of use");
                    want(r.warps <= kIdentWarps || r.cluster > 1 || r.pixels == IdentPixels::kNone,
                         "a warp per trial for the image only");
                }
    // 25 trials: 75 whole chunks and the last 4 samples of 8 trials to a task; no
    // part of a chunk; 27 samples, a trial to a task
    const int tasks[][3] = {{100, 25, 79}, {128, 25, 100}, {123, 25, 100}, {33, 9, 10}, {32, 9, 9}, {112, 25, 88}};
    for (auto& t : tasks) {
        const int got = ident_round_tasks(t[1], t[0]);
        if (got != t[2] && ++bad) std::printf("%d tasks for %d trials of %d samples\n", got, t[1], t[0]);
    }
    std::printf("%d violations\n", bad);
    return bad != 0;
}
