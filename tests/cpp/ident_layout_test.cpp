// ident_layout (ident_layout.hpp) over numbers of markers and SMs: blocks that
// the hardware holds, and for Gauss-Newton, where a cluster that waits for
// another one or a block that waits for an SM costs a whole call, launches that
// start at once wherever one of the layouts does.
#include <cstdio>
#include <initializer_list>

#include "ident_layout.hpp"

using namespace cctagb;

int main()
{
    int bad = 0;
    auto check = [&](bool ok, const char* what, int n, int sms, bool gn, bool block) {
        if (!ok && ++bad < 20) std::printf("%s: n %d sms %d gn %d block %d\n", what, n, sms, gn, block);
    };
    for (int sms : {16, 20, 66, 74, 108, 132, 144, 148, 160})
        for (int gn = 0; gn < 2; ++gn)
            for (int block = 0; block < 2; ++block)
                for (int k = 0; k < 4 * 8 * sms; ++k) {
                    const int n = k / 4 + 1, chunks = k % 4 + 1;
                    const IdentLayout r = ident_layout(n, sms, chunks, gn, block);
                    auto want = [&](bool ok, const char* what) { check(ok, what, n, sms, gn, block); };
                    want(r.cluster == 1 || r.cluster == 2 || r.cluster == 4 || r.cluster == 8, "cluster size");
                    want(!block || r.cluster == 1, "one block per marker asked for");
                    // 72 registers a thread; a quarter of the warps per register partition
                    want((r.perSm * r.warps + 3) / 4 * 32 * 72 <= 16384, "registers");
                    want(r.warps >= 4, "the warps that share out the set-up");
                    if (gn) {
                        // clusters share a GPC: not every SM is in a whole cluster
                        want(r.cluster == 1 || n * r.cluster <= sms - sms / (r.cluster > 4 ? 3 : 8),
                             "clusters side by side");
                        want(n > sms || r.cluster > 1 || r.perSm == 1, "a block per SM while there are SMs");
                        want(r.perSm < kGnBlocks || n > 2 * sms + sms / 4, "small blocks for many markers only");
                    } else {
                        want(r.cluster == 1 || n * r.cluster <= sms + sms / 4, "clusters nearly side by side");
                    }
                }
    std::printf("%d violations\n", bad);
    return bad != 0;
}
