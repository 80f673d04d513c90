// Blocks per marker and warps per block of an identification launch.
#pragma once

namespace cctagb {

struct IdentLayout {
    int cluster;  // blocks per marker (one cluster)
    int perSm;    // blocks meant to share an SM
    int warps;    // per block
};

constexpr int kMaxCluster = 8;   // blocks per marker at most
constexpr int kMaxIdWarps = 20;  // warps per block at most
constexpr int kGnBlocks = 7;     // blocks per SM of a large Gauss-Newton launch
constexpr int kGnWarps = 4;      // and their warps: one per chunk of 32 samples

// n markers, of `chunks` chunks of 32 samples per cut, on `sms` SMs; blockLayout: one block per marker asked for (it takes
// the least SM time).
//
// Grid: a round has one task per trial and chunk of 32 samples, 79 for 25
// trials of 100 samples (the partial chunks packed).  With few markers they
// spread over a cluster of 8 blocks of 10 warps, then 4 or 2 blocks of 20, as
// long as the blocks fit the SMs side by side, pairs up to a quarter beyond: the
// pairs that start late cost where all markers are alike (92 of 50 px radius 327
// us, a block each 253; 75 of 8-150 px 292 and 297), but a block each leaves a
// large one to a single SM (80 candidates of a 3840x2160 clutter frame, of up to
// 300 px, 387 us in pairs, 664 a block each).  With more markers a block each, of
// 20 warps while an SM has one marker, else two blocks of 12 warps on an SM.
//
// Gauss-Newton: an evaluation is one task per chunk and serial steps, so blocks
// beyond the chunks help the grid rounds before it only (8 markers of 100 samples:
// clusters of 8 and 4 112 and 111 us at 50 px radius, 151 and 161 at 400 px; of 64
// samples, two chunks, 141 and 134 at 260 px), and a cluster that has to wait for
// another one doubles the call.  The blocks of a cluster share a GPC,
// whose SMs are no multiple of them: of 148 SMs 12 clusters of 8 ran at once and
// 33 of 4, so these go up to two thirds and to seven eighths of the SMs (18
// markers of 150 px radius 138 us, 216 us in clusters of 8).  Then a block of 20
// warps per marker (37 markers 140-163 us, clusters of 4 150-187; 92 markers
// 154-171 us, pairs 196-278).  Two blocks of 12 warps on an SM up to a quarter
// beyond twice the SMs, then kGnBlocks of 4: of 8-150 px radius 297 markers 209
// and 293 us, 330 255 and 306, 400 292 and 310, 600 364 and 366, 1000 553 and
// 525; of 15 px 330 markers 244 and 242, 400 268 and 257, 1000 492 and 430.
inline IdentLayout ident_layout(int n, int sms, int chunks, bool gn, bool blockLayout)
{
    IdentLayout r{1, 1, kMaxIdWarps};
    if (gn) {
        if (!blockLayout && chunks > 2 && n <= (sms - sms / 3) / 8) r = {8, 1, 10};
        else if (!blockLayout && n <= (sms - sms / 8) / 4) r.cluster = 4;
        else if (n > 2 * sms + sms / 4) r = {1, kGnBlocks, kGnWarps};
        else if (n > sms) r = {1, 2, 12};
        return r;
    }
    if (!blockLayout) {
        if (n <= sms / kMaxCluster) r = {kMaxCluster, 1, 10};
        else if (n <= sms / 4) r.cluster = 4;
        else if (n <= (sms + sms / 4) / 2) r.cluster = 2;
    }
    if (n > sms) r = {1, 2, 12};
    return r;
}

}  // namespace cctagb
