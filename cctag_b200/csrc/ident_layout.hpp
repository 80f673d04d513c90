// Blocks per marker, warps per block and staged pixels of an identification launch.
#pragma once

namespace cctagb {

enum class IdentPixels {
    kNone,  // every marker reads the image
    kSome,  // room for the largest that leaves kIdentSpareL1 of the SM to the L1
    kAll    // room for the largest, as far as there is
};

struct IdentLayout {
    int cluster;         // blocks per marker (one cluster)
    int perSm;           // blocks meant to share an SM
    int warps;           // per block
    IdentPixels pixels;  // held in shared memory
};

constexpr int kMaxCluster = 8;       // blocks per marker at most
constexpr int kIdentWarps = 20;      // warps of a block with an SM to itself
constexpr int kIdentTrialWarps = 25; // one per trial, and the most that the registers allow
constexpr int kGnBlocks = 7;         // blocks per SM of a large Gauss-Newton launch
constexpr int kGnWarps = 4;          // and their warps: one per chunk of 32 samples
constexpr int kIdentSpareL1 = 40 * 1024;

// Sampling tasks of a grid round: one per trial and whole chunk of 32 samples, the
// partial chunks packed, several trials to a task.
inline int ident_round_tasks(int trials, int samples)
{
    const int tail = samples % 32;
    int width = 1;
    while (width < tail) width <<= 1;
    return trials * (samples / 32) + (tail ? (trials * width + 31) / 32 : 0);
}

// Whether a grid launch keeps no room for pixels: more than half of its markers
// would find none (see below).
inline bool ident_no_pixels(int n, int beyond) { return 2LL * beyond > n; }

struct IdentLaunch {
    int n, sms;
    int trials, samples;      // of a grid round; along a cut
    bool gn, blockLayout;     // blockLayout: one block per marker asked for (it takes the least SM time)
    int beyond, beyondHalf;   // markers whose pixels exceed the shared memory of a block with an SM to itself,
                              // of two on an SM
};

// Grid.  With few markers the tasks of a round (79 for 25 trials of 100 samples)
// spread over a cluster of 8 blocks of 10 warps, then 4 or 2 blocks of 20, or as
// many as share them out evenly, as long as the blocks fit the SMs side by side,
// pairs up to a quarter beyond: the pairs that start late cost where all markers
// are alike (92 of 50 px radius 327 us, a block each 253; 75 of 8-150 px 292 and
// 297), but a block each leaves a large one to a single SM (80 candidates of a
// 3840x2160 clutter frame, of up to 300 px, 346 us in pairs, 547 a block each).
// With more markers a block each, of 20 warps while an SM has one marker, else two
// blocks of 12 warps on an SM.
//
// Pixels.  A marker's pixels fit a block up to some 220 px of radius, of two on an
// SM up to 145 px.  One that does not fit reads the image through what the shared
// memory leaves of the L1, so that room kept for pixels in vain costs it twice
// (1000 markers of 400 px with all of the room taken 9.0 ms, with none 3.9 ms;
// 4.2 ms before there was any).  So: two blocks on an SM only where at most one
// marker in 16 does not fit them (1000 of 200 px 4.8 ms so, 1.9 ms a block each); a
// block each, and one that does not fit among them, leave 40 KB to the L1 (350 of
// 150 and 260 px 1.17 ms, 1.28 with all room taken, 1.51 with none); none at all
// where more than half do not fit (296 of 100-400 px 1.19 ms, 1.35 with 40 KB left;
// before 1.27), or in a launch that lasts as long as its largest marker (148 of
// 8-300 px 631 us, 775 with 40 KB left, 923 without; before 677).  A launch without
// pixels has a warp per trial, which reads all chunks of a cut at once (148 of 400
// px 628 us, 714 with a task per chunk).
//
// Gauss-Newton: an evaluation is one task per chunk and serial steps, so blocks
// beyond the chunks help the grid rounds before it only (8 markers of 100 samples:
// clusters of 8 and 4 112 and 111 us at 50 px radius, 151 and 161 at 400 px; of 64
// samples, two chunks, 141 and 134 at 260 px), and a cluster that has to wait for
// another one doubles the call.  The blocks of a cluster share a GPC, whose SMs are
// no multiple of them: of 148 SMs 12 clusters of 8 ran at once and 33 of 4, so these
// go up to two thirds and to seven eighths of the SMs (18 markers of 150 px radius
// 138 us, 216 us in clusters of 8).  Then a block of 20 warps per marker (37 markers
// 140-163 us, clusters of 4 150-187; 92 markers 154-171 us, pairs 196-278).  Two
// blocks of 12 warps on an SM up to a quarter beyond twice the SMs, then kGnBlocks
// of 4: of 8-150 px radius 297 markers 209 and 293 us, 330 255 and 306, 400 292 and
// 310, 600 364 and 366, 1000 553 and 525; of 15 px 330 markers 244 and 242, 400 268
// and 257, 1000 492 and 430.  (Its pixels: launch_identify.)
inline IdentLayout ident_layout(const IdentLaunch& a)
{
    IdentLayout r{1, 1, kIdentWarps, IdentPixels::kAll};
    const int n = a.n, sms = a.sms;
    if (a.gn) {
        if (!a.blockLayout && a.samples > 64 && n <= (sms - sms / 3) / 8) {
            r.cluster = 8;
            r.warps = 10;
        } else if (!a.blockLayout && n <= (sms - sms / 8) / 4) {
            r.cluster = 4;
        } else if (n > 2 * sms + sms / 4) {
            r.perSm = kGnBlocks;
            r.warps = kGnWarps;
        } else if (n > sms) {
            r.perSm = 2;
            r.warps = 12;
        }
        return r;
    }
    const bool none = ident_no_pixels(n, a.beyond);
    if (!a.blockLayout) {
        if (n <= sms / kMaxCluster) r.cluster = kMaxCluster;
        else if (n <= sms / 4) r.cluster = 4;
        else if (n <= (sms + (none ? 0 : sms / 4)) / 2) r.cluster = 2;
    }
    r.pixels = none ? IdentPixels::kNone : a.beyond ? IdentPixels::kSome : IdentPixels::kAll;
    if (r.cluster > 1) {
        const int share = (ident_round_tasks(a.trials, a.samples) + r.cluster - 1) / r.cluster;
        const int turns = (share + kIdentTrialWarps - 1) / kIdentTrialWarps;
        const int even = (share + turns - 1) / turns, least = r.cluster == kMaxCluster ? 10 : kIdentWarps;
        r.warps = even > least ? even : least;
    } else if (n > sms && !a.beyond && 16LL * a.beyondHalf <= n) {
        r.perSm = 2;
        r.warps = 12;
    } else {
        if (a.beyond && n <= sms) r.pixels = IdentPixels::kNone;
        if (r.pixels == IdentPixels::kNone && a.trials == kIdentTrialWarps) r.warps = kIdentTrialWarps;
    }
    return r;
}

}  // namespace cctagb
