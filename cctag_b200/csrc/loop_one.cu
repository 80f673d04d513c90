// Loop 1 and the outlier removal of loop 2 of the candidate stage on the GPU
// (see loop_one.hpp).  Built with --fmad=false: every floating-point
// expression here and in cand_shared.hpp is then evaluated with the same IEEE
// operations as the host restatement, so the candidates are the same bits.
//
// k_point_records one thread per edge point: gradient angle, first direction
//                 to try, votes received and the 8 neighbouring edge points,
//                 so that a linking step is one dependent load;
// k_seed_slots    marks each seed's record with its processing slot;
// k_link_seeds    one warp per seed: the two edge-linking walks
//                 (Vote.cpp:255-394) side by side, independent of the other
//                 seeds since each walk only avoids its own points; also
//                 lists the later seeds its segment marks processed;
// k_link_resolve  one block per level: the seeds in processing order,
//                 skipping those an earlier segment marked (Detection.cpp:
//                 609-627), in shared memory; then the candidates ranked by
//                 averageReceivedVote;
// k_filter        one block per loop-two candidate: children (Vote.cpp:
//                 396-412) and the LMedS outlier removal (Vote.cpp:414-576),
//                 128 random draws evaluated at once and accepted in draw
//                 order; the draws' random stream is generated in parallel
//                 with the PCG jump-ahead;
// k_pack          the kept candidates' filtered children, packed for download;
// k_refit_hull, k_refit, k_refit_pack
//                 one block per coarse-level marker: its level-0 hull points
//                 (Multiresolution.cpp:319-401), the same outlier removal on
//                 them, packed for download.
#include "loop_one.hpp"

#include <algorithm>
#include <cstring>

#include "cand_shared.hpp"

namespace cctagb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kResolveThreads = 1024;
constexpr int kResolveSmemMarks = 24576;

// Record of edge point i: r0 = {first neighbour direction to try (link_shift),
// angle bits, votes received, seed slot or -1}, r1 / r2 = the edge points at
// the 8 neighbours in the order of Vote.cpp:283-286 for direction +1 (-1 where
// none).
struct PointRec {
    int4 r0, r1, r2;
};

__device__ __forceinline__ PointRec load_rec(const int4* rec, int i)
{
    PointRec r;
    r.r0 = rec[3 * i];
    r.r1 = rec[3 * i + 1];
    r.r2 = rec[3 * i + 2];
    return r;
}
__device__ __forceinline__ int nbr(const PointRec& r, int k)
{
    const bool b0 = k & 1, b1 = k & 2, b2 = k & 4;
    const int e0 = b0 ? r.r1.y : r.r1.x, e1 = b0 ? r.r1.w : r.r1.z;
    const int e2 = b0 ? r.r2.y : r.r2.x, e3 = b0 ? r.r2.w : r.r2.z;
    const int f0 = b1 ? e1 : e0, f1 = b1 ? e3 : e2;
    return b2 ? f1 : f0;
}

__device__ __forceinline__ int px_(const LoopOneLevel& L, int i) { return L.exy[i] & 0xffff; }
__device__ __forceinline__ int py_(const LoopOneLevel& L, int i) { return L.exy[i] >> 16; }
__device__ __forceinline__ float gdx(const LoopOneLevel& L, int i) { return float(int16_t(L.grad[i] & 0xffff)); }
__device__ __forceinline__ float gdy(const LoopOneLevel& L, int i) { return float(int16_t(L.grad[i] >> 16)); }
__device__ __forceinline__ int voters(const LoopOneLevel& L, int i) { return L.voff[i + 1] - L.voff[i]; }
__device__ __forceinline__ float gnorm(const LoopOneLevel& L, int i)
{
    const float dx = gdx(L, i), dy = gdy(L, i);
    return sqrtf(dx * dx + dy * dy);
}
// Edge point at pixel (x, y), -1 if none: the word's first index plus its
// set bits below x.
__device__ __forceinline__ int at(const LoopOneLevel& L, int x, int y)
{
    if (x < 0 || x >= L.W || y < 0 || y >= L.H) return -1;
    const uint2 v = L.bitidx[size_t(y) * L.WW + (x >> 5)];
    const uint32_t bit = 1u << (x & 31);
    const int i = int(v.y) + __popc(v.x & (bit - 1u));
    return (v.x & bit) && i < L.E ? i : -1;
}

__global__ void __launch_bounds__(256) k_point_records(LoopOneArgs a, int4 total)
{
    // total.x..w: cumulative point counts of levels 0..3
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int cum[4] = {total.x, total.y, total.z, total.w};
    int l = 0;
    while (l < a.nl - 1 && t >= cum[l]) ++l;
    if (t >= cum[a.nl - 1]) return;
    const int i = t - (l ? cum[l - 1] : 0);
    const LoopOneLevel& L = a.lv[l];
    const int x = px_(L, i), y = py_(L, i);
    const int xoff[8] = {1, 1, 0, -1, -1, -1, 0, 1};
    const int yoff[8] = {0, -1, -1, -1, 0, 1, 1, 1};
    int n[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) n[k] = at(L, x + xoff[k], y + yoff[k]);
    const float angle = cand::link_angle(gdx(L, i), gdy(L, i));
    int4* rec = L.rec + 3 * size_t(i);
    rec[0] = make_int4(cand::link_shift(angle), __float_as_int(angle), voters(L, i), -1);
    rec[1] = make_int4(n[0], n[1], n[2], n[3]);
    rec[2] = make_int4(n[4], n[5], n[6], n[7]);
}

__global__ void __launch_bounds__(256) k_seed_slots(LoopOneArgs a)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int l = t / a.maxSlotsPerLevel, s = t % a.maxSlotsPerLevel;
    if (l >= a.nl) return;
    const LoopOneLevel& L = a.lv[l];
    if (s >= L.nProc) return;
    L.rec[3 * size_t(L.order[s])].w = s;
}

constexpr int kLinkThreads = 64;
constexpr int kLinkGroups = kLinkThreads / 32;  // one seed per warp: seeds do not diverge each other

__device__ __forceinline__ int4 shfl_int4(unsigned mask, int4 v, int src)
{
    return make_int4(__shfl_sync(mask, v.x, src), __shfl_sync(mask, v.y, src), __shfl_sync(mask, v.z, src),
                     __shfl_sync(mask, v.w, src));
}

// cand::link_average_vote with the division by the segment size + 1 (an
// integer up to 2 kLinkMaxLength + 2) correctly rounded by div_small.
__device__ __forceinline__ float link_average_vote_fast(float average, int segSize, int voters)
{
    const float n = __fadd_rn(__fmul_rn(average, float(segSize)), float(voters));
    const float d = float(segSize) + 1.f;
    if (segSize + 1 > 256) return n / d;
    return pm::div_small(n, d, __frcp_rn(d));
}

// The pixels around a seed that its walks can reach, one bit each: a walk
// takes at most kLinkMaxLength steps of one pixel and looks one further.
constexpr int kReach = cand::kLinkMaxLength + 1;
constexpr int kReachRow = 256;  // bits per row, >= 2 * kReach + 1
constexpr int kReachWords = (2 * kReach + 1) * kReachRow / 32;
constexpr int kReachSeed = kReach * kReachRow + kReach;  // the seed's bit
static_assert(2 * kReach + 1 <= kReachRow && kReachWords % 4 == 0, "rows of the reach map");

// Bit distance to neighbour k of the +1 order (Vote.cpp:283-286): x offsets
// 1 1 0 -1 -1 -1 0 1, y offsets 0 -1 -1 -1 0 1 1 1, two bits each.
__device__ __forceinline__ int reach_step(int k)
{
    const int dx = int(0x901Au >> (2 * k)) & 3, dy = int(0xA901u >> (2 * k)) & 3;
    return dy * kReachRow + dx - kReachRow - 1;
}

// One seed's segment in shared memory.  Direction d (0: +1, 1: -1) holds its
// points 1 .. n[d] away from the seed; entry n[d] + 1 of pt and pos is the
// point a walk looked at last when it stopped on the convexity test.
struct alignas(16) LinkSegment {
    uint32_t vis[2][kReachWords];                     // pixels a walk has visited
    int32_t pt[2][cand::kLinkMaxLength + 2];
    int32_t pos[2][cand::kLinkMaxLength + 2];         // their bits in the reach map
    int32_t votes[2][cand::kLinkMaxLength + 2];
    int32_t slot[2][cand::kLinkMaxLength + 2];
    float angle[2][cand::kLinkMaxLength + 1];         // of the point each step starts from
};

__device__ __forceinline__ bool visited(const uint32_t* vis, int pos) { return vis[pos >> 5] >> (pos & 31) & 1u; }

// Vote.cpp:272-394 edgeLinkingDir, one walk per group of 8 lanes (the active
// groups'; d: its direction): lane j examines the j-th neighbour of the search
// order, the first lane whose neighbour is an unvisited edge point decides the
// step.  r is the record of the group's current point, pos its bit, i the
// steps taken so far, n the points taken; all lanes of the warp call it.
// Returns the reference's stop code.  With useAverage the walk also ends when
// the running mean of the votes (segment size 1 + n + other) falls below
// averageVoteMin.
__device__ int link_walk(LinkSegment& S, const int4* recs, PointRec r, int pos, bool active, int d, uint32_t* vis,
                         int window, bool useAverage, float averageVoteMin, int other, int& i, int& n, int lane)
{
    const int j = lane & 7, gbase = lane & 24;
    const int dir = d ? -1 : 1;
    int stop = 0;
    float averageVote = float(r.r0.z);
    for (;;) {
        bool go = active && i < cand::kLinkMaxLength && stop >= 0;
        if (useAverage) go = go && averageVote >= averageVoteMin;
        if (!__any_sync(kFull, go)) break;
        const float angle = __int_as_float(r.r0.y);
        if (go && j == 0) S.angle[d][i] = angle;
        // direction -1 mirrors the y offsets: neighbour (8 - k) % 8 of the +1 table
        const int k = (d ? 8 - (r.r0.x + j) : 8 - r.r0.x + j) & 7;
        const int q = nbr(r, k), qpos = pos + reach_step(k);
        // every lane fetches its neighbour's record now; the step keeps one
        const bool look = go && q >= 0;
        PointRec rq = r;
        if (look) rq = load_rec(recs, q);
        const bool cand = look && !visited(vis, qpos);
        const unsigned hits = (__ballot_sync(kFull, cand) >> gbase) & 0xffu;
        // the angles of the last `window` points: the oldest and the newest
        const int count = min(i + 1, window);
        const float front = count == 1 ? angle : S.angle[d][go ? i + 1 - count : 0];
        const bool lost = cand::link_convexity_lost(front, angle, count == window, dir);
        const int src = gbase + (hits ? __ffs(hits) - 1 : 0);
        PointRec rn;
        rn.r0 = rq.r0;
        rn.r0.x = __shfl_sync(kFull, rq.r0.x, src);
        rn.r0.y = __shfl_sync(kFull, rq.r0.y, src);
        if (useAverage) rn.r0.z = __shfl_sync(kFull, rq.r0.z, src);
        rn.r1 = shfl_int4(kFull, rq.r1, src);
        rn.r2 = shfl_int4(kFull, rq.r2, src);
        const int npos = __shfl_sync(kFull, qpos, src);
        if (go) {
            ++i;
            if (!hits) {
                stop = cand::kEdgeNotFound;
            } else {
                if (lane == src) {
                    S.pt[d][n + 1] = q;
                    S.pos[d][n + 1] = qpos;
                }
                if (lost) {
                    stop = cand::kConvexityLost;
                } else {
                    ++n;
                    r = rn;
                    pos = npos;
                    if (lane == src) {
                        S.votes[d][n] = rq.r0.z;
                        S.slot[d][n] = rq.r0.w;
                        vis[qpos >> 5] |= 1u << (qpos & 31);
                    }
                    if (useAverage) averageVote = link_average_vote_fast(averageVote, 1 + n + other, r.r0.z);
                }
            }
        }
        __syncwarp();
    }
    return stop;
}

// How many points, counted from the front of the segment as it is when a walk
// ends, become processed (Vote.cpp:366-390).
__device__ __forceinline__ int link_marks(int i, int stop, int size, int window)
{
    if (i == cand::kLinkMaxLength || stop == cand::kConvexityLost) return size > window ? size - window : 0;
    return stop == cand::kEdgeNotFound ? size : 0;
}

// The reference walks in direction +1, then in direction -1 avoiding the
// points of the first walk.  Both walks are latency chains of up to 100 record
// loads, so they run side by side, each avoiding its own points; the -1 walk
// is the reference's up to the first point it took (or looked at last) that
// the +1 walk also took, and is redone from there with the +1 walk's points
// visited.  The walks are independent of each other otherwise unless the
// running mean of the votes can end them (averageVoteMin > 0, or NaN): then
// they run one after the other.  A step costs its instructions as much as its
// load: the visited points are bits of a pixel map around the seed, the first
// direction comes with the record and the convexity test is four comparisons.
// Measured (1080p frame, 540 seed slots on level 0, cold): 193 us with the
// walks in turn, a hashed set of points, and the sums and mark lists of a
// segment gathered by one lane from global memory; 102 us side by side;
// 71 us with the bit map (3840x2160 clutter frame: 223 us to 78 us).
__global__ void __launch_bounds__(kLinkThreads) k_link_seeds(LoopOneArgs a)
{
    __shared__ LinkSegment segments[kLinkGroups];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * kLinkGroups + w;
    if (t >= a.totalSlots) return;
    const int l = t / a.maxSlotsPerLevel, s = t % a.maxSlotsPerLevel;
    if (l >= a.nl) return;
    const LoopOneLevel& L = a.lv[l];
    if (s >= L.nProc) return;
    const int seed = L.order[s];
    LinkSegment& S = segments[w];
    const PointRec r0 = load_rec(L.rec, seed);
    for (int k = lane; k < 2 * kReachWords / 4; k += 32)
        reinterpret_cast<uint4*>(&S.vis[0][0])[k] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    if (lane < 2) S.vis[lane][kReachSeed >> 5] = 1u << (kReachSeed & 31);
    __syncwarp();
    const bool useAverage = !(a.averageVoteMin <= 0.f);
    const int g = lane >> 3;
    int i = 0, n = 0;
    int stop = link_walk(S, L.rec, r0, kReachSeed, g == 0 || (g == 1 && !useAverage), g & 1, S.vis[g & 1], a.window,
                         useAverage, a.averageVoteMin, 0, i, n, lane);
    const int nb = __shfl_sync(kFull, n, 0);
    const int m1 = link_marks(__shfl_sync(kFull, i, 0), __shfl_sync(kFull, stop, 0), 1 + nb, a.window);
    // the -1 walk: group 1's
    int iF = __shfl_sync(kFull, i, 8), nf = __shfl_sync(kFull, n, 8);
    int stopF = __shfl_sync(kFull, stop, 8);
    int redo = useAverage ? 1 : 0;  // its first step to redo (from 1; 0: none)
    if (!useAverage) {
        const int seen = nf + (stopF == cand::kConvexityLost ? 1 : 0);
        for (int k0 = 1; k0 <= seen && !redo; k0 += 32) {
            const bool taken = k0 + lane <= seen && visited(S.vis[0], S.pos[1][k0 + lane]);
            const unsigned m = __ballot_sync(kFull, taken);
            if (m) redo = k0 + __ffs(m) - 1;
        }
    }
    if (redo) {
        nf = iF = redo - 1;
        for (int k = 1 + lane; k <= nf; k += 32) atomicOr(&S.vis[0][S.pos[1][k] >> 5], 1u << (S.pos[1][k] & 31));
        const PointRec rf = nf ? load_rec(L.rec, S.pt[1][nf]) : r0;
        const int posF = nf ? S.pos[1][nf] : kReachSeed;
        __syncwarp();
        stopF = link_walk(S, L.rec, rf, posF, g == 0, 1, S.vis[0], a.window, useAverage, a.averageVoteMin, nb, iF, nf,
                          lane);
        stopF = __shfl_sync(kFull, stopF, 0);
        iF = __shfl_sync(kFull, iF, 0);
        nf = __shfl_sync(kFull, nf, 0);
    }
    const int size = 1 + nf + nb;
    const int m2 = link_marks(iF, stopF, size, a.window);
    // the segment, its votes, and the later seeds the marks reach: points
    // [0, m1) of (seed, back...) after the +1 walk, points [0, m2) of the
    // whole segment after the -1 walk
    int32_t* segc = a.seg + size_t(t) * kSegSlot + kSegHalf;
    int32_t* ml = a.mlist + size_t(t) * kMarkCap;
    int nReceived = 0, nVoted = 0, nm = 0;
    const unsigned lower = (1u << lane) - 1u;
    for (int p0 = 0; p0 < size; p0 += 32) {
        const int p = p0 + lane, k = p - nf;
        int v = 0, sl = -1;
        if (p < size) {
            const int d = k < 0 ? 1 : 0, q = k < 0 ? -k : k;
            segc[k] = k == 0 ? seed : S.pt[d][q];
            v = k == 0 ? r0.r0.z : S.votes[d][q];
            sl = k == 0 ? s : S.slot[d][q];
        }
        nReceived += v;
        nVoted += v > 0 ? 1 : 0;
        const bool later = sl > s;
        const unsigned f1 = __ballot_sync(kFull, later && k >= 0 && k < m1);
        if (later && k >= 0 && k < m1) ml[nm + __popc(f1 & lower)] = sl;
        nm += __popc(f1);
        const unsigned f2 = __ballot_sync(kFull, later && p < m2);
        if (later && p < m2) ml[nm + __popc(f2 & lower)] = sl;
        nm += __popc(f2);
    }
    nReceived = __reduce_add_sync(kFull, nReceived);
    nVoted = __reduce_add_sync(kFull, nVoted);
    if (lane == 0) {
        int32_t* info = a.sinfo + size_t(t) * 4;
        info[0] = nf;
        info[1] = nb;
        info[2] = nm;
        info[3] = 0;
        a.skey[t] = cand::received_vote_key(nReceived, nVoted);
    }
}

// Inclusive sum over the block's threads of v (every thread calls it).
__device__ __forceinline__ int block_inclusive(int v, int* sWarp, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) sWarp[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int u = lane < nw ? sWarp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(kFull, u, o);
            if (lane >= o) u += x;
        }
        sWarp[lane] = u;
    }
    __syncthreads();
    if (warp > 0) v += sWarp[warp - 1];
    total = sWarp[31];
    __syncthreads();
    return v;
}

// The seeds in processing order, skipping those an earlier segment marked.
// The order is a serial chain, taken 32 seeds (a window) at a time: the marks
// that stay inside a seed's own window are gathered into one word per seed
// beforehand, so that the chain inside a window is a few register operations
// per unmarked seed, and the window's candidates then set the flags of later
// seeds all at once, one warp each.
// Measured (1080p frame, 540 seeds on level 0, cold): the chain seed by seed
// with the lists copied by one thread per seed 77 us, by windows 24 us
// (3840x2160 clutter frame: 155 us to 47 us).
__global__ void __launch_bounds__(kResolveThreads) k_link_resolve(LoopOneArgs a)
{
    static_assert(kResolveThreads == 1024, "one warp per seed of a window");
    const int l = blockIdx.x;
    const LoopOneLevel& L = a.lv[l];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ int smem[];
    // [flags: maxSlots][marks offsets: maxSlots + 1][window marks, then keys: maxSlots]
    // [marks: kResolveSmemMarks, 16 bits each]; flags become the made candidates
    int* flags = smem;
    int* moff = flags + a.maxSlotsPerLevel;
    unsigned* wmarks = reinterpret_cast<unsigned*>(moff + a.maxSlotsPerLevel + 1);
    uint16_t* marks = reinterpret_cast<uint16_t*>(wmarks + a.maxSlotsPerLevel);
    __shared__ int sWarp[32];
    __shared__ unsigned sOpen;
    const int n = L.nProc;
    if (tid == 0) moff[0] = 0;
    int carry = 0;
    for (int s0 = 0; s0 < n; s0 += kResolveThreads) {
        const int s = s0 + tid;
        const int c = s < n ? a.sinfo[size_t(L.slot0 + s) * 4 + 2] : 0;
        int total;
        const int incl = block_inclusive(c, sWarp, total);
        if (s < n) {
            flags[s] = 0;
            moff[s + 1] = carry + incl;
        }
        carry += total;
    }
    __syncthreads();
    const bool inSmem = carry <= kResolveSmemMarks;
    for (int s = warp; s < n; s += 32) {
        const int32_t* ml = a.mlist + size_t(L.slot0 + s) * kMarkCap;
        const int m0 = moff[s], cnt = moff[s + 1] - m0;
        unsigned own = 0u;
        for (int k = lane; k < cnt; k += 32) {
            const int v = ml[k];
            if (inSmem) marks[m0 + k] = uint16_t(v);
            if (v >> 5 == s >> 5) own |= 1u << (v & 31);
        }
        own = __reduce_or_sync(kFull, own);
        if (lane == 0) wmarks[s] = own;
    }
    __syncthreads();
    int32_t* made = a.made + size_t(l) * a.maxSlotsPerLevel;
    int m = 0;
    for (int s0 = 0; s0 < n; s0 += 32) {
        if (warp == 0) {
            const bool in = s0 + lane < n;
            unsigned open = __ballot_sync(kFull, in && !flags[in ? s0 + lane : 0]);
            const unsigned wm = in ? wmarks[s0 + lane] : 0u;
            // a seed marks only later ones: every open seed with marks, in order
            for (unsigned todo = open & __ballot_sync(kFull, wm != 0u); todo;) {
                const int i = __ffs(todo) - 1;
                const unsigned marked = __shfl_sync(kFull, wm, i);
                open &= ~marked;
                todo &= ~marked & ~(1u << i);
            }
            if (lane == 0) sOpen = open;
            if (open >> lane & 1u) made[m + __popc(open & ((1u << lane) - 1u))] = s0 + lane;
        }
        __syncthreads();
        const unsigned open = sOpen;
        m += __popc(open);
        const int s = s0 + warp;
        if (open >> warp & 1u) {
            const int m0 = moff[s], cnt = moff[s + 1] - m0;
            const int32_t* ml = a.mlist + size_t(L.slot0 + s) * kMarkCap;
            for (int k = lane; k < cnt; k += 32) flags[inSmem ? int(marks[m0 + k]) : ml[k]] = 1;
        }
        __syncthreads();
    }
    if (tid == 0) a.meta[size_t(a.nl) * a.n2max * 4 + l] = m;
    float* keys = reinterpret_cast<float*>(wmarks);
    int* order = flags;
    for (int i = tid; i < m; i += kResolveThreads) {
        order[i] = made[i];
        keys[i] = a.skey[L.slot0 + made[i]];
    }
    __syncthreads();
    // Loop-1 order: averageReceivedVote descending, the newer candidate first
    // on equal keys (Detection.cpp:619-622).
    const int n2 = min(m, a.n2max);
    int32_t* meta = a.meta + size_t(l) * a.n2max * 4;
    for (int i = tid; i < m; i += blockDim.x) {
        const float ki = keys[i];
        int rank = 0;
        for (int j = 0; j < m; ++j) {
            const float kj = keys[j];
            rank += (kj > ki || (!(ki > kj) && j > i)) ? 1 : 0;
        }
        if (rank < n2) meta[rank * 4] = order[i];
    }
}

// Ascending bitonic sort of 64 keys held by a warp, key `lane` in a and key
// `lane + 32` in b.
__device__ __forceinline__ void bitonic64(uint32_t& a, uint32_t& b, int lane)
{
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j == 32) {  // partners lane and lane + 32, both ascending at k = 64
                const uint32_t lo = min(a, b), hi = max(a, b);
                a = lo;
                b = hi;
            } else {
                const uint32_t ya = __shfl_xor_sync(kFull, a, j), yb = __shfl_xor_sync(kFull, b, j);
                const int ea = lane, eb = lane + 32;
                const bool keepLowA = ((ea & j) == 0) == ((ea & k) == 0);
                const bool keepLowB = ((eb & j) == 0) == ((eb & k) == 0);
                a = keepLowA ? min(a, ya) : max(a, ya);
                b = keepLowB ? min(b, yb) : max(b, yb);
            }
        }
    }
}

__device__ __forceinline__ float key_value(uint32_t k)
{
    if (k == 0xffffffffu) return __int_as_float(0x7fffffff);
    const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// Draw kinds after evaluation
constexpr int kDrawFail = 0;      // counted: no usable ellipse
constexpr int kDrawUsable = 1;    // S holds its median
constexpr int kDrawNotReal = 2;   // the reference's exception: not counted
constexpr int kDrawNoGain = 3;    // counted: its median cannot beat the best so far

// Five distinct residues read from mods[p0...] (rand_5_k without rejected
// outputs); returns the position after the last one read, or -1 when the
// pool ends first.  Registers only.
__device__ __forceinline__ int draw_from(const uint8_t* mods, int p0, int g[5])
{
    int n = 0, q = p0;
    int g0 = -1, g1 = -1, g2 = -1, g3 = -1, g4 = -1;
    while (n < 5) {
        if (q >= kRawPool) return -1;
        const int r = mods[q++];
        const bool seen = r == g0 || r == g1 || r == g2 || r == g3;
        if (seen) continue;
        if (n == 0) g0 = r;
        else if (n == 1) g1 = r;
        else if (n == 2) g2 = r;
        else if (n == 3) g3 = r;
        else g4 = r;
        ++n;
    }
    g[0] = g0;
    g[1] = g1;
    g[2] = g2;
    g[3] = g3;
    g[4] = g4;
    return q;
}

// How many of the np (weighted) distances d(Q, p) * w of dist_point_ellipse are
// below S, exactly: an estimate with the approximate reciprocal (relative error
// below 2^-20) settles the points that are more than 2e-5 (relative) away from
// S; if any point is closer, or its estimate is not finite or its denominator
// beyond the reciprocal's range (or S near the denormals), all are counted with
// the IEEE expression.
__device__ __forceinline__ int count_below(const geo::Mat3& Q, const geo::Pt* pts, const float* wts, int np,
                                           bool weighted, float S)
{
    const float lo = S * 0.99998f, hi = S * 1.00002f;
    int below = 0;
    bool close = !(S > 1e-30f);
#pragma unroll 4
    for (int i = 0; i < np; ++i) {
        const float x = pts[i].x, y = pts[i].y;
        const float aux0 = x * x, aux1 = 2 * x * y, aux2 = 2 * x, aux3 = y * y, aux4 = 2 * y;
        const float t1 = x * Q.m[0][0] + y * Q.m[0][1] + Q.m[0][2];
        const float t2 = x * Q.m[0][1] + y * Q.m[1][1] + Q.m[1][2];
        const float denom = t1 * t1 + t2 * t2;
        const float dot = aux0 * Q.m[0][0] + aux1 * Q.m[0][1] + aux2 * Q.m[0][2] + aux3 * Q.m[1][1] +
                          aux4 * Q.m[1][2] + Q.m[2][2];
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(denom));
        float v = dot * dot * r;
        if (weighted) v *= wts[i];
        const bool less = v < lo, more = v > hi && v <= 3.4e38f;
        close = close || !(less || more) || !(denom < 1e37f);
        below += less ? 1 : 0;
    }
    if (close) {
        below = 0;
        for (int i = 0; i < np; ++i) {
            float d = geo::dist_point_ellipse(Q, pts[i].x, pts[i].y);
            if (weighted) d *= wts[i];
            below += d < S ? 1 : 0;
        }
    }
    return below;
}

constexpr int kRawPer = kRawPool / kFilterThreads;  // random outputs per thread
constexpr int kRawEnd = kRawPool;                    // start position past the last output
constexpr int kRawDead = kRawPool + 1;               // ... and after a draw the pool does not hold whole
constexpr int kFirstMedians = 12;                    // draws of the first batch whose median is taken outright

// Shared state of one outlier removal.
struct LmedsShared {
    geo::Pt pts[kLmedsMaxPts];
    float wts[kLmedsMaxPts];
    uint32_t raws[kRawPool];
    alignas(8) uint8_t mods[kRawPool + 16];          // raws mod np; 255 past the end
    int16_t next[kRawDead + 1];                      // where the draw at a position ends
    int16_t jump[2][kRawDead + 1];                   // ... 2^b draws on
    int8_t perms[kFilterThreads][5];
    int kinds[kFilterThreads];
    float svals[kFilterThreads];
    float Q[kFilterThreads][9];
    float bestQ[9];
    long long target[kLmedsMaxPts + 1];
    int npts, done, nd, counter, draws, warpCnt[4][kFilterThreads / 32];
    float sm;
    unsigned long long state, inc;
};

// The draws (Statistic.cpp:16-29 rand_5_k) held by the pool of random outputs
// in S.mods: a draw consumes outputs until it has 5 distinct residues.  Every
// position's draw length is found in parallel (the residues of the next
// outputs as bits of a 64-bit word, np <= 64); the k-th draw's start is the
// k-fold chain of those lengths from position 0, followed by pointer doubling,
// one thread per draw.  Sets S.nd, S.perms and the stream's next state.
// (A chain walked by one thread, with the lengths read byte by byte, took
// 30 k of a batch's 75 k cycles.)
__device__ __forceinline__ void lmeds_draws(LmedsShared& S)
{
    const int tid = threadIdx.x;
    uint64_t bit[kRawPer + 11];
#pragma unroll
    for (int k = 0; k < kRawPer + 11; ++k) {
        const int v = S.mods[min(tid * kRawPer + k, kRawPool + 15)];
        bit[k] = v < 64 ? 1ull << v : 0ull;
    }
#pragma unroll
    for (int k = 0; k < kRawPer; ++k) {
        const int p = tid * kRawPer + k;
        uint64_t m = bit[k] | bit[k + 1] | bit[k + 2] | bit[k + 3] | bit[k + 4];
        int len = 5, have = __popcll(m);
#pragma unroll
        for (int q = 5; q < 12; ++q) {
            len += have < 5 ? 1 : 0;
            m |= bit[k + q];
            have = have < 5 ? __popcll(m) : have;
        }
        int end = p + len;
        if (have < 5 || end > kRawEnd) {  // longer than 12 outputs, or past the pool
            int g[5];
            const int q = draw_from(S.mods, p, g);
            end = q > 0 ? q : kRawDead;
        }
        S.next[p] = S.jump[0][p] = int16_t(end);
    }
    if (tid < 2) S.next[kRawEnd + tid] = S.jump[0][kRawEnd + tid] = S.jump[1][kRawEnd + tid] = int16_t(kRawDead);
    __syncthreads();
    int p = 0;  // start of draw tid
    for (int b = 0; 1 << b < kFilterThreads; ++b) {
        const int16_t* J = S.jump[b & 1];
        if (tid >> b & 1) p = J[p];
        int16_t* N = S.jump[(b & 1) ^ 1];
#pragma unroll
        for (int k = 0; k < kRawPer; ++k) {
            const int q = k * kFilterThreads + tid;
            N[q] = J[J[q]];
        }
        __syncthreads();
    }
    const bool whole = p < kRawEnd && S.next[p] <= kRawEnd;  // and so are all draws before it
    const int nd = __syncthreads_count(whole);
    if (whole) {
        int g[5];
        const int end = draw_from(S.mods, p, g);
#pragma unroll
        for (int i = 0; i < 5; ++i) S.perms[tid][i] = int8_t(g[i]);
        if (tid == nd - 1) {
            geo::Pcg32 r;
            r.state = S.state;
            r.inc = S.inc;
            r.advance(uint64_t(end));
            S.state = r.state;
        }
    }
    if (tid == 0) S.nd = nd;
}

// The median (rank np / 2, NaN last) of draw d's distances, by a warp: two
// points per lane, then a 64-key bitonic sort.
__device__ __forceinline__ float lmeds_median(const LmedsShared& S, int d, int np, bool weighted, int lane)
{
    geo::Mat3 Q;
#pragma unroll
    for (int k = 0; k < 9; ++k) Q.m[k / 3][k % 3] = S.Q[d][k];
    uint32_t key[2] = {0xffffffffu, 0xffffffffu};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        if (i < np) {
            float v = geo::dist_point_ellipse(Q, S.pts[i].x, S.pts[i].y);
            if (weighted) v *= S.wts[i];
            key[h] = geo::order_key(v);
        }
    }
    bitonic64(key[0], key[1], lane);
    const int r = np / 2;
    return key_value(__shfl_sync(kFull, r < 32 ? key[0] : key[1], r & 31));
}

// Block-wide outlierRemoval (Vote.cpp:414-576) with maxSize 60 over the n
// edge points idx[0, n) of level L: LMedS ellipse from random 5-point subsets
// of a regular subsample, drawn from `rng`, kFilterThreads at a time and
// accepted in draw order; then idx is compacted in place (order kept) to the
// points whose distance (times 255 / |gradient| when weighted) is below
// threshold * the best median.  Returns their number (0 when fewer than 5
// points are subsampled).  Every thread of the block must call it.
//
// Latency-bound (one block of 4 warps per candidate, 1-3 batches of draws).  A
// draw's median costs a warp some 900 cycles, so only draws that can improve
// get one: those with enough distances below a median known to come before
// them, the first batch's bound being the least of its first kFirstMedians.
// Measured (1080p frame, cold): k_filter 124 us with the draws chained by one
// thread, a median per usable draw and the children gathered by one warp, 58 us
// now (3840x2160 clutter: 149 us and 63 us); the re-fit's removal 46 us.
__device__ int lmeds_outliers(const LoopOneLevel& L, int32_t* idx, int n, bool weighted, float threshold,
                              const geo::Pcg32 rng0, int32_t* err)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ LmedsShared S;
    const int nchild = n;
    int32_t* children = idx;
    // The reference scans the children and takes child i when i equals
    // size_t(float(k) * step) for the next k: the taken indices are those
    // targets while they increase strictly and stay below nchild.
    const int nSub = min(nchild, 60);
    if (nSub < 5) return 0;
    if (tid <= kLmedsMaxPts) {
        const float step = float(nchild) / float(nSub);
        S.target[tid] = (long long)size_t(float(size_t(tid)) * step);
    }
    if (tid < 16) S.mods[kRawPool + tid] = 255;
    __syncthreads();
    {
        // the targets taken: a prefix of them
        const bool take = tid <= kLmedsMaxPts && S.target[tid] < nchild && (tid == 0 || S.target[tid] > S.target[tid - 1]);
        const unsigned m = __ballot_sync(kFull, take);
        if (lane == 0) S.warpCnt[0][warp] = m == kFull ? 32 : __ffs(~m) - 1;
    }
    if (tid == 0) {
        for (int k = 0; k < 9; ++k) S.bestQ[k] = 0.f;
        S.sm = 10000000.0f;
        S.done = 0;
        S.counter = 0;
        S.draws = 0;
        S.state = rng0.state;
        S.inc = rng0.inc;
    }
    __syncthreads();
    int np = 0;
    for (int w = 0; w < kFilterThreads / 32; ++w) {
        np += S.warpCnt[0][w];
        if (S.warpCnt[0][w] < 32) break;
    }
    if (np > kLmedsMaxPts) {
        if (tid == 0) atomicOr(err, kLoopOneErrPoints);
        return 0;
    }
    if (tid < np) {
        const int e = children[S.target[tid]];
        S.pts[tid] = {float(px_(L, e)), float(py_(L, e))};
        S.wts[tid] = 255.f / gnorm(L, e);
    }
    __syncthreads();
    // ... then random 5-point conics, 128 draws at a time, accepted in order.
    const uint32_t rejectBelow = uint32_t(-uint32_t(np)) % uint32_t(np);
    for (bool first = true; !S.done; first = false) {
        // the next kRawPool outputs of the candidate's stream, 8 per thread.
        // A bounded draw rejects an output only below 2^32 mod np (< 64 of
        // 2^32 values).
        bool rejects = false;
        {
            geo::Pcg32 g;
            g.state = S.state;
            g.inc = S.inc;
            g.advance(uint64_t(tid) * kRawPer);
            uint32_t packed[2] = {0u, 0u};
#pragma unroll
            for (int k = 0; k < kRawPer; ++k) {
                const uint32_t r = g.next();
                S.raws[tid * kRawPer + k] = r;
                packed[k >> 2] |= (r % uint32_t(np)) << (8 * (k & 3));
                rejects = rejects || r < rejectBelow;
            }
            *reinterpret_cast<uint2*>(S.mods + tid * kRawPer) = make_uint2(packed[0], packed[1]);
        }
        rejects = __syncthreads_or(rejects);
        if (!rejects) {
            lmeds_draws(S);
        } else if (tid == 0) {
            int ptr = 0, nd = 0;
            while (nd < kFilterThreads) {
                int perm[5] = {-1, -1, -1, -1, -1};
                const int start = ptr;
                bool complete = true;
                for (int i = 0; i < 5 && complete; ++i) {
                    for (;;) {
                        if (ptr >= kRawPool) {
                            complete = false;
                            break;
                        }
                        const uint32_t raw = S.raws[ptr];
                        const int r = S.mods[ptr];
                        ++ptr;
                        if (raw < rejectBelow) continue;
                        bool seen = false;
                        for (int q = 0; q < i; ++q) seen = seen || perm[q] == r;
                        if (seen) continue;
                        perm[i] = r;
                        break;
                    }
                }
                if (!complete) {
                    ptr = start;
                    break;
                }
                for (int i = 0; i < 5; ++i) S.perms[nd][i] = int8_t(perm[i]);
                ++nd;
            }
            S.nd = nd;
            geo::Pcg32 g;
            g.state = S.state;
            g.inc = S.inc;
            g.advance(uint64_t(ptr));
            S.state = g.state;
        }
        __syncthreads();
        const int nd = S.nd;
        if (nd == 0) {
            if (tid == 0) atomicOr(err, kLoopOneErrRandom);
            break;
        }
        geo::Mat3 Q = geo::Mat3::zero();
        int kind = kDrawNotReal;
        if (tid < nd) {
            int perm[5];
            for (int i = 0; i < 5; ++i) perm[i] = S.perms[tid][i];
            kind = cand::lmeds_conic(S.pts, perm, Q);
            S.kinds[tid] = kind;
            S.svals[tid] = 0.f;
#pragma unroll
            for (int k = 0; k < 9; ++k) S.Q[tid][k] = Q.m[k / 3][k % 3];
        }
        __syncthreads();
        float bound = S.sm;
        if (first) {
            for (int d = warp; d < min(nd, kFirstMedians); d += kFilterThreads / 32)
                if (S.kinds[d] == kDrawUsable) {
                    const float med = lmeds_median(S, d, np, weighted, lane);
                    if (lane == 0) S.svals[d] = med;
                }
            __syncthreads();
            for (int d = 0; d < min(nd, kFirstMedians); ++d)
                if (S.kinds[d] == kDrawUsable) bound = fminf(bound, S.svals[d]);
        }
        // the draws that may improve: more than half of their distances are
        // below a median that comes before them
        bool needS = false;
        if (kind == kDrawUsable && tid < nd && !(first && tid < kFirstMedians)) {
            needS = count_below(Q, S.pts, S.wts, np, weighted, bound) >= np / 2 + 1;
            if (!needS) S.kinds[tid] = kDrawNoGain;
        }
        __syncwarp();
        for (unsigned m = __ballot_sync(kFull, needS); m; m &= m - 1) {
            const int d = warp * 32 + __ffs(m) - 1;
            const float med = lmeds_median(S, d, np, weighted, lane);
            if (lane == 0) S.svals[d] = med;
        }
        __syncthreads();
        // Acceptance in draw order (Vote.cpp:478-545) by warp 0, 32 draws at a
        // time: draw j improves when its median is below the best before it,
        // which is the minimum of the carried best and every usable median
        // before j; the no-gain counter restarts at each improvement, and the
        // loop stops before the first draw at which it has reached 70 (or the
        // draws 7000).
        if (warp == 0) {
            int counter = S.counter, draws = S.draws, best = -1;
            float Sm = S.sm;
            bool stopped = false;
            for (int c0 = 0; c0 < nd && !stopped; c0 += 32) {
                const int j = c0 + lane;
                const bool valid = j < nd;
                const int kind = valid ? S.kinds[j] : kDrawNotReal;
                const bool usable = valid && kind == kDrawUsable;
                const float Sj = usable ? S.svals[j] : __int_as_float(0x7f800000);
                float incl = Sj;
                for (int o = 1; o < 32; o <<= 1) {
                    const float v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl = fminf(incl, v);
                }
                float excl = __shfl_up_sync(kFull, incl, 1);
                if (lane == 0) excl = __int_as_float(0x7f800000);
                const bool improving = usable && Sj < fminf(Sm, excl);
                const bool counted = valid && (kind == kDrawFail || kind == kDrawNoGain || (usable && !improving));
                const unsigned impM = __ballot_sync(kFull, improving);
                const unsigned cntM = __ballot_sync(kFull, counted);
                const unsigned lower = (1u << lane) - 1u;
                const unsigned impBefore = impM & lower;
                int cb;
                if (impBefore) {
                    const int last = 31 - __clz(impBefore);
                    cb = __popc(cntM & lower & ~((2u << last) - 1u));
                } else {
                    cb = counter + __popc(cntM & lower);
                }
                const bool stopHere = valid && !(cb < 70 && draws + lane < 7000);
                const unsigned stopM = __ballot_sync(kFull, stopHere);
                const int n = min(nd - c0, 32);
                const int js = stopM ? __ffs(stopM) - 1 : n;
                const unsigned proc = js >= 32 ? 0xffffffffu : ((1u << js) - 1u);
                const unsigned impP = impM & proc;
                if (impP) {
                    const int last = 31 - __clz(impP);
                    best = c0 + last;
                    Sm = __shfl_sync(kFull, Sj, last);
                    counter = __popc(cntM & proc & ~((2u << last) - 1u));
                } else {
                    counter += __popc(cntM & proc);
                }
                draws += js;
                stopped = stopM != 0;
            }
            if (best >= 0 && lane < 9) S.bestQ[lane] = S.Q[best][lane];
            if (lane == 0) {
                S.counter = counter;
                S.draws = draws;
                S.sm = Sm;
                if (stopped || !(counter < 70 && draws < 7000)) S.done = 1;
            }
        }
        __syncthreads();
    }
    // the children whose weighted distance is below threshold * median, in
    // order, four per thread at once so that their loads overlap
    geo::Mat3 Q;
    for (int k = 0; k < 9; ++k) Q.m[k / 3][k % 3] = S.bestQ[k];
    const float thr = threshold * S.sm;
    int nflt = 0;
    for (int c0 = 0; c0 < nchild; c0 += 4 * kFilterThreads) {
        int e[4];
        bool pass[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int i = c0 + h * kFilterThreads + tid;
            e[h] = i < nchild ? children[i] : -1;
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            pass[h] = false;
            if (e[h] >= 0) {
                float d = geo::dist_point_ellipse(Q, float(px_(L, e[h])), float(py_(L, e[h])));
                if (weighted) d = d * 255 / gnorm(L, e[h]);
                pass[h] = d < thr;
            }
        }
        unsigned mask[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            mask[h] = __ballot_sync(kFull, pass[h]);
            if (lane == 0) S.warpCnt[h][warp] = __popc(mask[h]);
        }
        __syncthreads();  // and every element of the chunk read before any is overwritten
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            int off = nflt;
            for (int w = 0; w < kFilterThreads / 32; ++w) {
                const int c = S.warpCnt[h][w];
                off += w < warp ? c : 0;
                nflt += c;
            }
            if (pass[h]) children[off + __popc(mask[h] & ((1u << lane) - 1u))] = e[h];
        }
        __syncthreads();
    }
    return nflt;
}


__global__ void __launch_bounds__(kFilterThreads) k_filter(LoopOneArgs a)
{
    const int l = blockIdx.x / a.n2max, rank = blockIdx.x % a.n2max;
    const LoopOneLevel& L = a.lv[l];
    const int tid = threadIdx.x, lane = tid & 31;
    const int madeCount = a.meta[size_t(a.nl) * a.n2max * 4 + l];
    if (rank >= min(madeCount, a.n2max)) return;
    int32_t* meta = a.meta + (size_t(l) * a.n2max + rank) * 4;
    const int s = meta[0];
    const int t = L.slot0 + s;
    const int32_t* info = a.sinfo + size_t(t) * 4;
    const int nf = info[0], nb = info[1];
    const int32_t* segc = a.seg + size_t(t) * kSegSlot + kSegHalf;
    const int len = nf + 1 + nb;
    int32_t* children = a.children + size_t(blockIdx.x) * a.childCap;
    if (threadIdx.x == 0) a.cflow[blockIdx.x] = L.flow[L.order[s]];

    // children (Vote.cpp:396-412): voters of the points with >= voteMax/14
    // votes, in segment order: each thread takes two neighbouring points, and
    // child o belongs to the last point whose offset is at most o
    __shared__ int sWarp[32], sOff[2 * kFilterThreads], sBase[2 * kFilterThreads], sMax;
    static_assert(kSegSlot <= 2 * kFilterThreads, "two points per thread");
    if (tid == 0) sMax = 1;
    __syncthreads();
    int base[2] = {0, 0}, cnt[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (2 * tid + h < len) {
            const int e = segc[-nf + 2 * tid + h];
            base[h] = L.voff[e];
            cnt[h] = L.voff[e + 1] - base[h];
        }
    const int vmx = __reduce_max_sync(kFull, max(cnt[0], cnt[1]));
    if (lane == 0) atomicMax(&sMax, vmx);
    __syncthreads();
    const int vmax = sMax;
#pragma unroll
    for (int h = 0; h < 2; ++h)
        if (cnt[h] < vmax / 14) cnt[h] = 0;
    int nchild;
    const int incl = block_inclusive(cnt[0] + cnt[1], sWarp, nchild);
    sOff[2 * tid] = incl - cnt[0] - cnt[1];
    sOff[2 * tid + 1] = incl - cnt[1];
    sBase[2 * tid] = base[0];
    sBase[2 * tid + 1] = base[1];
    __syncthreads();
    for (int o = tid; o < min(nchild, a.childCap); o += kFilterThreads) {
        int w = 0;
#pragma unroll
        for (int h = kFilterThreads; h > 0; h >>= 1)
            if (sOff[w + h] <= o) w += h;
        children[o] = L.vlist[sBase[w] + (o - sOff[w])];
    }
    __syncthreads();
    if (nchild > a.childCap) {
        if (tid == 0) {
            atomicOr(a.err, kLoopOneErrChildren);
            meta[0] = L.order[s];
            meta[1] = nchild;
            meta[2] = 0;
            meta[3] = 0;
        }
        return;
    }
    if (nchild < a.minPoints) {
        if (tid == 0) {
            meta[0] = L.order[s];
            meta[1] = 0;
            meta[2] = 0;
            meta[3] = 0;
        }
        return;
    }

    // outlierRemoval with inverse-gradient weights (Detection.cpp:131-133)
    const int nflt = lmeds_outliers(L, children, nchild, true, a.threshold,
                                    cand::candidate_rng(L.level, uint64_t(rank), 0), a.err);
    if (tid == 0) {
        meta[0] = L.order[s];
        meta[1] = nchild;
        meta[2] = nflt >= 5 ? 1 : 0;
        meta[3] = nflt;
    }
}

// float -> int as the host's conversion does it on x86-64: out of range and
// NaN give INT_MIN (the device instruction would saturate instead).
__device__ __forceinline__ int host_int(float f)
{
    return (f >= -2147483648.0f && f < 2147483648.0f) ? int(f) : int(0x80000000u);
}

// Multiresolution.cpp:43-142 intersectLineToTwoEllipses for row y: whether the
// row counts, and up to two x ranges to scan.
__device__ bool refit_row(const geo::Mat3& Qi, const geo::Mat3& Qo, int W, int y, int& nr, int xb[2], int xe[2])
{
    float io[2], ii[2];
    const int no = geo::intersect_line_q(Qo, float(y), true, io);
    const int ni = geo::intersect_line_q(Qi, float(y), true, ii);
    nr = 0;
    if (no == 2 && ni == 2) {
        nr = 2;
        xb[0] = max(0, host_int(io[0]));
        xe[0] = min(W - 1, host_int(ii[0]));
        xb[1] = max(0, host_int(ii[1]));
        xe[1] = min(W - 1, host_int(io[1]));
    } else if (no == 2 && ni <= 1) {
        nr = 1;
        xb[0] = max(0, host_int(io[0]));
        xe[0] = min(W - 1, host_int(io[1]));
    } else if (no == 1 && ni == 0) {
        if (io[0] >= 0 && io[0] < float(W)) {
            nr = 1;
            xb[0] = xe[0] = host_int(io[0]);
        }
    } else {
        return false;
    }
    return true;
}

// Multiresolution.cpp:319-401: level-0 hull of one coarse-level marker (rows
// from the center row down the image until one misses the hull, then from
// the center row up), one block per marker: 8 lanes per row, 128 rows at once,
// each lane a contiguous part of the row's bitmap words, which it reads twice
// (counting, then writing past a block scan of the counts: the second time
// from L1), so that the points keep the order of rows and columns.
// Measured (13 markers of a 1080p frame, cold): 18 us here and 46 us in the
// outlier removal, 125 us with a thread per run of rows in the removal's block
// of 128 threads (43 markers of a 3840x2160 clutter frame: 27 + 62 us, 188 us).
constexpr int kHullThreads = 1024;
constexpr int kHullLanes = 8;
__global__ void __launch_bounds__(kHullThreads) k_refit_hull(LoopOneLevel L, const RefitTask* tasks, int32_t* hullAll,
                                                             int hullCap, int32_t* counts)
{
    const int b = blockIdx.x, tid = threadIdx.x;
    const RefitTask& T = tasks[b];
    int32_t* hull = hullAll + size_t(b) * hullCap;
    geo::Mat3 Qi, Qo;
    for (int k = 0; k < 9; ++k) {
        Qi.m[k / 3][k % 3] = T.qin[k];
        Qo.m[k / 3][k % 3] = T.qout[k];
    }
    const int maxY = max(host_int(T.yc), 0);
    const int minY = min(host_int(T.yc), L.H - 1);
    __shared__ int sUpEnd, sDownEnd, sWarp[32];
    if (tid == 0) {
        sUpEnd = L.H;
        sDownEnd = -1;
    }
    __syncthreads();
    int nr, xb[2], xe[2];
    for (int y = maxY + tid; y < L.H; y += kHullThreads)
        if (!refit_row(Qi, Qo, L.W, y, nr, xb, xe)) atomicMin(&sUpEnd, y);
    for (int y = minY - tid; y >= 0; y -= kHullThreads)
        if (!refit_row(Qi, Qo, L.W, y, nr, xb, xe)) atomicMax(&sDownEnd, y);
    __syncthreads();
    const int rUp = max(sUpEnd - maxY, 0), rDown = max(minY - sDownEnd, 0);
    const int R = rUp + rDown;
    const int j = tid % kHullLanes;
    int total = 0;
    for (int r0 = 0; r0 < R; r0 += kHullThreads / kHullLanes) {
        const int r = r0 + tid / kHullLanes;
        const int y = r < rUp ? maxY + r : minY - (r - rUp);
        // this lane's words [t0, t1) of the row's: w[0] words of the first x
        // range, then those of the second
        int w[2] = {0, 0}, t0 = 0, t1 = 0;
        if (r < R && refit_row(Qi, Qo, L.W, y, nr, xb, xe)) {
            for (int q = 0; q < nr; ++q)
                if (xb[q] <= xe[q]) w[q] = (xe[q] >> 5) - (xb[q] >> 5) + 1;
            const int per = (w[0] + w[1] + kHullLanes - 1) / kHullLanes;
            t0 = min(j * per, w[0] + w[1]);
            t1 = min(t0 + per, w[0] + w[1]);
        }
        // the edge points of those words that are taken into the hull, in x
        // order; f(e) is called for each
        auto each = [&](auto&& f) {
            const uint2* row = L.bitidx + size_t(y) * L.WW;
            for (int t = t0; t < t1; ++t) {
                const int q = t < w[0] ? 0 : 1;
                const int wx = (xb[q] >> 5) + t - (q ? w[0] : 0), lo = wx << 5;
                const uint2 word = row[wx];
                uint32_t m = word.x;
                if (xb[q] > lo) m &= 0xffffffffu << (xb[q] - lo);
                if (xe[q] < lo + 31) m &= 0xffffffffu >> (31 - (xe[q] - lo));
                for (; m; m &= m - 1) {
                    const int bit = __ffs(m) - 1;
                    const int e = int(word.y) + __popc(word.x & ((1u << bit) - 1u));
                    if (e >= L.E) break;  // past a clamped edge count
                    const float cx = T.inCx - float(lo + bit), cy = T.inCy - float(y);
                    if (gdx(L, e) * cx + gdy(L, e) * cy < 0) f(e);
                }
            }
        };
        int n = 0;
        each([&](int) { ++n; });
        int sum;
        int off = total + block_inclusive(n, sWarp, sum) - n;
        total += sum;
        if (total <= hullCap)
            each([&](int e) { hull[off++] = e; });
    }
    if (tid == 0) {
        if (total > hullCap) atomicOr(counts + gridDim.x, kLoopOneErrChildren);
        counts[b] = total > hullCap || total < 5 ? -1 : total;
    }
}

// ... then the outlier removal without weights.
__global__ void __launch_bounds__(kFilterThreads) k_refit(LoopOneLevel L, const RefitTask* tasks, int32_t* hullAll,
                                                        int hullCap, int32_t* counts)
{
    const int b = blockIdx.x;
    const int total = counts[b];
    if (total < 5) return;
    const geo::Pcg32 rng(271828, (uint64_t(1) << 62) | uint64_t(tasks[b].marker));
    const int nflt =
        lmeds_outliers(L, hullAll + size_t(b) * hullCap, total, false, 20.0f, rng, counts + gridDim.x);
    if (threadIdx.x == 0) counts[b] = nflt;
}

__global__ void __launch_bounds__(256) k_refit_pack(const int32_t* hullAll, int hullCap, const int32_t* counts,
                                                    int32_t* packed)
{
    const int b = blockIdx.x;
    __shared__ int sOff;
    const int n = counts[b];
    if (n <= 0) return;
    if (threadIdx.x == 0) {
        int off = 0;
        for (int q = 0; q < b; ++q) off += max(counts[q], 0);
        sOff = off;
    }
    __syncthreads();
    const int32_t* src = hullAll + size_t(b) * hullCap;
    for (int i = threadIdx.x; i < n; i += blockDim.x) packed[sOff + i] = src[i];
}

// Kept candidates' filtered children, in candidate order, into one array.
// The link chains of the packed filtered children: point i of level l (the
// levels' entries are contiguous, from first[l]) walks len alternating
// before / after links, as addCandidateFlowtoCCTag does (EllipseGrowing.cpp:
// 63-178).
struct ChainLevels {
    const int32_t* before[kMaxLevels];
    const int32_t* after[kMaxLevels];
    int first[kMaxLevels + 1];
};

__global__ void __launch_bounds__(256) k_chains(const int32_t* __restrict__ packed, int total, int len,
                                                ChainLevels cl, int nl, int32_t* __restrict__ chain)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int l = 0;
    while (l < nl - 1 && i >= cl.first[l + 1]) ++l;
    int q = packed[i];
    for (int j = 0; j < len; ++j) {
        q = q < 0 ? -1 : (j & 1) ? cl.after[l][q] : cl.before[l][q];
        chain[size_t(i) * len + j] = q;
    }
}

__global__ void __launch_bounds__(256) k_pack(LoopOneArgs a, int32_t* packed)
{
    const int b = blockIdx.x;
    const int l = b / a.n2max, rank = b % a.n2max;
    __shared__ int sOff;
    const int n2 = min(a.meta[size_t(a.nl) * a.n2max * 4 + l], a.n2max);
    if (rank >= n2) return;
    const int32_t* meta = a.meta + size_t(b) * 4;
    if (!meta[2]) return;
    // the kept candidates before this one: a block sum (one thread adding up to
    // b dependent loads took 18 us on a 1080p frame)
    int before = 0;
    for (int q = threadIdx.x; q < b; q += blockDim.x) {
        const int lq = q / a.n2max, rq = q % a.n2max;
        const int n2q = min(a.meta[size_t(a.nl) * a.n2max * 4 + lq], a.n2max);
        if (rq < n2q && a.meta[size_t(q) * 4 + 2]) before += a.meta[size_t(q) * 4 + 3];
    }
    if (threadIdx.x == 0) sOff = 0;
    __syncthreads();
    before = __reduce_add_sync(kFull, before);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sOff, before);
    __syncthreads();
    const int32_t* src = a.children + size_t(b) * a.childCap;
    for (int i = threadIdx.x; i < meta[3]; i += blockDim.x) packed[sOff + i] = src[i];
}

template <class T>
T* dev_alloc(std::vector<void*>& list, size_t n)
{
    void* p = nullptr;
    CCTAGB_CUDA(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
    list.push_back(p);
    return static_cast<T*>(p);
}

}  // namespace

LoopOneGpu::LoopOneGpu(const cctagb_params& p, int max_h, const std::vector<int>& caps) : p_(p)
{
    if (p.windowSizeOnInnerEllipticSegment < 1 || p.windowSizeOnInnerEllipticSegment > cand::kLinkMaxWindow)
        throw Error{CCTAGB_BAD_ARG, "windowSizeOnInnerEllipticSegment must be in [1, 64]"};
    if (p.maximumNbCandidatesLoopTwo < 1 || p.maximumNbCandidatesLoopTwo > 1024)
        throw Error{CCTAGB_BAD_ARG, "maximumNbCandidatesLoopTwo must be in [1, 1024]"};
    nl_ = int(caps.size());
    n2max_ = p.maximumNbCandidatesLoopTwo;
    waiter_.init(p.hostSpinMicros);
    // seeds processed per level: max(rows / 2, maximumNbSeeds) (Detection.cpp:603-605);
    // level 0 has the most rows
    maxSlotsPerLevel_ = std::max(max_h / 2, p.maximumNbSeeds);
    maxH_ = max_h;
    totalSlots_ = nl_ * maxSlotsPerLevel_;
    size_t nrec = 0;
    for (int l = 0; l < nl_; ++l) {
        caps_.push_back(caps[size_t(l)]);
        nrec += size_t(caps[size_t(l)]);
    }
    args_.seg = dev_alloc<int32_t>(allocs_, size_t(totalSlots_) * kSegSlot);
    args_.sinfo = dev_alloc<int32_t>(allocs_, size_t(totalSlots_) * 4);
    args_.mlist = dev_alloc<int32_t>(allocs_, size_t(totalSlots_) * kMarkCap);
    args_.skey = dev_alloc<float>(allocs_, size_t(totalSlots_));
    args_.made = dev_alloc<int32_t>(allocs_, size_t(totalSlots_));
    const size_t metaN = size_t(nl_) * n2max_ * 4 + nl_ + 1;
    args_.meta = dev_alloc<int32_t>(allocs_, metaN);
    args_.cflow = dev_alloc<float>(allocs_, size_t(nl_) * n2max_);
    args_.err = args_.meta + size_t(nl_) * n2max_ * 4 + nl_;

    d_order_ = dev_alloc<int32_t>(allocs_, size_t(totalSlots_));
    d_rec_ = dev_alloc<int4>(allocs_, nrec * 3);
    for (int l = 0; l < nl_; ++l) maxCap_ = std::max(maxCap_, size_t(caps[size_t(l)]));
    grow_children(std::min<size_t>(kChildCap, maxCap_ + 1));
    CCTAGB_CUDA(cudaMallocHost(&h_order_, sizeof(int32_t) * std::max(totalSlots_, 1)));
    CCTAGB_CUDA(cudaMallocHost(&h_meta_, sizeof(int32_t) * metaN));
    CCTAGB_CUDA(cudaMallocHost(&h_cflow_, sizeof(float) * size_t(nl_) * n2max_));
    h_flt_cap_ = size_t(nl_) * n2max_ * 512;
    CCTAGB_CUDA(cudaMallocHost(&h_flt_, sizeof(int32_t) * h_flt_cap_));
    args_.maxSlotsPerLevel = maxSlotsPerLevel_;
    args_.totalSlots = totalSlots_;
    args_.nl = nl_;
    args_.window = p.windowSizeOnInnerEllipticSegment;
    args_.averageVoteMin = p.averageVoteMin;
    args_.n2max = n2max_;
    args_.minPoints = p.minPointsSegmentCandidate;
    args_.threshold = p.threshRobustEstimationOfOuterEllipse;
    // The attribute is per kernel and shared by every handle: set it to what
    // the device allows, so that no handle lowers it below another's need.
    int dev = 0, optin = 0;
    CCTAGB_CUDA(cudaGetDevice(&dev));
    CCTAGB_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const int maxSmem = optin - 1024;  // room for the kernel's static shared memory
    if (resolve_smem() > maxSmem)
        throw Error{CCTAGB_BAD_ARG, "maximumNbSeeds / frame height too large for the loop-one resolve kernel"};
    CCTAGB_CUDA(cudaFuncSetAttribute(k_link_resolve, cudaFuncAttributeMaxDynamicSharedMemorySize, maxSmem));
}

int LoopOneGpu::resolve_smem() const
{
    return int(sizeof(int) * (3 * size_t(maxSlotsPerLevel_) + 1) + sizeof(uint16_t) * kResolveSmemMarks);
}

LoopOneGpu::~LoopOneGpu()
{
    for (void* q : allocs_) cudaFree(q);
    if (args_.children) cudaFree(args_.children);
    if (d_packed_) cudaFree(d_packed_);
    for (void* q : {static_cast<void*>(d_rtask_), static_cast<void*>(d_rhull_), static_cast<void*>(d_rcount_), static_cast<void*>(d_rpacked_)})
        if (q) cudaFree(q);
    if (h_rtask_) cudaFreeHost(h_rtask_);
    if (h_rcount_) cudaFreeHost(h_rcount_);
    if (h_rpacked_) cudaFreeHost(h_rpacked_);
    if (h_order_) cudaFreeHost(h_order_);
    if (h_meta_) cudaFreeHost(h_meta_);
    if (h_cflow_) cudaFreeHost(h_cflow_);
    if (h_flt_) cudaFreeHost(h_flt_);
    if (d_chain_) cudaFree(d_chain_);
    if (h_chain_) cudaFreeHost(h_chain_);
}

void LoopOneGpu::launch(const Levels& lv, const int* E, const std::vector<const std::vector<int32_t>*>& seeds,
                        cudaStream_t s)
{
    if (lv.n != nl_ || int(seeds.size()) != nl_) throw Error{CCTAGB_BAD_ARG, "loop one: level count changed"};
    h2d_ = d2h_ = 0;
    size_t roff = 0;
    int cum[kMaxLevels] = {};
    for (int l = 0; l < nl_; ++l) {
        const LevelView& v = lv.l[l];
        LoopOneLevel& L = args_.lv[l];
        L.W = v.W;
        L.H = v.H;
        L.WW = v.WW;
        L.E = E[l];
        L.exy = v.exy;
        L.grad = v.grad;
        L.voff = v.voff;
        L.vlist = v.vlist;
        L.bitidx = v.bitidx;
        L.before = v.before;
        L.after = v.after;
        L.flow = v.flow;
        L.level = l;
        L.slot0 = l * maxSlotsPerLevel_;
        const size_t nMax = size_t(std::max(v.H / 2, p_.maximumNbSeeds));
        L.nProc = int(std::min(seeds[l]->size(), nMax));
        L.order = d_order_ + L.slot0;
        std::copy(seeds[l]->begin(), seeds[l]->begin() + L.nProc, h_order_ + L.slot0);
        if (v.cap > caps_[size_t(l)]) throw Error{CCTAGB_INTERNAL, "loop one: level capacity changed"};
        if (E[l] > caps_[size_t(l)]) throw Error{CCTAGB_INTERNAL, "loop one: more edge points than capacity"};
        L.rec = d_rec_ + 3 * roff;
        roff += size_t(caps_[size_t(l)]);
        cum[l] = (l ? cum[l - 1] : 0) + E[l];
        if (L.nProc)
            CCTAGB_CUDA(cudaMemcpyAsync(d_order_ + L.slot0, h_order_ + L.slot0, sizeof(int32_t) * L.nProc,
                                        cudaMemcpyHostToDevice, s));
        h2d_ += 4LL * L.nProc;
    }
    for (int l = nl_; l < kMaxLevels; ++l) cum[l] = cum[nl_ - 1];
    cum_ = make_int4(cum[0], cum[1], cum[2], cum[3]);
    run_kernels(s);
}

void LoopOneGpu::grow_children(size_t cap)
{
    if (args_.children) cudaFree(args_.children);
    if (d_packed_) cudaFree(d_packed_);
    args_.children = nullptr;
    d_packed_ = nullptr;
    args_.childCap = 0;
    const size_t n = size_t(nl_) * n2max_ * cap;
    CCTAGB_CUDA(cudaMalloc(&args_.children, sizeof(int32_t) * n));
    CCTAGB_CUDA(cudaMalloc(&d_packed_, sizeof(int32_t) * n));
    args_.childCap = int(cap);
}

void LoopOneGpu::run_kernels(cudaStream_t s)
{
    const size_t metaN = size_t(nl_) * n2max_ * 4 + nl_ + 1;
    CCTAGB_CUDA(cudaMemsetAsync(args_.meta, 0, sizeof(int32_t) * metaN, s));
    const int cumv[kMaxLevels] = {cum_.x, cum_.y, cum_.z, cum_.w};
    const int npts = nl_ > 0 ? cumv[nl_ - 1] : 0;
    if (npts > 0) {
        k_point_records<<<(npts + 255) / 256, 256, 0, s>>>(args_, cum_);
        CCTAGB_CUDA(cudaGetLastError());
    }
    k_seed_slots<<<(totalSlots_ + 255) / 256, 256, 0, s>>>(args_);
    CCTAGB_CUDA(cudaGetLastError());
    k_link_seeds<<<(totalSlots_ + kLinkGroups - 1) / kLinkGroups, kLinkThreads, 0, s>>>(args_);
    CCTAGB_CUDA(cudaGetLastError());
    k_link_resolve<<<nl_, kResolveThreads, resolve_smem(), s>>>(args_);
    CCTAGB_CUDA(cudaGetLastError());
    k_filter<<<nl_ * n2max_, kFilterThreads, 0, s>>>(args_);
    CCTAGB_CUDA(cudaGetLastError());
    k_pack<<<nl_ * n2max_, 256, 0, s>>>(args_, d_packed_);
    CCTAGB_CUDA(cudaGetLastError());
    CCTAGB_CUDA(cudaMemcpyAsync(h_meta_, args_.meta, sizeof(int32_t) * metaN, cudaMemcpyDeviceToHost, s));
    CCTAGB_CUDA(cudaMemcpyAsync(h_cflow_, args_.cflow, sizeof(float) * size_t(nl_) * n2max_,
                                cudaMemcpyDeviceToHost, s));
    d2h_ += 4LL * metaN + 4LL * nl_ * n2max_;
}

void LoopOneGpu::collect(cudaStream_t s, std::vector<LoopTwoIn>& out)
{
    chainLaunches_ = 0;
    waiter_.wait(s);
    const int32_t* made = h_meta_ + size_t(nl_) * n2max_ * 4;
    // a candidate with more voters than the room: more room, same kernels
    // (no list can hold more points than its level)
    while ((made[nl_] & kLoopOneErrChildren) && size_t(args_.childCap) <= maxCap_) {
        grow_children(std::min(size_t(args_.childCap) * 4, maxCap_ + 1));
        run_kernels(s);
        waiter_.wait(s);
    }
    const int err = made[nl_];
    if (err & kLoopOneErrChildren)
        throw Error{CCTAGB_OVERFLOW_VOTERS, "a loop-two candidate gathers more voters than its level has points"};
    if (err) throw Error{CCTAGB_INTERNAL, "loop one: error bits " + std::to_string(err)};
    size_t total = 0;
    for (int l = 0; l < nl_; ++l) {
        const int n2 = std::min(made[l], n2max_);
        for (int r = 0; r < n2; ++r) {
            const int32_t* m = h_meta_ + (size_t(l) * n2max_ + r) * 4;
            if (m[2]) total += size_t(m[3]);
        }
    }
    if (total > h_flt_cap_) {
        cudaFreeHost(h_flt_);
        h_flt_ = nullptr;
        h_flt_cap_ = 0;
        CCTAGB_CUDA(cudaMallocHost(&h_flt_, sizeof(int32_t) * total));
        h_flt_cap_ = total;
    }
    // the link chains of the filtered children (the host's flow assembling
    // walks them; the links themselves stay on the device)
    const int len = 2 * p_.nCrowns - 1;
    ChainLevels cl{};
    {
        size_t off = 0;
        for (int l = 0; l < nl_; ++l) {
            cl.before[l] = args_.lv[l].before;
            cl.after[l] = args_.lv[l].after;
            cl.first[l] = int(off);
            const int n2 = std::min(made[l], n2max_);
            for (int r = 0; r < n2; ++r) {
                const int32_t* m = h_meta_ + (size_t(l) * n2max_ + r) * 4;
                if (m[2]) off += size_t(m[3]);
            }
        }
        cl.first[nl_] = int(off);
    }
    if (total * len > chain_cap_) {
        if (d_chain_) cudaFree(d_chain_);
        if (h_chain_) cudaFreeHost(h_chain_);
        d_chain_ = nullptr;
        h_chain_ = nullptr;
        chain_cap_ = 0;
        const size_t cap = std::max(total * len, size_t(65536));
        CCTAGB_CUDA(cudaMalloc(&d_chain_, sizeof(int32_t) * cap));
        CCTAGB_CUDA(cudaMallocHost(&h_chain_, sizeof(int32_t) * cap));
        chain_cap_ = cap;
    }
    if (total) {
        k_chains<<<int((total + 255) / 256), 256, 0, s>>>(d_packed_, int(total), len, cl, nl_, d_chain_);
        CCTAGB_CUDA(cudaGetLastError());
        ++chainLaunches_;
        CCTAGB_CUDA(cudaMemcpyAsync(h_flt_, d_packed_, sizeof(int32_t) * total, cudaMemcpyDeviceToHost, s));
        CCTAGB_CUDA(cudaMemcpyAsync(h_chain_, d_chain_, sizeof(int32_t) * total * len, cudaMemcpyDeviceToHost, s));
        waiter_.wait(s);
    }
    d2h_ += 4LL * total * (1 + len);
    out.assign(size_t(nl_), {});
    size_t off = 0;
    for (int l = 0; l < nl_; ++l) {
        LoopTwoIn& o = out[size_t(l)];
        const int n2 = std::min(made[l], n2max_);
        o.chainLen = len;
        o.foff.push_back(0);
        for (int r = 0; r < n2; ++r) {
            const int32_t* m = h_meta_ + (size_t(l) * n2max_ + r) * 4;
            o.seed.push_back(m[0]);
            o.flow.push_back(h_cflow_[size_t(l) * n2max_ + r]);
            o.score.push_back(m[1]);
            o.keep.push_back(uint8_t(m[2]));
            if (m[2]) {
                o.flt.insert(o.flt.end(), h_flt_ + off, h_flt_ + off + m[3]);
                o.chain.insert(o.chain.end(), h_chain_ + off * len, h_chain_ + (off + m[3]) * len);
                off += size_t(m[3]);
            }
            o.foff.push_back(int32_t(o.flt.size()));
        }
    }
}

void LoopOneGpu::ensure_refit_capacity(int n)
{
    if (n <= refitCap_) return;
    for (void* q : {static_cast<void*>(d_rtask_), static_cast<void*>(d_rhull_), static_cast<void*>(d_rcount_), static_cast<void*>(d_rpacked_)})
        if (q) cudaFree(q);
    if (h_rtask_) cudaFreeHost(h_rtask_);
    if (h_rcount_) cudaFreeHost(h_rcount_);
    d_rtask_ = nullptr;
    d_rhull_ = d_rcount_ = d_rpacked_ = nullptr;
    h_rtask_ = nullptr;
    h_rcount_ = nullptr;
    refitCap_ = 0;
    const int cap = std::max(n, 64);
    CCTAGB_CUDA(cudaMalloc(&d_rtask_, sizeof(RefitTask) * cap));
    CCTAGB_CUDA(cudaMalloc(&d_rhull_, sizeof(int32_t) * size_t(cap) * hullCap_));
    CCTAGB_CUDA(cudaMalloc(&d_rcount_, sizeof(int32_t) * (cap + 1)));
    CCTAGB_CUDA(cudaMalloc(&d_rpacked_, sizeof(int32_t) * size_t(cap) * hullCap_));
    CCTAGB_CUDA(cudaMallocHost(&h_rtask_, sizeof(RefitTask) * cap));
    CCTAGB_CUDA(cudaMallocHost(&h_rcount_, sizeof(int32_t) * (cap + 1)));
    refitCap_ = cap;
}

void LoopOneGpu::refit(const Levels& lv, const std::vector<RefitTask>& tasks, cudaStream_t s,
                       std::vector<std::vector<int32_t>>& filtered)
{
    const int n = int(tasks.size());
    filtered.assign(size_t(n), {});
    if (n == 0) return;
    ensure_refit_capacity(n);
    const LevelView& v = lv.l[0];
    if (v.H > maxH_) throw Error{CCTAGB_INTERNAL, "refit: frame taller than the handle"};
    LoopOneLevel L = args_.lv[0];  // level-0 view of the frame loop one ran on
    std::copy(tasks.begin(), tasks.end(), h_rtask_);
    CCTAGB_CUDA(cudaMemcpyAsync(d_rtask_, h_rtask_, sizeof(RefitTask) * n, cudaMemcpyHostToDevice, s));
    // the hull of one marker holds at most every level-0 point and a row twice
    const size_t hullMax = size_t(L.E) + size_t(L.W) + 1;
    for (;;) {
        CCTAGB_CUDA(cudaMemsetAsync(d_rcount_ + n, 0, sizeof(int32_t), s));
        k_refit_hull<<<n, kHullThreads, 0, s>>>(L, d_rtask_, d_rhull_, hullCap_, d_rcount_);
        CCTAGB_CUDA(cudaGetLastError());
        k_refit<<<n, kFilterThreads, 0, s>>>(L, d_rtask_, d_rhull_, hullCap_, d_rcount_);
        CCTAGB_CUDA(cudaGetLastError());
        k_refit_pack<<<n, 256, 0, s>>>(d_rhull_, hullCap_, d_rcount_, d_rpacked_);
        CCTAGB_CUDA(cudaGetLastError());
        CCTAGB_CUDA(cudaMemcpyAsync(h_rcount_, d_rcount_, sizeof(int32_t) * (n + 1), cudaMemcpyDeviceToHost, s));
        waiter_.wait(s);
        if (!(h_rcount_[n] & kLoopOneErrChildren) || size_t(hullCap_) > hullMax) break;
        // more room for the hulls, same kernels
        hullCap_ = int(std::min(size_t(hullCap_) * 4, hullMax + 1));
        const int keep = refitCap_;
        refitCap_ = 0;
        ensure_refit_capacity(keep);
        std::copy(tasks.begin(), tasks.end(), h_rtask_);
        CCTAGB_CUDA(cudaMemcpyAsync(d_rtask_, h_rtask_, sizeof(RefitTask) * n, cudaMemcpyHostToDevice, s));
    }
    const int err = h_rcount_[n];
    if (err & kLoopOneErrChildren)
        throw Error{CCTAGB_OVERFLOW_VOTERS, "a re-fit hull holds more points than level 0"};
    if (err) throw Error{CCTAGB_INTERNAL, "refit: error bits " + std::to_string(err)};
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += size_t(std::max(h_rcount_[i], 0));
    if (total > h_rpacked_cap_) {
        if (h_rpacked_) cudaFreeHost(h_rpacked_);
        h_rpacked_ = nullptr;
        h_rpacked_cap_ = 0;
        CCTAGB_CUDA(cudaMallocHost(&h_rpacked_, sizeof(int32_t) * std::max<size_t>(total, 4096)));
        h_rpacked_cap_ = std::max<size_t>(total, 4096);
    }
    if (total) {
        CCTAGB_CUDA(cudaMemcpyAsync(h_rpacked_, d_rpacked_, sizeof(int32_t) * total, cudaMemcpyDeviceToHost, s));
        waiter_.wait(s);
    }
    h2d_ += (long long)sizeof(RefitTask) * n;
    d2h_ += 4LL * (n + 1) + 4LL * (long long)total;
    size_t off = 0;
    for (int i = 0; i < n; ++i) {
        const int c = std::max(h_rcount_[i], 0);
        filtered[size_t(i)].assign(h_rpacked_ + off, h_rpacked_ + off + c);
        off += size_t(c);
    }
}

}  // namespace cctagb
