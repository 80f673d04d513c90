// Cut collection and selection on the GPU (identify_step_1: geometry/
// Ellipse.cpp:259-300 getSortedOuterPoints, Identification.cpp:396-459
// cutInterpolated, :471-496 collectCuts, :546-601 selectCutCheapUniform,
// :604-709 outerEdgeRefinement / convImageCut; EllipseFromPoints.cpp:29-48
// pointOnEllipse), one thread block per marker.
//
// Every expression is the host restatement's, evaluated with explicit IEEE
// roundings in the same order (no contraction into FMAs; the file is built with
// --fmad=false for the double arithmetic of pmath's atan2), so the selected cut
// ends are the same bits as the host's.  The cosine and sine of the ellipse
// angle come from the host.
//
// The work is a chain of phases on few blocks, bound by the length of a
// thread's chain of instructions, so each phase is spread over the block: the
// sort over a key per thread, in registers within a warp's keys; a cut's
// samples over four lanes, which walk the running sums of its positions to
// their share and leave the values in shared memory; the running mean and
// variance, a chain by definition, a thread per cut, while other warps refine
// the cut ends, four lanes each.  Measured (28 markers of a 1080p frame, cold):
// one kernel sorting with 256 threads and one with a thread per cut 24 + 72 us,
// 40 us now (80 markers of a 3840x2160 clutter frame 48 + 82 us, 49 us).
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <string>

#include "common.hpp"
#include "ident_host.hpp"
#include "cctag_b200/portable/pmath.hpp"

namespace cctagb {

namespace {

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fd(float a, float b) { return __fdiv_rn(a, b); }

// Identification.hpp:197-219, as the host: ((p0 w1 + p1 w2) + p2 w3 + p3 w4) / 2
__device__ __forceinline__ float bilinear_host(const uint8_t* img, int W, float x, float y)
{
    const int px = int(x), py = int(y);
    const uint8_t* p0 = img + px + size_t(py) * W;
    const float fx = fs(x, float(px)), fy = fs(y, float(py));
    const float fx1 = fs(1.0f, fx), fy1 = fs(1.0f, fy);
    const float w1 = fm(fx1, fy1), w2 = fm(fx, fy1), w3 = fm(fx1, fy), w4 = fm(fx, fy);
    float t = fm(float(p0[0]), w1);
    t = fa(t, fm(float(p0[1]), w2));
    t = fa(t, fm(float(p0[W]), w3));
    t = fa(t, fm(float(p0[W + 1]), w4));
    return fm(t, 0.5f);  // the division by 2, exact
}

constexpr int kThreads = 1024;
constexpr int kRefineQuads = (kThreads - kMaxOuterPoints) / 4;
static_assert(kThreads == 4 * kMaxOuterPoints, "four lanes per cut");

// Samples [k0, k1) of cutInterpolated from (xs, ys) in steps of (stepX, stepY),
// the positions by the reference's running sums; false when one of them is not
// in [1, W-1) x [1, H-1).
__device__ __forceinline__ bool sample_cut(const uint8_t* img, int W, int H, float xs, float ys, float stepX,
                                           float stepY, int k0, int k1, float* out)
{
    float x = xs, y = ys;
#pragma unroll 5
    for (int k = 0; k < k0; ++k) {
        x = fa(x, stepX);
        y = fa(y, stepY);
    }
    bool inside = true;
    constexpr int kGroup = 5;  // samples whose reads overlap
    for (int i0 = k0; i0 < k1; i0 += kGroup) {
        float gx[kGroup], gy[kGroup];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
            gx[k] = x;
            gy[k] = y;
            if (i0 + k < k1) inside = inside && (x >= 1.f && x < float(W - 1) && y >= 1.f && y < float(H - 1));
            x = fa(x, stepX);
            y = fa(y, stepY);
        }
        if (!inside) break;
        float v[kGroup];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) v[k] = i0 + k < k1 ? bilinear_host(img, W, gx[k], gy[k]) : 0.f;
#pragma unroll
        for (int k = 0; k < kGroup; ++k)
            if (i0 + k < k1) out[i0 + k] = v[k];
    }
    return inside;
}

// Ascending bitonic sort of the block's m keys (a power of two, at most
// kCutSortCap), key e in thread e mod kThreads; s_key holds them at the end.
// Steps within 32 neighbouring keys by shuffles, the others through s_key.
__device__ void sort_keys(unsigned long long* s_key, unsigned long long (&v)[kCutSortCap / kThreads], int m)
{
    constexpr int kPer = kCutSortCap / kThreads;
    const int t = threadIdx.x;
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kPer; ++q)
                    if (q * kThreads < m) s_key[q * kThreads + t] = v[q];
                __syncthreads();
            }
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (q * kThreads < m) {
                    const int e = q * kThreads + t;
                    const unsigned long long o = j >= 32 ? s_key[e ^ j] : __shfl_xor_sync(0xffffffffu, v[q], j);
                    const bool low = ((e & j) == 0) == ((e & k) == 0);
                    v[q] = low == (o < v[q]) ? o : v[q];
                }
        }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; ++q)
        if (q * kThreads < m) s_key[q * kThreads + t] = v[q];
    __syncthreads();
}

// Values of the three derivative kernels of convImageCut (Identification.cpp:630-632).
__constant__ float cEdge[3][9] = {
    {-0.0000f, -0.0003f, -0.1065f, -0.7863f, .0f, 0.7863f, 0.1065f, 0.0003f, 0.0000f},
    {-0.0044f, -0.0540f, -0.2376f, -0.3450f, .0f, 0.3450f, 0.2376f, 0.0540f, 0.0044f},
    {-0.0366f, -0.1113f, -0.1801f, -0.1594f, .0f, 0.1594f, 0.1801f, 0.1113f, 0.0366f}};

}  // namespace

__global__ void __launch_bounds__(kThreads) k_cut_select(const uint8_t* __restrict__ img, int W, int H,
                                                         const CutSelectIn* __restrict__ ins,
                                                         const DirPoint* __restrict__ pts, IdentTask* tasks,
                                                         int* status, CutSelectParams cp)
{
    // the sort keys, then the cuts' samples (a row of sampleStride per cut) and
    // the refinement's (a row of refineStride per quad)
    extern __shared__ unsigned long long s_key[];
    __shared__ int16_t s_pick[kMaxOuterPoints];
    __shared__ float s_x[kMaxOuterPoints], s_y[kMaxOuterPoints], s_wmax[kMaxOuterPoints / 32];
    __shared__ float s_rcp[kMaxSamples + 1], s_edge[27];
    __shared__ int s_keep[kMaxOuterPoints], s_wcnt[kMaxOuterPoints / 32];
    __shared__ uint8_t s_ok[kMaxOuterPoints], s_ref[kMaxOuterPoints];
    const CutSelectIn in = ins[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    IdentTask& T = tasks[blockIdx.x];
    for (int i = t; i <= kMaxSamples; i += kThreads) s_rcp[i] = __frcp_rn(float(i));
    if (t < 27) s_edge[t] = cEdge[t / 9][t % 9];
    if (t < kMaxOuterPoints) s_ok[t] = s_ref[t] = 0;

    // ---- the outer points sorted by angle and subsampled
    int count;
    if (in.presorted) {  // the host sorted and subsampled them
        count = in.count;
        for (int k = t; k < count; k += kThreads) s_pick[k] = int16_t(k);
        __syncthreads();
    } else {
        const int n = in.count;  // <= kCutSortCap (the host presorts larger sets)
        int m = 1;
        while (m < n) m <<= 1;
        unsigned long long v[kCutSortCap / kThreads];
#pragma unroll
        for (int q = 0; q < kCutSortCap / kThreads; ++q) {
            const int e = q * kThreads + t;
            v[q] = ~0ull;
            if (e < n) {
                const DirPoint p = pts[in.first + e];
                const float a = pm::atan2f_(p.y - in.cy, p.x - in.cx);
                // (angle, index): a total order, so the reference's std::sort order
                v[q] = (unsigned long long)geo::order_key(a) << 32 | unsigned(e);
            }
        }
        sort_keys(s_key, v, m);
        // pick k is the sorted point int(k * step) while that is < n; nothing
        // with fewer than two points (the reference's step divides by zero)
        const int nOuter = min(cp.nOuter, n);
        bool pick = false;
        if (nOuter >= 2 && t < kMaxOuterPoints) {
            const float step = fmaxf(1.f, fd(float(n), float(nOuter - 1)));
            const int i = int(fm(float(t), step));
            pick = i < n;
            if (pick) s_pick[t] = int16_t(s_key[i] & 0xffffffffu);
        }
        // k * step reaches n before k = nOuter <= kMaxOuterPoints, and i grows with k
        count = __syncthreads_count(pick);
    }
    if (count < 5) {  // identify_step_1's TOO_FEW_OUTER_POINTS
        if (t == 0) {
            T.ncuts = 0;
            status[blockIdx.x] = CCTAGB_TOO_FEW_OUTER_POINTS;
        }
        return;
    }

    // ---- the cuts' samples, four lanes per cut
    float* const values = reinterpret_cast<float*>(s_key);
    const int sampleStride = cp.nSamples | 1, refineStride = cp.nRefine | 1;
    {
        const int i = t >> 2, q = t & 3;
        bool inside = false;
        if (i < count) {
            const DirPoint op = pts[in.first + s_pick[i]];
            const float dX = fs(op.x, in.cx), dY = fs(op.y, in.cy);
            float xs = in.cx, ys = in.cy;
            if (cp.beginSig != 0.f) {
                xs = fa(in.cx, fm(dX, cp.beginSig));
                ys = fa(in.cy, fm(dY, cp.beginSig));
            }
            const float den = fs(float(cp.nSamples), 1.f);
            const float stepX = fd(fs(op.x, xs), den), stepY = fd(fs(op.y, ys), den);
            const int seg = (cp.nSamples + 3) >> 2, k0 = min(q * seg, cp.nSamples), k1 = min(k0 + seg, cp.nSamples);
            inside = sample_cut(img, W, H, xs, ys, stepX, stepY, k0, k1, values + i * sampleStride);
        }
        const unsigned quad = (__ballot_sync(0xffffffffu, inside) >> (lane & 28)) & 0xfu;
        if (q == 0 && i < count) s_ok[i] = quad == 0xfu;
    }
    __syncthreads();

    // ---- mean and variance of each cut (the first warps) and the refinement of
    // its end (the others)
    float var = 0.f;
    const bool ok = t < count && s_ok[t];
    if (t < kMaxOuterPoints) {
        if (ok) {
            // MeanVar::add; the divisions by the counts are correctly rounded
            // (div_small: the operands here are zero or normal)
            const float* g = values + t * sampleStride;
            float mean = 0.f;
#pragma unroll 4
            for (int k = 0; k < cp.nSamples; ++k) {
                const float v = g[k], fc = float(k + 1), fc1 = float(k), rc = s_rcp[k + 1];
                mean = pm::div_small(fa(fm(mean, fc1), v), fc, rc);
                const float d = fs(v, mean);
                const float nv = fa(pm::div_small(fm(var, fc1), fc, rc), pm::div_small(fm(d, d), fc1, s_rcp[k]));
                if (k > 0) var = nv;
            }
        }
    } else {
        const int quadId = (t - kMaxOuterPoints) >> 2, q = t & 3;
        const unsigned quad = 0xfu << (lane & 28);
        float* const sig = values + min(max(cp.nOuter, in.presorted ? count : 0), kMaxOuterPoints) * sampleStride +
                           quadId * refineStride;
        const int n = cp.nRefine;
        for (int i = quadId; i < count; i += kRefineQuads) {
            if (!s_ok[i]) continue;
            const DirPoint op = pts[in.first + s_pick[i]];
            // pointOnEllipse with the host's cos / sin of the angle
            const float x = fs(op.x, in.cx), y = fs(op.y, in.cy);
            float tx = fa(fm(x, in.cosA), fm(y, in.sinA));
            float ty = fa(fm(-x, in.sinA), fm(y, in.cosA));
            const float cs = __fsqrt_rn(fa(fd(fm(tx, tx), fm(in.a, in.a)), fd(fm(ty, ty), fm(in.b, in.b))));
            tx = fd(tx, cs);
            ty = fd(ty, cs);
            const float sx = fa(fs(fm(tx, in.cosA), fm(ty, in.sinA)), in.cx);
            const float sy = fa(fa(fm(tx, in.sinA), fm(ty, in.cosA)), in.cy);
            // outerEdgeRefinement: the cut end moves to the strongest
            // derivative response along its gradient
            const float len = fm(fm(3.f, __fsqrt_rn(2.f)), in.scale);
            const float hw = fd(len, 2.f);
            const float gn = __fsqrt_rn(fa(fm(op.dx, op.dx), fm(op.dy, op.dy)));
            const float gx = fd(op.dx, gn), gy = fd(op.dy, gn);
            const float ax = fs(sx, fm(hw, gx)), ay = fs(sy, fm(hw, gy));
            const float bx = fa(sx, fm(hw, gx)), by = fa(sy, fm(hw, gy));
            const float den = fs(float(n), 1.f);
            const int seg = (n + 3) >> 2, k0 = min(q * seg, n), k1 = min(k0 + seg, n);
            const bool inside =
                sample_cut(img, W, H, ax, ay, fd(fs(bx, ax), den), fd(fs(by, ay), den), k0, k1, sig);
            const bool all = (__ballot_sync(quad, inside) & quad) == quad;
            __syncwarp(quad);
            if (all) {
                // convImageCut with clamped borders; std::map<float, float>
                // insert of the three kernels: the largest response wins, an
                // equal later one does not replace an earlier one
                float best = 0.f;
                int at = 0x7fffffff;
                for (int e = q; e < 3 * n; e += 4) {
                    const int kernel = e / n, loc = e - kernel * n;
                    float r = 0.f;
#pragma unroll
                    for (int j = 0; j < 9; ++j)
                        r = fa(r, fm(sig[min(max(loc - 4 + j, 0), n - 1)], s_edge[9 * kernel + j]));
                    if (at == 0x7fffffff || r > best) {
                        best = r;
                        at = e;
                    }
                }
#pragma unroll
                for (int o = 1; o < 4; o <<= 1) {
                    const float ob = __shfl_xor_sync(quad, best, o);
                    const int oat = __shfl_xor_sync(quad, at, o);
                    if (oat != 0x7fffffff && (at == 0x7fffffff || ob > best || (ob == best && oat < at))) {
                        best = ob;
                        at = oat;
                    }
                }
                const float step = fd(len, den), loc = float(at % n);
                if (q == 0) {
                    s_x[i] = fa(ax, fm(fm(step, loc), gx));
                    s_y[i] = fa(ay, fm(fm(step, loc), gy));
                    s_ref[i] = 1;
                }
            }
            __syncwarp(quad);  // the samples are read before the next cut's
        }
    }
    __syncthreads();

    // ---- selectCutCheapUniform over the collected (in-image) cuts, in order,
    // block-parallel.  The variances are finite and >= +0 (means and squares
    // of finite samples), so the largest one has a single bit pattern and any
    // reduction order gives the serial first-max.
    constexpr int kCutWarps = kMaxOuterPoints / 32;
    float vm = ok ? var : -1.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vm = fmaxf(vm, __shfl_xor_sync(0xffffffffu, vm, o));
    if (lane == 0 && warp < kCutWarps) s_wmax[warp] = vm;
    const int nOk = __syncthreads_count(ok);
    if (nOk == 0) {
        if (t == 0) {
            T.ncuts = 0;
            status[blockIdx.x] = CCTAGB_NO_COLLECTED_CUTS;
        }
        return;
    }
    float varMax = s_wmax[0];
#pragma unroll
    for (int w = 1; w < kCutWarps; ++w) varMax = fmaxf(varMax, s_wmax[w]);
    // the kept cuts, compacted in point order: rank = kept cuts before t
    const bool kp = ok && s_ref[t] && fd(var, varMax) > 0.5f;
    const unsigned kb = __ballot_sync(0xffffffffu, kp);
    if (lane == 0 && warp < kCutWarps) s_wcnt[warp] = __popc(kb);
    __syncthreads();
    int rank = __popc(kb & ((1u << lane) - 1u)), nKeep = 0;
#pragma unroll
    for (int w = 0; w < kCutWarps; ++w) {
        rank += w < warp ? s_wcnt[w] : 0;
        nKeep += s_wcnt[w];
    }
    if (kp) s_keep[rank] = t;
    __syncthreads();
    // The serial loop's k-th pick is keep[int(k * step)] while k < selectSize
    // and that index < nKeep; the index is non-decreasing in k, so the picks
    // are the prefix of k where both hold, one thread per k.
    const int selectSize = min(cp.maxSelect, nOk);
    const float step = fmaxf(1.f, fd(float(nKeep), float(selectSize)));
    const int j = int(fm(float(t), step));
    const bool pick = t < selectSize && j < nKeep;
    if (pick) {
        T.stop[t][0] = s_x[s_keep[j]];
        T.stop[t][1] = s_y[s_keep[j]];
    }
    const int nCuts = __syncthreads_count(pick);
    if (t == 0) {
        T.ncuts = nCuts;
        status[blockIdx.x] = nCuts == 0 ? CCTAGB_NO_SELECTED_CUTS : CCTAGB_ID_RELIABLE;
    }
}

void launch_cut_select(const uint8_t* d_img, int W, int H, const CutSelectIn* d_ins, const DirPoint* d_pts,
                       IdentTask* d_tasks, int* d_status, int n, const CutSelectParams& cp, cudaStream_t s)
{
    if (n <= 0) return;
    if (cp.nOuter < 0 || cp.nOuter > kMaxOuterPoints)
        throw Error{CCTAGB_BAD_ARG, "nSamplesOuterEllipse above " + std::to_string(kMaxOuterPoints)};
    if (cp.nSamples < 2 || cp.nSamples > kMaxSamples) throw Error{CCTAGB_BAD_ARG, "sampleCutLength out of range"};
    if (cp.nRefine < 2 || cp.nRefine > kMaxRefineSamples)
        throw Error{CCTAGB_BAD_ARG, "numSamplesOuterEdgePointsRefinement out of range"};
    // sort keys, or the samples of up to nOuter cuts and of the refining quads
    const size_t samples = sizeof(float) * (size_t(std::max(cp.nOuter, 1)) * (cp.nSamples | 1) +
                                            size_t(kRefineQuads) * (cp.nRefine | 1));
    const size_t smem = std::max(samples, sizeof(unsigned long long) * kCutSortCap);
    CCTAGB_CUDA(cudaFuncSetAttribute(k_cut_select, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    k_cut_select<<<n, kThreads, smem, s>>>(d_img, W, H, d_ins, d_pts, d_tasks, d_status, cp);
    CCTAGB_CUDA(cudaGetLastError());
}

}  // namespace cctagb
