// Identification on sm_100a: imaged-center refinement and ID reading, a thread
// block or a cluster of them per marker (Identification.cpp:813-1158
// refineConicFamilyGlob / imageCenterOptimizationGlob / costFunctionGlob /
// getSignals, and :50-193 orazioDistanceRobust, :1408-1436 ID vote).
//
// Grid refinement: each round evaluates a gridN x gridN set of trial centres
// (getNearbyPoints, conditioned by the ellipse).  A trial's homography maps the
// unit circle to the outer ellipse and the origin to the trial centre
// (computeHomographyFromEllipseAndImagedCenter); every cut is resampled in the
// marker plane along the ray to its back-projected end.
//
// The reference marks a cut "out of bounds" the first time any of its samples
// leaves the image, for every later trial and round (the flag lives in the cut
// object).  This kernel reproduces that order: the flags of all trials of a
// round are computed first (a cut's samples lie on the image of a segment, so
// its two end samples decide), then a prefix OR in trial order gives each
// trial the set of cuts the reference would still use.
//
// Cost: the reference's mean over cut pairs of sum_k (s_i[k] - s_j[k])^2, here
// in the equivalent form n * sum_i (s_i[k] - mean_k)^2 summed over k, divided
// by the n(n-1)/2 pairs (shifted FP32 sums per sample, FP64 over samples).
//
// The kernel is bound by instruction issue and by the reads of the samples: a
// 22-cut, 100-sample, 25-trial round is 55,000 bilinear samples, whose lanes lie
// along a ray and so on many lines of the L1 (read from the image, four bytes
// each, they kept it 90 % busy).  So the marker's pixels are staged in shared
// memory, with rows an odd number of words apart; the sample loop is kept to
// some 45 instructions a sample (no IEEE division, the clamp and the integer
// part of a coordinate in one operation, constant factors left to the end); no
// lane idles on the samples past a multiple of 32 (they are packed several
// trials to a warp); and the serial parts (statistics of a signal, medians, the
// distances to the bank) are spread over lanes, warps and blocks.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>

#include <cooperative_groups.h>

#include "common.hpp"
#include "ident_host.hpp"
#include "ident_layout.hpp"
#include "cctag_b200/portable/pmath.hpp"

namespace cctagb {

namespace {

constexpr int kMaxTrials = 25;
static_assert(kIdentTrialWarps == kMaxTrials, "a warp per trial");
constexpr int kThreads = 32 * kMaxTrials;  // of the cost kernels
constexpr int kWarps = kThreads / 32;
// The samples along a cut come in chunks of 32 (one per lane).  Per-chunk sums
// are formed the same way in every block layout and added in chunk order, so
// all layouts give the same bits.
constexpr int kChunk = 32;
constexpr int kMaxChunks = kMaxSamples / kChunk;
static_assert(kGnWarps == kMaxChunks, "a warp per chunk");

__device__ __forceinline__ void mat_mul(const float* a, const float* b, float* r)
{
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) r[i * 3 + j] = a[i * 3] * b[j] + a[i * 3 + 1] * b[3 + j] + a[i * 3 + 2] * b[6 + j];
}

__device__ __forceinline__ bool mat_inv(const float* a, float* r)
{
    const float c00 = a[4] * a[8] - a[5] * a[7];
    const float c01 = a[5] * a[6] - a[3] * a[8];
    const float c02 = a[3] * a[7] - a[4] * a[6];
    const float det = a[0] * c00 + a[1] * c01 + a[2] * c02;
    if (det == 0.f || !isfinite(det)) return false;
    const float id = 1.f / det;
    r[0] = c00 * id;
    r[1] = (a[2] * a[7] - a[1] * a[8]) * id;
    r[2] = (a[1] * a[5] - a[2] * a[4]) * id;
    r[3] = c01 * id;
    r[4] = (a[0] * a[8] - a[2] * a[6]) * id;
    r[5] = (a[2] * a[3] - a[0] * a[5]) * id;
    r[6] = c02 * id;
    r[7] = (a[1] * a[6] - a[0] * a[7]) * id;
    r[8] = (a[0] * a[4] - a[1] * a[3]) * id;
    return true;
}

__device__ __forceinline__ void apply_h(const float* H, float x, float y, float& ox, float& oy, float& w)
{
    const float u = H[0] * x + H[1] * y + H[2];
    const float v = H[3] * x + H[4] * y + H[5];
    w = H[6] * x + H[7] * y + H[8];
    ox = u / w;
    oy = v / w;
}

// The image a candidate is read from: a device image with its row pitch and
// the candidate's rectangle [x0, x1) x [y0, y1) (the whole frame in a
// detection; one crop of an atlas in the batched form).
struct Roi {
    const uint8_t* img;
    size_t pitch;
    int x0, y0, x1, y1;
};

__device__ __forceinline__ Roi make_roi(const uint8_t* img, size_t pitch, const IdentTask& T)
{
    if (T.local)  // coordinates relative to the rectangle's corner
        return Roi{img + size_t(T.roi[1]) * pitch + size_t(T.roi[0]), pitch, 0, 0, T.roi[2], T.roi[3]};
    return Roi{img, pitch, T.roi[0], T.roi[1], T.roi[0] + T.roi[2], T.roi[1] + T.roi[3]};
}

// Identification.hpp:197-219
__device__ __forceinline__ float bilinear(const Roi& R, float x, float y)
{
    const int px = int(x), py = int(y);
    const uint8_t* p0 = R.img + px + size_t(py) * R.pitch;
    const float fx = x - float(px), fy = y - float(py);
    const float fx1 = 1.0f - fx, fy1 = 1.0f - fy;
    const float p1 = __ldg(p0), p2 = __ldg(p0 + 1), p3 = __ldg(p0 + R.pitch), p4 = __ldg(p0 + R.pitch + 1);
    return (p1 * (fx1 * fy1) + p2 * (fx * fy1) + p3 * (fx1 * fy) + p4 * (fx * fy)) / 2;
}

// The reference's test "x >= 0 && x < cols - 1 && y >= 0 && y < rows - 1",
// on the candidate's rectangle.
__device__ __forceinline__ bool inside(const Roi& R, float x, float y)
{
    return x >= float(R.x0) && x < float(R.x1 - 1) && y >= float(R.y0) && y < float(R.y1 - 1);
}

// Ellipse.cpp:103-159 semi axes of a conic (for the conditioned ellipse).
__device__ void conic_axes(const float* Q, float& a, float& b)
{
    const float p0 = Q[0], p1 = 2.f * Q[1], p2 = Q[4], p3 = 2.f * Q[2], p4 = 2.f * Q[5], p5 = Q[8];
    const float th = 0.5f * atan2f(p1, p0 - p2);
    float st, ct;
    sincosf(th, &st, &ct);
    const float s2 = st * st, c2 = ct * ct, cs = st * ct;
    const float Au = p3 * ct + p4 * st, Av = -p3 * st + p4 * ct;
    const float Auu = p0 * c2 + p2 * s2 + p1 * cs, Avv = p0 * s2 + p2 * c2 - p1 * cs;
    if (Auu == 0.f || Avv == 0.f) {
        a = b = 0.f;
        return;
    }
    const float tu = -Au / (2.f * Auu), tv = -Av / (2.f * Avv);
    const float wc = p5 - Auu * tu * tu - Avv * tv * tv;
    a = sqrtf(fabsf(-wc / Auu));
    b = sqrtf(fabsf(-wc / Avv));
}

// Ellipse.cpp:161-214 canonic form: C (canonical conic), Tp (primal), Td (dual).
__device__ void canonic_form(const float* Q, float* C, float* Tp, float* Td)
{
    const float q1 = Q[0], q2 = Q[1], q3 = Q[2], q4 = Q[4], q5 = Q[5], q6 = Q[8];
    const float par1 = q1, par2 = 2 * q2, par3 = q4, par4 = 2 * q3, par5 = 2 * q5;
    const float th = 0.5f * atan2f(par2, par1 - par3);
    const float ct = cosf(th), st = sinf(th);
    const float s2 = st * st, c2 = ct * ct, cs = st * ct;
    const float Au = par4 * ct + par5 * st, Av = -par4 * st + par5 * ct;
    const float Auu = par1 * c2 + par3 * s2 + par2 * cs, Avv = par1 * s2 + par3 * c2 - par2 * cs;
    const float tu = -Au / (2 * Auu), tv = -Av / (2 * Avv);
    const float uc = tu * ct - tv * st, vc = tu * st + tv * ct;
    const float t1 = ct * (ct * q1 + q2 * st) + st * (ct * q2 + q4 * st);
    const float t2 = ct * (ct * q2 + q4 * st) - st * (ct * q1 + q2 * st);
    const float t3 = ct * q3 + q5 * st + uc * (ct * q1 + q2 * st) + vc * (ct * q2 + q4 * st);
    const float t4 = ct * (ct * q4 - q2 * st) - st * (ct * q2 - q1 * st);
    const float t5 = ct * q5 - q3 * st + uc * (ct * q2 - q1 * st) + vc * (ct * q4 - q2 * st);
    const float t6 = q6 + uc * (q3 + q1 * uc + q2 * vc) + vc * (q5 + q2 * uc + q4 * vc) + q3 * uc + q5 * vc;
    C[0] = t1; C[1] = t2; C[2] = t3; C[3] = t2; C[4] = t4; C[5] = t5; C[6] = t3; C[7] = t5; C[8] = t6;
    Tp[0] = ct;  Tp[1] = st; Tp[2] = -ct * uc - st * vc;
    Tp[3] = -st; Tp[4] = ct; Tp[5] = st * uc - ct * vc;
    Tp[6] = 0;   Tp[7] = 0;  Tp[8] = ct * ct + st * st;
    Td[0] = ct; Td[1] = -st; Td[2] = uc;
    Td[3] = st; Td[4] = ct;  Td[5] = vc;
    Td[6] = 0;  Td[7] = 0;   Td[8] = 1.f;
}

// Identification.cpp:739-798: homography (plane -> image) sending the unit
// circle to the ellipse and the origin to (x, y).
__device__ void homography_from_center(const float* C, const float* Tp, const float* Td, float x, float y, float* H)
{
    float xc, yc, w;
    apply_h(Tp, x, y, xc, yc, w);
    const float Q11 = C[0], Q22 = C[4], Q33 = C[8];
    float h[9];
    h[0] = Q33;      h[1] = Q22 * xc * yc;           h[2] = -Q33 * xc;
    h[3] = 0.f;      h[4] = -Q11 * xc * xc - Q33;    h[5] = -Q33 * yc;
    h[6] = -Q11 * xc; h[7] = Q22 * yc;               h[8] = -Q33;
    const float d0 = sqrtf((Q22 * Q33 / Q11 * (Q11 * xc * xc + Q22 * yc * yc + Q33)));
    const float d1 = Q33;
    const float d2 = sqrtf(-Q22 * (Q11 * xc * xc + Q33));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        h[i * 3 + 0] *= d0;
        h[i * 3 + 1] *= d1;
        h[i * 3 + 2] *= d2;
    }
    mat_mul(Td, h, H);
}

// The image of a cut's samples under a trial homography: sample k is at
// (U0 + k dU, V0 + k dV) / (W0 + k dW).  One entry of padding per trial keeps
// lanes that read different trials on different banks.
struct TrialLines {
    float4* uv;  // U0 dU V0 dV, entry t * stride + cut
    float2* w;   // W0 dW
    int stride;
};
__device__ __forceinline__ TrialLines trial_lines(void* work, int trials, int ncuts)
{
    float4* uv = static_cast<float4*>(work);
    return TrialLines{uv, reinterpret_cast<float2*>(uv + trials * (ncuts + 1)), ncuts + 1};
}
struct GnChunk {  // Gauss-Newton, one chunk of samples
    float s[kMaxCuts][kChunk];            // value
    float dx[kMaxCuts][kChunk];           // d value / d center x
    float dy[kMaxCuts][kChunk];           // d value / d center y
};
// Cuts x samples whose values and derivatives Gauss-Newton has room for at least;
// a block with an SM to itself has it for all of its marker's.
constexpr int kGnWhole = 2400;
constexpr int kSigStride = kMaxSamples + 1;
// What the reading of the cuts keeps once the center is found.
struct FinalWork {
    float sig[kMaxCuts][kSigStride];                // final signals
    uint32_t black[kMaxBankIds][kMaxSamples / 32];  // per bank row: samples inside an odd number of its rings
    float barcode[kMaxSamples];
};
// Dynamic shared memory: the lines of the grid rounds (an entry of padding past
// the cuts) or Gauss-Newton's samples, then the marker's pixels; at the end
// FinalWork in their place.
__host__ __device__ constexpr size_t align16(size_t v) { return (v + 15) & ~size_t(15); }
__host__ __device__ constexpr size_t grid_work(int trials, int ncuts)
{
    return align16(size_t(trials) * (ncuts + 1) * (sizeof(float4) + sizeof(float2)));
}
constexpr size_t kGnWork = 3 * sizeof(float) * kGnWhole;
static_assert(sizeof(GnChunk) <= kGnWork, "the chunk form fits");

struct Shared {
    float C[9], Tp[9], Td[9];
    float mT[9], mTi[9];
    float nsScale;                 // max semi axis of the conditioned ellipse
    float cx, cy;                  // current center
    float Hopt[9];
    float minRes;
    uint32_t oob;                  // sticky out-of-bounds cut mask
    int rounds;
    int fail;
    float trialH[kMaxTrials][9], trialHi[kMaxTrials][9];
    int trialOk[kMaxTrials];       // the homography has an inverse
    float trialPt[kMaxTrials][2];
    // Gauss-Newton state
    float gH[9], gHi[9], gdH[2][9], gdHi[2][9];  // homography at the trial center, inverse, center derivatives
    float gTry[2];                               // trial center
    uint32_t gOob;                               // cuts whose end samples leave the rectangle at the trial
    float gBack[kMaxCuts][6];                    // back-projected cut ends and their center derivatives
    double gPart[2][kMaxChunks][6];              // per-chunk sums (cost, J^T r, J^T J) by parity
    double gSum[6];
    double gA[3], gG[2], gBest, gLambda;         // normal equations at the best center, its cost, damping
    int gHave, gStop, iterations;
    uint32_t trialOob[kMaxTrials];
    int box[4];                              // the staged pixels' rectangle x0 y0 x1 y1 (empty: none), as roi
    int direct;                              // a sample of the round lies outside them
    double part[2][kMaxChunks][kMaxTrials];  // per-chunk shares of each trial's cost (by round parity)
    float radius[kMaxSamples];               // the samples' plane radii
    float rcp[kMaxSamples + 1];              // 1 / i, rounded
    float stats[kMaxCuts][4];                // of a cut's signal: black and white mean, 1 / (2 variance) (a double)
    int winner[kMaxCuts];
    float vwin[kMaxCuts];
};

// 1 / w without the fix-up for denormals and the largest floats, which a
// homography's scale does not reach.
__device__ __forceinline__ float fast_rcp(float w)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(w));
    return r;
}

// Whether a sample's pixels are staged: a pixel's distance from the edges of
// the staged rectangle, for the rounding of samples between two such ends (at
// an edge that is the candidate's rectangle's own, as that is read).
__device__ __forceinline__ bool in_box(const Shared& S, const Roi& R, float x, float y)
{
    return x >= float(S.box[0] + (S.box[0] > R.x0 ? 1 : 0)) && x < float(S.box[2] - (S.box[2] < R.x1 ? 2 : 1)) &&
           y >= float(S.box[1] + (S.box[1] > R.y0 ? 1 : 0)) && y < float(S.box[3] - (S.box[3] < R.y1 ? 2 : 1));
}

// Bytes per row of the staged pixels: an odd number of words, so that a column
// of them spreads over all banks.
__device__ __forceinline__ int box_pitch(const Shared& S) { return (((S.box[2] - S.box[0] + 3) >> 2) | 1) << 2; }

// The rectangle that holds the marker's samples with their neighbours (the
// segments from the cut ends to near the center), clipped to the candidate's
// rectangle; empty when it takes more than `room` bytes.  By a warp.
__device__ void find_box(Shared& S, const IdentTask& T, const Roi& R, size_t room, int lane)
{
    float x = T.x0, y = T.y0;
    if (lane < T.ncuts) {
        x = T.stop[lane][0];
        y = T.stop[lane][1];
    }
    float x0 = fminf(x, T.x0), x1 = fmaxf(x, T.x0), y0 = fminf(y, T.y0), y1 = fmaxf(y, T.y0);
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
        y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
        x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
        y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    }
    if (lane == 0) {
        // finite (checked by the host, or refined image points); clipped as
        // floats first, so that the conversions are in range
        S.box[0] = int(fminf(fmaxf(x0 - 2.f, float(R.x0)), float(R.x1)));
        S.box[1] = int(fminf(fmaxf(y0 - 2.f, float(R.y0)), float(R.y1)));
        S.box[2] = int(fminf(fmaxf(x1 + 4.f, float(R.x0)), float(R.x1)));
        S.box[3] = int(fminf(fmaxf(y1 + 4.f, float(R.y0)), float(R.y1)));
        // a row start on a word boundary, where the image's rows are
        const int down = int(reinterpret_cast<size_t>(R.img + S.box[0]) & 3);
        if (R.pitch % 4 == 0 && S.box[0] - down >= R.x0) S.box[0] -= down;
        const int w = S.box[2] - S.box[0], h = S.box[3] - S.box[1];
        if (w < 4 || h < 4 || size_t(box_pitch(S)) * size_t(h) > room)
            S.box[0] = S.box[1] = S.box[2] = S.box[3] = 0;
    }
}

// The pixels of the box into shared memory, a word of four at a time: a word
// on a boundary by an asynchronous copy, another one put together from the two
// it straddles (inside the row only), the ends of a row byte by byte.  The
// caller's next barrier must follow cp.async.wait_all of every thread.
__device__ void stage_box(const Shared& S, const Roi& R, uint8_t* px)
{
    const int w = S.box[2] - S.box[0], h = S.box[3] - S.box[1];
    if (w <= 0) return;
    const int pitch = box_pitch(S), words = (w + 3) >> 2;
    const int nwarps = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (int y = threadIdx.x >> 5; y < h; y += nwarps) {
        const uint8_t* row = R.img + size_t(S.box[1] + y) * R.pitch + size_t(S.box[0]);
        const int shift = int(reinterpret_cast<size_t>(row) & 3);
        uint32_t* out = reinterpret_cast<uint32_t*>(px + size_t(y) * pitch);
#pragma unroll 4
        for (int j = lane; j < words; j += 32) {
            const uint8_t* p = row + 4 * j;
            if (shift == 0 && 4 * j + 4 <= w) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                 unsigned(__cvta_generic_to_shared(out + j))),
                             "l"(p)
                             : "memory");
                continue;
            }
            uint32_t v;
            if (shift != 0 && j > 0 && 4 * j + 8 <= w) {
                const uint32_t* q = reinterpret_cast<const uint32_t*>(p - shift);
                v = __funnelshift_r(__ldg(q), __ldg(q + 1), 8 * shift);
            } else {
                v = 0u;
                for (int k = 0; k < 4 && 4 * j + k < w; ++k) v |= uint32_t(__ldg(p + k)) << (8 * k);
            }
            out[j] = v;
        }
    }
}

// The image line of cut c under trial t's homography, and whether its end
// samples leave the rectangle.
__device__ __forceinline__ void setup_cut(Shared& S, const TrialLines& lines, const IdentTask& T, int t, int c,
                                          const IdentParams& ip, const Roi& R)
{
    const float* Hm = S.trialH[t];
    float bx, by, w;
    if (S.trialOk[t]) apply_h(S.trialHi[t], T.stop[c][0], T.stop[c][1], bx, by, w);
    else bx = by = NAN;
    const float xs = bx * ip.beginSig, ys = by * ip.beginSig;
    const float sx = (bx - xs) / (float(ip.nSamples) - 1.f), sy = (by - ys) / (float(ip.nSamples) - 1.f);
    // sample k is (xs + k sx, ys + k sy) in the marker plane; its image in
    // homogeneous coordinates is linear in k: H (xs, ys, 1) + k H (sx, sy, 0)
    float cp[6];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        cp[2 * i] = __fmaf_rn(Hm[3 * i], xs, __fmaf_rn(Hm[3 * i + 1], ys, Hm[3 * i + 2]));
        cp[2 * i + 1] = __fmaf_rn(Hm[3 * i], sx, __fmul_rn(Hm[3 * i + 1], sy));
    }
    lines.uv[t * lines.stride + c] = make_float4(cp[0], cp[1], cp[2], cp[3]);
    lines.w[t * lines.stride + c] = make_float2(cp[4], cp[5]);
    // end samples, with the sample loop's own arithmetic
    const float kl = float(ip.nSamples - 1);
    const float w0 = cp[4], w1 = __fmaf_rn(kl, cp[5], cp[4]);
    const float r0 = fast_rcp(w0), r1 = fast_rcp(w1);
    const float x0 = __fmul_rn(cp[0], r0), y0 = __fmul_rn(cp[2], r0);
    const float x1 = __fmul_rn(__fmaf_rn(kl, cp[1], cp[0]), r1), y1 = __fmul_rn(__fmaf_rn(kl, cp[3], cp[2]), r1);
    bool bad = !(w0 > 0.f && w1 > 0.f) && !(w0 < 0.f && w1 < 0.f);
    bad = bad || !inside(R, x0, y0) || !inside(R, x1, y1);
    if (bad) atomicOr(&S.trialOob[t], 1u << c);
    else if (!(in_box(S, R, x0, y0) && in_box(S, R, x1, y1))) S.direct = 1;
}

// Byte -> float without a conversion instruction (exponent 2^23 trick).
__device__ __forceinline__ float byte_to_float(uint32_t b) { return __uint_as_float(0x4B000000u | b) - 8388608.f; }

// floor(x) for 0 <= x < 2^22 without a conversion instruction: adding 2^23
// with round-toward-zero leaves floor(x) in the mantissa.  Returns the
// integer and stores its float value in fl.
__device__ __forceinline__ int floor_small(float x, float& fl)
{
    const float t = __fadd_rz(x, 8388608.f);
    fl = t - 8388608.f;
    return __float_as_int(t) - 0x4B000000;
}

// Identification.hpp:197-219 for a sample inside the rectangle (explicit
// roundings, so that every caller gets the same bits).
__device__ __forceinline__ float bilinear_value(const float p[4], float fx, float fy)
{
    const float fx1 = __fsub_rn(1.0f, fx), fy1 = __fsub_rn(1.0f, fy);
    float a = __fmul_rn(p[0], __fmul_rn(fx1, fy1));
    a = __fmaf_rn(p[1], __fmul_rn(fx, fy1), a);
    a = __fmaf_rn(p[2], __fmul_rn(fx1, fy), a);
    a = __fmaf_rn(p[3], __fmul_rn(fx, fy), a);
    return __fmul_rn(a, 0.5f);
}

// Same value and its gradient in x and y (the derivative of the bilinear
// patch the sample falls in).
__device__ __forceinline__ float bilinear_value_grad(const float p[4], float fx, float fy, float& gx, float& gy)
{
    const float fx1 = 1.0f - fx, fy1 = 1.0f - fy;
    gx = ((p[1] - p[0]) * fy1 + (p[3] - p[2]) * fy) * 0.5f;
    gy = ((p[2] - p[0]) * fx1 + (p[3] - p[1]) * fx) * 0.5f;
    return bilinear_value(p, fx, fy);
}
// Row i of H applied to (x, y, 1), explicit roundings.
__device__ __forceinline__ float hrow(const float* Hm, int i, float x, float y)
{
    return __fmaf_rn(Hm[3 * i], x, __fmaf_rn(Hm[3 * i + 1], y, Hm[3 * i + 2]));
}

// The pixels as the sample loop reads them, from the image or staged: the
// first pixel, and what turns the integer part of a coordinate (in the mantissa
// of x + 2^23) into a pixel's index, clamped so that rounding at the border
// never reads outside.
template <bool STAGED>
struct SampleArea {
    const uint8_t* corner;
    size_t pitch;
    int biasX, biasY, maxX, maxY;
};
__device__ __forceinline__ SampleArea<false> image_area(const Roi& R)
{
    return {R.img + size_t(R.y0) * R.pitch + size_t(R.x0), R.pitch, -0x4B000000 - R.x0, -0x4B000000 - R.y0,
            R.x1 - R.x0 - 2, R.y1 - R.y0 - 2};
}
__device__ __forceinline__ SampleArea<true> staged_area(const Shared& S, const uint8_t* px)
{
    return {px, size_t(box_pitch(S)), -0x4B000000 - S.box[0], -0x4B000000 - S.box[1], S.box[2] - S.box[0] - 2,
            S.box[3] - S.box[1] - 2};
}

// The four pixels around (x, y), zero-extended, and the fractional offsets.
template <bool STAGED>
__device__ __forceinline__ void area_taps(const SampleArea<STAGED>& A, float x, float y, uint32_t p[4], float& fx,
                                          float& fy)
{
    const float tx = __fadd_rz(fmaxf(x, 0.f), 8388608.f), ty = __fadd_rz(fmaxf(y, 0.f), 8388608.f);
    fx = __fsub_rn(x, __fsub_rn(tx, 8388608.f));
    fy = __fsub_rn(y, __fsub_rn(ty, 8388608.f));
    const int px = __viaddmin_s32_relu(__float_as_int(tx), A.biasX, A.maxX);
    const int py = __viaddmin_s32_relu(__float_as_int(ty), A.biasY, A.maxY);
    if (STAGED) {
        const int pitch = int(A.pitch), at = py * pitch + px;
        p[0] = A.corner[at];
        p[1] = A.corner[at + 1];
        p[2] = A.corner[at + pitch];
        p[3] = A.corner[at + pitch + 1];
    } else {
        const uint8_t* p0 = A.corner + size_t(unsigned(py)) * A.pitch + unsigned(px);
        const uint8_t* p1 = p0 + A.pitch;
        p[0] = __ldg(p0);
        p[1] = __ldg(p0 + 1);
        p[2] = __ldg(p1);
        p[3] = __ldg(p1 + 1);
    }
}

// 2^-22 times the bilinear value (Identification.hpp:197-219) of a sample of a
// cut: its point on the cut's image line, then the read.  The operations and
// their roundings are those of bilinear_value on scaled pixels: a byte taken as
// the bits of a float is its value times 2^-149, and one product brings it to
// 2^-23 of the pixel, exactly; the factor and the value's 1/2 are powers of two
// that trial sums carry to their end (kTermScale).
template <bool STAGED>
__device__ __forceinline__ float cut_sample(const SampleArea<STAGED>& A, const float4& l, const float2& lw, float kf)
{
    const float r = fast_rcp(__fmaf_rn(kf, lw.y, lw.x));
    const float x = __fmul_rn(__fmaf_rn(kf, l.y, l.x), r), y = __fmul_rn(__fmaf_rn(kf, l.w, l.z), r);
    uint32_t p[4];
    float fx, fy;
    area_taps(A, x, y, p, fx, fy);
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __fmul_rn(__uint_as_float(p[q]), 0x1p126f);
    const float fx1 = __fsub_rn(1.0f, fx), fy1 = __fsub_rn(1.0f, fy);
    float a = __fmul_rn(v[0], __fmul_rn(fx1, fy1));
    a = __fmaf_rn(v[1], __fmul_rn(fx, fy1), a);
    a = __fmaf_rn(v[2], __fmul_rn(fx1, fy), a);
    return __fmaf_rn(v[3], __fmul_rn(fx, fy), a);
}
constexpr double kTermScale = 0x1p44;  // (2^22)^2

// Sum over the 32 lanes (the same butterfly, so the same bits, everywhere).
__device__ __forceinline__ double lane_sum(double v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Share of a trial's cost of one whole chunk (a warp, lane = sample within the
// chunk): over the valid cuts in order, a few at a time so that their reads
// overlap.  Per sample the cut values are shifted by the first valid cut's
// value before the FP32 sums (the term n * sum(d^2) - (sum d)^2 does not change
// under a common shift, and the shifted sums stay small), then summed over the
// lanes in FP64.
template <bool STAGED>
__device__ __forceinline__ double trial_chunk(const TrialLines& lines, const SampleArea<STAGED>& A, int t,
                                              uint32_t valid, int k)
{
    constexpr int G = 4;  // cuts per step
    const int n = __popc(valid);
    float v0 = 0.f, s1 = 0.f, s2 = 0.f;
    const float kf = float(k);
    if (n >= 2) {
        bool first = true;  // the same in every lane, as valid: uniform branches
        for (uint32_t m = valid; m;) {
            const int have = __popc(m);
            float val[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int i = t * lines.stride + (m ? __ffs(m) - 1 : 0);  // past the last valid cut: read, not used
                m &= m - 1;
                val[g] = cut_sample(A, lines.uv[i], lines.w[i], kf);
            }
            if (first) v0 = val[0];  // first valid cut: the shift
            first = false;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (g >= have) break;
                const float d = __fsub_rn(val[g], v0);
                s1 = __fadd_rn(s1, d);
                s2 = __fmaf_rn(d, d, s2);
            }
        }
    }
    return lane_sum(n >= 2 ? kTermScale * double(__fsub_rn(__fmul_rn(float(n), s2), __fmul_rn(s1, s1))) : 0.0);
}

// The last, partial chunk (tail < 32 samples) of several trials at once: groups
// of `width` lanes (a power of two >= tail), each its own trial t with its own
// valid cuts; every lane of the warp calls it.  The same sums as
// trial_chunk's with the lanes past the tail contributing zero.
template <bool STAGED>
__device__ __forceinline__ double trial_tail(const TrialLines& lines, const SampleArea<STAGED>& A, int t,
                                             uint32_t valid, int k, bool live, int width)
{
    constexpr int G = 4;
    const int n = __popc(valid);
    float v0 = 0.f, s1 = 0.f, s2 = 0.f;
    const float kf = float(k);
    bool first = true;
    for (uint32_t m = n >= 2 ? valid : 0u; __any_sync(0xffffffffu, m != 0u);) {
        float val[G];
        bool use[G];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            use[g] = m != 0u;
            const int c = m ? __ffs(m) - 1 : 0;
            m &= m - 1;
            const int i = t * lines.stride + c;
            val[g] = use[g] ? cut_sample(A, lines.uv[i], lines.w[i], kf) : 0.f;
        }
        if (first) v0 = val[0];
        first = false;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float d = use[g] ? __fsub_rn(val[g], v0) : 0.f;
            s1 = __fadd_rn(s1, d);
            s2 = __fmaf_rn(d, d, s2);
        }
    }
    double v = (n >= 2 && live) ? kTermScale * double(__fsub_rn(__fmul_rn(float(n), s2), __fmul_rn(s1, s1))) : 0.0;
    for (int o = width >> 1; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The same shares of all chunks of a trial, for pixels read from the image: the
// reads of a cut's chunks overlap, two cuts at a time.  Lanes past the last sample
// read it again (in bounds, no branch) and contribute zero.
__device__ __forceinline__ void trial_chunks(const TrialLines& lines, const SampleArea<false>& A, int t,
                                             uint32_t valid, int samples, int lane, double out[kMaxChunks])
{
    constexpr int G = 2;  // cuts per step
    const int n = __popc(valid);
    float v0[kMaxChunks], s1[kMaxChunks], s2[kMaxChunks], kf[kMaxChunks];
#pragma unroll
    for (int q = 0; q < kMaxChunks; ++q) {
        kf[q] = float(min(q * kChunk + lane, samples - 1));
        v0[q] = s1[q] = s2[q] = 0.f;
    }
    if (n >= 2) {
        bool first = true;
        for (uint32_t m = valid; m;) {
            const int have = __popc(m);
            float val[G][kMaxChunks];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const int i = t * lines.stride + (m ? __ffs(m) - 1 : 0);  // past the last valid cut: read, not used
                m &= m - 1;
                const float4 l = lines.uv[i];
                const float2 lw = lines.w[i];
#pragma unroll
                for (int q = 0; q < kMaxChunks; ++q) val[g][q] = cut_sample(A, l, lw, kf[q]);
            }
#pragma unroll
            for (int q = 0; q < kMaxChunks; ++q)
                if (first) v0[q] = val[0][q];  // first valid cut: the shift
            first = false;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                if (g >= have) break;
#pragma unroll
                for (int q = 0; q < kMaxChunks; ++q) {
                    const float d = __fsub_rn(val[g][q], v0[q]);
                    s1[q] = __fadd_rn(s1[q], d);
                    s2[q] = __fmaf_rn(d, d, s2[q]);
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kMaxChunks; ++q)
        out[q] = lane_sum(n >= 2 && q * kChunk + lane < samples
                              ? kTermScale * double(__fsub_rn(__fmul_rn(float(n), s2[q]), __fmul_rn(s1[q], s1[q])))
                              : 0.0);
}

// The sampling tasks of a round, spread over the warps of the cluster: one per
// trial and whole chunk, chunk by chunk (a block keeps to a band of the
// marker), then the packed partial chunks; `valid` is trial `lane`'s cuts.
struct Tasks {
    int nTrials, whole, tail, width, packed;  // whole chunks, samples of the last one, its lanes, its trials per warp
    __device__ int nWhole() const { return nTrials * whole; }
    __device__ int count() const { return nWhole() + (tail ? (nTrials + packed - 1) / packed : 0); }
};
template <bool STAGED>
__device__ __forceinline__ void sample_round(Shared& S, const TrialLines& lines, const SampleArea<STAGED>& A,
                                             const Tasks& K, uint32_t valid, int par, int first, int step, int csize,
                                             int lane)
{
    // every block of the cluster gets every share: lane q stores to block q
    namespace cg = cooperative_groups;
    auto put = [&](int j, int t, double c, int from, int by) {
        if (csize == 1) {
            if (from == 0) S.part[par][j][t] = c;
        } else {
            for (int q = from; q < csize; q += by) *cg::this_cluster().map_shared_rank(&S.part[par][j][t], q) = c;
        }
    };
    for (int task = first; task < K.count(); task += step) {
        if (task < K.nWhole()) {
            const int j = task / K.nTrials, t = task - j * K.nTrials;
            const double c = trial_chunk(lines, A, t, __shfl_sync(0xffffffffu, valid, t), j * kChunk + lane);
            put(j, t, c, lane, 32);
        } else {
            const int own = (task - K.nWhole()) * K.packed + lane / K.width, t = min(own, K.nTrials - 1);
            const int k = lane % K.width;
            const bool live = k < K.tail && own < K.nTrials;  // each lane of the group ends with its sum
            const double c = trial_tail(lines, A, t, __shfl_sync(0xffffffffu, valid, t),
                                        K.whole * kChunk + min(k, K.tail - 1), live, K.width);
            if (own < K.nTrials) put(K.whole, t, c, k, K.width);
        }
    }
}

// Ascending sort of a thread's 32 values: Batcher's odd-even merge network
// (K. E. Batcher, "Sorting networks and their applications", AFIPS 1968), its
// steps as templates so that every index is a constant (registers only).
template <int P, int K>
__device__ __forceinline__ void sort_network(float (&v)[kMaxCuts])
{
    static_assert(kMaxCuts == 32, "a power of two");
#pragma unroll
    for (int j = K % P; j + K < kMaxCuts; j += 2 * K)
#pragma unroll
        for (int i = j; i < j + K; ++i)
            if (i + K < kMaxCuts && i / (2 * P) == (i + K) / (2 * P)) {
                const float a = v[i], b = v[i + K];
                v[i] = fminf(a, b);
                v[i + K] = fmaxf(a, b);
            }
    if constexpr (K > 1) sort_network<P, K / 2>(v);
    else if constexpr (2 * P < kMaxCuts) sort_network<2 * P, 2 * P>(v);
}

// Identification.hpp:373-384, with val = +1 (white: even ratio count) or -1
// and the division by 2 var done as a product with rvar2 = 1 / double(2 var).
__device__ __forceinline__ float dis_r(float sig, bool white, float mub, float muw, double rvar2)
{
    const float d = white ? fminf(__fsub_rn(sig, muw), 0.f) : fmaxf(__fsub_rn(sig, mub), 0.f);
    return float(double(__fmul_rn(d, d)) * rvar2);
}


// ------------------------------------------------------- center derivatives --
// A value with its derivatives along the two imaged-center coordinates
// (forward mode), for the homography of a trial center.
struct D2 {
    float v, a, b;
};
__device__ __forceinline__ D2 d2c(float v) { return D2{v, 0.f, 0.f}; }
__device__ __forceinline__ D2 operator+(D2 p, D2 q) { return D2{p.v + q.v, p.a + q.a, p.b + q.b}; }
__device__ __forceinline__ D2 operator*(D2 p, float s) { return D2{p.v * s, p.a * s, p.b * s}; }
__device__ __forceinline__ D2 operator+(D2 p, float s) { return D2{p.v + s, p.a, p.b}; }
__device__ __forceinline__ D2 operator*(D2 p, D2 q) { return D2{p.v * q.v, p.a * q.v + p.v * q.a, p.b * q.v + p.v * q.b}; }
__device__ __forceinline__ D2 operator/(D2 p, D2 q)
{
    const float r = p.v / q.v;
    return D2{r, (p.a - r * q.a) / q.v, (p.b - r * q.b) / q.v};
}
__device__ __forceinline__ D2 dsqrt(D2 p)
{
    const float r = sqrtf(p.v);
    const float h = 0.5f / r;
    return D2{r, p.a * h, p.b * h};
}

// homography_from_center and its derivatives with respect to (x, y).
__device__ void homography_center_derivs(const float* C, const float* Tp, const float* Td, float x, float y,
                                         float* H, float* dHx, float* dHy)
{
    const D2 X{x, 1.f, 0.f}, Y{y, 0.f, 1.f};
    const D2 u = X * Tp[0] + Y * Tp[1] + Tp[2];
    const D2 v = X * Tp[3] + Y * Tp[4] + Tp[5];
    const D2 w = X * Tp[6] + Y * Tp[7] + Tp[8];
    const D2 xc = u / w, yc = v / w;
    const float Q11 = C[0], Q22 = C[4], Q33 = C[8];
    D2 h[9];
    h[0] = d2c(Q33);        h[1] = xc * yc * Q22;          h[2] = xc * (-Q33);
    h[3] = d2c(0.f);        h[4] = xc * xc * (-Q11) + (-Q33); h[5] = yc * (-Q33);
    h[6] = xc * (-Q11);     h[7] = yc * Q22;               h[8] = d2c(-Q33);
    const D2 e0 = dsqrt((xc * xc * Q11 + yc * yc * Q22 + Q33) * (Q22 * Q33 / Q11));
    const D2 e2 = dsqrt((xc * xc * Q11 + Q33) * (-Q22));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        h[i * 3 + 0] = h[i * 3 + 0] * e0;
        h[i * 3 + 1] = h[i * 3 + 1] * Q33;
        h[i * 3 + 2] = h[i * 3 + 2] * e2;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const D2 r = h[j] * Td[i * 3] + h[3 + j] * Td[i * 3 + 1] + h[6 + j] * Td[i * 3 + 2];
            H[i * 3 + j] = r.v;
            dHx[i * 3 + j] = r.a;
            dHy[i * 3 + j] = r.b;
        }
}

// Back-projected end of a cut (stop point through Hi, normalised) and its
// derivatives along the center, given dHi for both center coordinates.
__device__ __forceinline__ void back_project(const float* Hi, const float* dHi0, const float* dHi1, float px, float py,
                                             float& bx, float& by, float db[2][2])
{
    const float z0 = Hi[0] * px + Hi[1] * py + Hi[2];
    const float z1 = Hi[3] * px + Hi[4] * py + Hi[5];
    const float z2 = Hi[6] * px + Hi[7] * py + Hi[8];
    bx = z0 / z2;
    by = z1 / z2;
    const float* d[2] = {dHi0, dHi1};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float e0 = d[q][0] * px + d[q][1] * py + d[q][2];
        const float e1 = d[q][3] * px + d[q][4] * py + d[q][5];
        const float e2 = d[q][6] * px + d[q][7] * py + d[q][8];
        db[q][0] = (e0 - bx * e2) / z2;
        db[q][1] = (e1 - by * e2) / z2;
    }
}

// dHi = -Hi dH Hi
__device__ __forceinline__ void inverse_derivative(const float* Hi, const float* dH, float* dHi)
{
    float t[9];
    mat_mul(dH, Hi, t);
    mat_mul(Hi, t, dHi);
#pragma unroll
    for (int k = 0; k < 9; ++k) dHi[k] = -dHi[k];
}

// Sample k of a cut for Gauss-Newton at the trial homography S.gH: its value
// and, in ds, its derivatives along the two center coordinates (through H, and
// through the back-projected cut end (bx, by) whose derivatives are db).
template <bool STAGED>
__device__ __forceinline__ float gn_sample(const Shared& S, const SampleArea<STAGED>& area, float bs, float den,
                                          float bx, float by, const float db[2][2], int k, float ds[2])
{
    const float xs = bx * bs, ys = by * bs;
    const float sx = (bx - xs) / den, sy = (by - ys) / den;
    const float kf = float(k);
    const float x = __fmaf_rn(kf, sx, xs), y = __fmaf_rn(kf, sy, ys);
    const float t = bs + kf * (1.f - bs) / den;
    const float* Hm = S.gH;
    const float u = hrow(Hm, 0, x, y), v = hrow(Hm, 1, x, y), w = hrow(Hm, 2, x, y);
    const float r = __frcp_rn(w);
    const float qx = __fmul_rn(u, r), qy = __fmul_rn(v, r);
    float gx, gy;
    uint32_t pb[4];
    float p[4], fx, fy;
    area_taps(area, qx, qy, pb, fx, fy);
#pragma unroll
    for (int q = 0; q < 4; ++q) p[q] = byte_to_float(pb[q]);
    const float val = bilinear_value_grad(p, fx, fy, gx, gy);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const float* dH = S.gdH[q];
        const float dxq = __fmul_rn(t, db[q][0]), dyq = __fmul_rn(t, db[q][1]);
        const float du = __fmaf_rn(Hm[0], dxq, __fmaf_rn(Hm[1], dyq, hrow(dH, 0, x, y)));
        const float dv = __fmaf_rn(Hm[3], dxq, __fmaf_rn(Hm[4], dyq, hrow(dH, 1, x, y)));
        const float dw = __fmaf_rn(Hm[6], dxq, __fmaf_rn(Hm[7], dyq, hrow(dH, 2, x, y)));
        const float ex = __fmul_rn(__fmaf_rn(-qx, dw, du), r);
        const float ey = __fmul_rn(__fmaf_rn(-qy, dw, dv), r);
        ds[q] = __fmaf_rn(gx, ex, __fmul_rn(gy, ey));
    }
    return val;
}

// The Gauss-Newton sums of one chunk (lane = sample): cost, J^T r and J^T J
// of the residuals s_ik - mean_k, from per-lane shifted FP32 sums over the
// valid cuts in cut order, then FP64 over the lanes.  at(c, v, a, b) reads
// sample value v and its center derivatives a, b of cut c.
template <class At>
__device__ __forceinline__ void gn_chunk_sums(uint32_t valid, int n, bool live, double acc[6], At at)
{
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = 0.0;
    if (live && n >= 2) {
        float v0 = 0.f, s1 = 0.f, s2 = 0.f, a1 = 0.f, b1 = 0.f, aa = 0.f, ab = 0.f, bb = 0.f, ad = 0.f, bd = 0.f;
        bool first = true;
        uint32_t m = valid;
        while (m) {
            const int c = __ffs(m) - 1;
            m &= m - 1;
            float v, a, b;
            at(c, v, a, b);
            if (first) {
                v0 = v;
                first = false;
            }
            const float d = __fsub_rn(v, v0);
            s1 = __fadd_rn(s1, d);
            s2 = __fmaf_rn(d, d, s2);
            a1 = __fadd_rn(a1, a);
            b1 = __fadd_rn(b1, b);
            aa = __fmaf_rn(a, a, aa);
            ab = __fmaf_rn(a, b, ab);
            bb = __fmaf_rn(b, b, bb);
            ad = __fmaf_rn(a, d, ad);
            bd = __fmaf_rn(b, d, bd);
        }
        const float fn = float(n);
        acc[0] = double(__fsub_rn(__fmul_rn(fn, s2), __fmul_rn(s1, s1)));
        acc[1] = double(__fsub_rn(ad, __fdiv_rn(__fmul_rn(a1, s1), fn)));
        acc[2] = double(__fsub_rn(bd, __fdiv_rn(__fmul_rn(b1, s1), fn)));
        acc[3] = double(__fsub_rn(aa, __fdiv_rn(__fmul_rn(a1, a1), fn)));
        acc[4] = double(__fsub_rn(ab, __fdiv_rn(__fmul_rn(a1, b1), fn)));
        acc[5] = double(__fsub_rn(bb, __fdiv_rn(__fmul_rn(b1, b1), fn)));
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = lane_sum(acc[q]);
}

// Levenberg-Marquardt on the cut-consistency cost (CCTAGB_REFINE_GAUSS_NEWTON):
// residuals r_ik = s_ik - mean_k over the valid cuts i and samples k, whose
// sum of squares is the reference's pair cost up to the factor n / pairs;
// Jacobian d r_ik / d center from the forward derivatives of the trial
// homography, its inverse (which moves the back-projected cut ends) and the
// bilinear patch.  Each block of the cluster sums its chunks; the sums meet
// through distributed shared memory and every block takes the same step.
// Starts from the grid's center; a step that raises the cost is rejected and
// the damping raised.  Stops when a step is below 1e-3 px, or after
// gnIterations cost evaluations.
template <bool CLUSTER>
__device__ void gn_refine(Shared& S, void* work, int room, const uint8_t* px, const IdentTask& T, const Roi& roi,
                          const IdentParams& ip, uint32_t cutMask, int crank, int csize)
{
    namespace cg = cooperative_groups;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nthreads = blockDim.x, nwarps = nthreads >> 5;
    GnChunk& chunk = *static_cast<GnChunk*>(work);
    const int nS = ip.nSamples;
    const int nch = (nS + kChunk - 1) / kChunk;
    const float bs = ip.beginSig;
    const float den = float(nS) - 1.f;
    if (tid == 0) {
        S.gTry[0] = S.cx;
        S.gTry[1] = S.cy;
        S.gHave = 0;
        S.gStop = 0;
        S.gLambda = 1e-3;
    }
    __syncthreads();
    for (int it = 0; it < ip.gnIterations; ++it) {
        if (tid == 0) {
            homography_center_derivs(S.C, S.Tp, S.Td, S.gTry[0], S.gTry[1], S.gH, S.gdH[0], S.gdH[1]);
            if (!mat_inv(S.gH, S.gHi)) {
                S.gStop = 1;
            } else {
                inverse_derivative(S.gHi, S.gdH[0], S.gdHi[0]);
                inverse_derivative(S.gHi, S.gdH[1], S.gdHi[1]);
            }
        }
        __syncthreads();
        if (S.gStop) break;
        // cuts whose end samples leave the rectangle at this center, and (once
        // per cut) their back-projected ends
        if (warp == nwarps - 1 && lane < T.ncuts) {
            float bx, by, db[2][2];
            back_project(S.gHi, S.gdHi[0], S.gdHi[1], T.stop[lane][0], T.stop[lane][1], bx, by, db);
            float* o = S.gBack[lane];
            o[0] = bx;
            o[1] = by;
            o[2] = db[0][0];
            o[3] = db[0][1];
            o[4] = db[1][0];
            o[5] = db[1][1];
        }
        if (warp == 0) {
            bool bad = false, out = false;
            if (lane < T.ncuts) {
                float bx, by, w;
                apply_h(S.gHi, T.stop[lane][0], T.stop[lane][1], bx, by, w);
                const float xs = bx * bs, ys = by * bs;
                const float sx = (bx - xs) / den, sy = (by - ys) / den;
                float x0, y0, w0, x1, y1, w1;
                apply_h(S.gH, xs, ys, x0, y0, w0);
                apply_h(S.gH, xs + den * sx, ys + den * sy, x1, y1, w1);
                bad = !(w0 > 0.f && w1 > 0.f) && !(w0 < 0.f && w1 < 0.f);
                bad = bad || !inside(roi, x0, y0) || !inside(roi, x1, y1);
                out = !bad && !(in_box(S, roi, x0, y0) && in_box(S, roi, x1, y1));
            }
            const uint32_t m = __ballot_sync(0xffffffffu, bad);
            out = __any_sync(0xffffffffu, out);
            if (lane == 0) {
                S.gOob = m & cutMask;
                S.direct = out;
            }
        }
        __syncthreads();
        const uint32_t valid = ~(S.oob | S.gOob) & cutMask;
        const int n = __popc(valid);
        const int par = it & 1;
        // One block doing every chunk, with room for all samples: the threads
        // compute the samples, then a warp sums a chunk.  The per-chunk sums
        // are the same operations in the same order as the chunk-at-a-time
        // path, so both give the same bits.
        const bool direct = S.direct;
        auto sample = [&](int c, int k, float ds[2]) {
            const float* o = S.gBack[c];
            const float db[2][2] = {{o[2], o[3]}, {o[4], o[5]}};
            return direct ? gn_sample(S, image_area(roi), bs, den, o[0], o[1], db, k, ds)
                          : gn_sample(S, staged_area(S, px), bs, den, o[0], o[1], db, k, ds);
        };
        if (!CLUSTER && nwarps <= kMaxChunks) {
            // a small block, one of several on its SM: a warp takes a chunk's
            // samples and sums them as they come
            for (int j = warp; j < nch; j += nwarps) {
                const int k = j * kChunk + lane;
                double acc[6];
                gn_chunk_sums(valid, n, k < nS, acc, [&](int c, float& v, float& a, float& b) {
                    float ds[2];
                    v = sample(c, k, ds);
                    a = ds[0];
                    b = ds[1];
                });
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 6; ++q) S.gPart[par][j][q] = acc[q];
            }
            __syncthreads();
        } else if (!CLUSTER && T.ncuts * nS <= room) {
            float* gs = static_cast<float*>(work);
            float* gdx = gs + room;
            float* gdy = gdx + room;
            for (int i = tid; i < T.ncuts * nS; i += nthreads) {
                const int c = i / nS;
                if (!((valid >> c) & 1u)) continue;
                float ds[2];
                gs[i] = sample(c, i - c * nS, ds);
                gdx[i] = ds[0];
                gdy[i] = ds[1];
            }
            __syncthreads();
            for (int j = warp; j < nch; j += nwarps) {
                const int k = j * kChunk + lane;
                double acc[6];
                gn_chunk_sums(valid, n, k < nS, acc, [&](int c, float& v, float& a, float& b) {
                    v = gs[c * nS + k];
                    a = gdx[c * nS + k];
                    b = gdy[c * nS + k];
                });
                if (lane == 0)
#pragma unroll
                    for (int q = 0; q < 6; ++q) S.gPart[par][j][q] = acc[q];
            }
            __syncthreads();
        } else {
            for (int j = crank; j < nch; j += csize) {
                // this chunk's samples: value and its derivatives along the center
                const int k = j * kChunk + lane;
                for (int c = warp; c < T.ncuts; c += nwarps) {
                    if (!((valid >> c) & 1u) || k >= nS) continue;
                    float ds[2];
                    chunk.s[c][lane] = sample(c, k, ds);
                    chunk.dx[c][lane] = ds[0];
                    chunk.dy[c][lane] = ds[1];
                }
                __syncthreads();
                if (warp == 0) {
                    double acc[6];
                    gn_chunk_sums(valid, n, k < nS, acc, [&](int c, float& v, float& a, float& b) {
                        v = chunk.s[c][lane];
                        a = chunk.dx[c][lane];
                        b = chunk.dy[c][lane];
                    });
                    if (lane == 0)
#pragma unroll
                        for (int q = 0; q < 6; ++q) S.gPart[par][j][q] = acc[q];
                }
                __syncthreads();
            }
        }
        // every chunk's sums are in; a parity's array is rewritten two
        // evaluations later, past the next barrier of the cluster
        if constexpr (CLUSTER) cg::this_cluster().sync();
        if (warp == 0 && lane < 6) {
            double a = 0.0;
            for (int j = 0; j < nch; ++j) {
                const double* src = &S.gPart[par][j][0];
                if constexpr (CLUSTER) src = cg::this_cluster().map_shared_rank(src, j % csize);
                a += src[lane];
            }
            S.gSum[lane] = a;
        }
        __syncthreads();
        if (tid == 0) {
            const double cost = n >= 2 ? S.gSum[0] / (0.5 * double(n) * double(n - 1)) : DBL_MAX;
            ++S.iterations;
            if (n >= 2 && (!S.gHave || cost < S.gBest)) {
                S.gHave = 1;
                S.gBest = cost;
                S.cx = S.gTry[0];
                S.cy = S.gTry[1];
                S.oob |= S.gOob;
                for (int q = 0; q < 9; ++q) S.Hopt[q] = S.gH[q];
                S.minRes = float(cost);
                S.gG[0] = S.gSum[1];
                S.gG[1] = S.gSum[2];
                S.gA[0] = S.gSum[3];
                S.gA[1] = S.gSum[4];
                S.gA[2] = S.gSum[5];
                S.gLambda = fmax(S.gLambda * 0.1, 1e-7);
            } else {
                S.gLambda *= 10.0;
            }
            if (!S.gHave) {
                S.gStop = 1;
            } else {
                const double a = S.gA[0] * (1.0 + S.gLambda), b = S.gA[1], c = S.gA[2] * (1.0 + S.gLambda);
                const double det = a * c - b * b;
                if (!(det > 0.0)) {
                    S.gStop = 1;
                } else {
                    const double dx = -(c * S.gG[0] - b * S.gG[1]) / det;
                    const double dy = -(a * S.gG[1] - b * S.gG[0]) / det;
                    if (dx * dx + dy * dy < 1e-6) S.gStop = 1;
                    S.gTry[0] = float(double(S.cx) + dx);
                    S.gTry[1] = float(double(S.cy) + dy);
                }
            }
        }
        __syncthreads();
        if (S.gStop) break;
    }
}

}  // namespace

// One marker per cluster (CLUSTER, blocks of one marker side by side) or per
// block; any number of warps up to kIdentTrialWarps.  72 registers: 25 warps on an SM put 7
// on one of its four register partitions (one block of 25, or two of 12).
// TRIALS: one block per marker with a warp per trial, no pixels staged (grid only).
template <bool CLUSTER, bool TRIALS>
__global__ void __maxnreg__(72)
    k_identify(const uint8_t* __restrict__ img, size_t pitch, const IdentTask* __restrict__ tasks, IdentResult* res,
               const float* __restrict__ bankInv, IdentParams ip, int workBytes, int boxBytes)
{
    namespace cg = cooperative_groups;
    __shared__ Shared S;
    extern __shared__ float4 work[];  // workBytes, then room for boxBytes of pixels; at least FinalWork
    uint8_t* const px = reinterpret_cast<uint8_t*>(work) + workBytes;
    FinalWork& F = *reinterpret_cast<FinalWork*>(work);
    int crank = 0, csize = 1;
    if constexpr (CLUSTER) {
        crank = int(cg::this_cluster().block_rank());
        csize = int(cg::this_cluster().num_blocks());
    }
    const int marker = blockIdx.x / csize;
    const IdentTask& T = tasks[marker];
    const Roi roi = make_roi(img, pitch, T);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nthreads = blockDim.x, nwarps = nthreads >> 5;
    const int nS = ip.nSamples;
    const int nch = (nS + kChunk - 1) / kChunk;
    const int gridN = ip.gridN;
    const int nTrials = gridN * gridN;
    const uint32_t cutMask = (T.ncuts >= 32) ? 0xffffffffu : ((1u << T.ncuts) - 1u);
    if (T.ncuts <= 0) {  // nothing to refine or read (identify_step_1 stopped it)
        if (tid == 0 && crank == 0) {
            IdentResult& R0 = res[marker];
            R0 = IdentResult{};
            R0.x = T.x0;
            R0.y = T.y0;
            R0.id = -1;
            R0.status = CCTAGB_NO_SELECTED_CUTS;
        }
        return;
    }
    // A block's shared memory may be reached from another one once it runs: each
    // arrives here (the return above is taken by whole clusters) and waits before
    // the rounds, whose shares go to every block, behind the set-up and staging.
    if constexpr (CLUSTER) cg::this_cluster().barrier_arrive();

    if (tid == 0) {
        canonic_form(T.Q, S.C, S.Tp, S.Td);
        // conditionerFromEllipse (conditioner.hpp:22-44) with meanAB of this ellipse
        const float sqrt2 = sqrtf(2.f);
        const float meanAB = (T.a + T.b) / 2.f;
        float mT[9] = {sqrt2 / meanAB, 0.f, -sqrt2 * T.cx / meanAB, 0.f, sqrt2 / meanAB, -sqrt2 * T.cy / meanAB,
                       0.f, 0.f, 1.f};
        float mTi[9];
        // no conditioner for axes of no or unlimited mean: no trial center then
        if (!mat_inv(mT, mTi))
            for (int k = 0; k < 9; ++k) mTi[k] = NAN;
        float tq[9], Qc[9], mTiT[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) mTiT[i * 3 + j] = mTi[j * 3 + i];
        mat_mul(T.Q, mTi, tq);
        mat_mul(mTiT, tq, Qc);
        float ca, cb;
        conic_axes(Qc, ca, cb);
        S.nsScale = fmaxf(ca, cb);
        for (int k = 0; k < 9; ++k) {
            S.mT[k] = mT[k];
            S.mTi[k] = mTi[k];
        }
        S.cx = T.x0;
        S.cy = T.y0;
        S.minRes = FLT_MAX;
        S.oob = 0u;
        S.fail = 0;
        // refineConicFamilyGlob loop bound (Identification.cpp:869-885)
        const float maxSemiAxis = fmaxf(T.a, T.b);
        float ns = ip.neighbourSize;
        int r = 0;
        while (ns * maxSemiAxis > 0.02f && r < 64) {
            ++r;
            ns /= float((gridN - 1) / 2);
        }
        if (ip.refineMode == CCTAGB_REFINE_GAUSS_NEWTON) r = min(r, ip.coarseRounds);
        S.rounds = r;
        S.iterations = r;
    }
    if (warp == 2) find_box(S, T, roi, size_t(boxBytes), lane);
    if (tid == 32) {  // plane radii of the samples, by the reference's running sum
        const float step = (1.f - ip.beginSig) / (float(nS) - 1.f);
        float x = ip.beginSig;
        for (int k = 0; k < nS; ++k) {
            S.radius[k] = x;
            x += step;
        }
    }
    for (int i = tid; i <= kMaxSamples; i += nthreads) S.rcp[i] = __frcp_rn(float(i));
    __syncthreads();
    stage_box(S, roi, px);
    asm volatile("cp.async.wait_all;" ::: "memory");  // before the first barrier below
    const TrialLines lines = trial_lines(work, nTrials, T.ncuts);
    Tasks K{nTrials, nS / kChunk, nS % kChunk, 1, 0};
    while (K.width < K.tail) K.width <<= 1;
    K.packed = kChunk / K.width;
    if constexpr (CLUSTER) cg::this_cluster().barrier_wait();
    float ns = ip.neighbourSize;
    for (int round = 0; round < S.rounds; ++round) {
        // getNearbyPoints (Identification.cpp:1071-1109): a lane per trial
        if (tid == 32) S.direct = 0;
        if (warp == 0 && lane < nTrials) {
            const float size = ns * S.nsScale;
            const float half = size / 2.f, step = size / float(gridN - 1);
            const float ccx = S.mT[0] * S.cx + S.mT[1] * S.cy + S.mT[2];
            const float ccy = S.mT[3] * S.cx + S.mT[4] * S.cy + S.mT[5];
            const int i = lane / gridN, j = lane % gridN;
            const float qx = ccx - half + float(i) * step, qy = ccy - half + float(j) * step;
            float px, py, w;
            apply_h(S.mTi, qx, qy, px, py, w);
            float Hm[9], Hi[9];
            homography_from_center(S.C, S.Tp, S.Td, px, py, Hm);
            const bool ok = mat_inv(Hm, Hi);
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                S.trialH[lane][k] = Hm[k];
                S.trialHi[lane][k] = Hi[k];
            }
            S.trialOk[lane] = ok;
            S.trialOob[lane] = 0u;
            S.trialPt[lane][0] = px;
            S.trialPt[lane][1] = py;
        }
        __syncthreads();
        for (int i = tid; i < nTrials * T.ncuts; i += nthreads) {
            const int t = i / T.ncuts;
            setup_cut(S, lines, T, t, i - t * T.ncuts, ip, roi);
        }
        __syncthreads();
        // sticky out-of-bounds flags in trial order (every warp for itself):
        // inclusive OR scan; lane t then holds trial t's valid cuts
        uint32_t flags = lane < nTrials ? S.trialOob[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, flags, o);
            if (lane >= o) flags |= v;
        }
        flags |= S.oob;
        const uint32_t valid = lane < nTrials ? ~flags & cutMask : 0u;
        const int par = round & 1;
        const int firstTask = crank * nwarps + warp, stepTask = csize * nwarps;
        if constexpr (TRIALS) {
            double c[kMaxChunks];
            trial_chunks(lines, image_area(roi), warp, __shfl_sync(0xffffffffu, valid, warp), nS, lane, c);
#pragma unroll
            for (int q = 0; q < kMaxChunks; ++q)
                if (lane == 0) S.part[par][q][warp] = c[q];
        } else if (S.direct) {
            sample_round(S, lines, image_area(roi), K, valid, par, firstTask, stepTask, csize, lane);
        } else {
            sample_round(S, lines, staged_area(S, px), K, valid, par, firstTask, stepTask, csize, lane);
        }
        // All chunks of the marker are in, in every block; this parity's array
        // is written again two rounds later, after the next cluster barrier,
        // when every block has finished reading it.
        if constexpr (CLUSTER) cg::this_cluster().sync();
        else __syncthreads();
        if (warp == 0) {
            double acc = 0.0;
            if (lane < nTrials)
                for (int j = 0; j < nch; ++j) acc += S.part[par][j][lane];
            const int n = __popc(valid);
            const float cost = n >= 2 ? float(acc / (0.5 * double(n) * double(n - 1))) : FLT_MAX;
            // imageCenterOptimizationGlob: first strict minimum in trial order
            // (costs below FLT_MAX; key = orderable cost bits, then index)
            unsigned long long key = ~0ull;
            if (lane < nTrials && cost < FLT_MAX) {
                const uint32_t b = __float_as_uint(cost);
                const uint32_t ord = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
                key = (static_cast<unsigned long long>(ord) << 32) | unsigned(lane);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
                key = k2 < key ? k2 : key;
            }
            const bool readable = __any_sync(0xffffffffu, n >= 2);
            const uint32_t last = __shfl_sync(0xffffffffu, flags, nTrials - 1);
            const int bi = int(key & 0xffffffffull);
            const bool found = readable && key != ~0ull;
            if (found && lane < 9) S.Hopt[lane] = S.trialH[bi][lane];
            if (found && lane == bi) {
                S.cx = S.trialPt[bi][0];
                S.cy = S.trialPt[bi][1];
                S.minRes = cost;
            }
            if (lane == 0) {
                S.oob = last;
                if (!found) S.fail = 1;
            }
        }
        __syncthreads();
        if (S.fail) break;
        ns /= float((gridN - 1) / 2);
    }
    if (!TRIALS && ip.refineMode == CCTAGB_REFINE_GAUSS_NEWTON && !S.fail && S.rounds > 0)
        gn_refine<CLUSTER>(S, work, workBytes / int(3 * sizeof(float)), px, T, roi, ip, cutMask, crank, csize);
    const bool read = !S.fail && S.rounds > 0;
    IdentResult& R = res[marker];
    if (!read && tid == 0 && crank == 0) {
        R.status = CCTAGB_OPTI_HAS_DIVERGED;
        R.id = -1;
        R.x = S.cx;
        R.y = S.cy;
        for (int k = 0; k < 9; ++k) R.H[k] = 0.f;
        R.residual = FLT_MAX;
        R.score = 0.f;
        R.nvalid = 0;
        R.iterations = S.iterations;
    }
    // The reading of the cuts is spread over the cluster: the first block takes
    // the signals of all cuts, for the barcode; the others (or the only one) the
    // cuts' distances to the bank, a share each.  No block leaves while another
    // may still use its shared memory.
    if (!read) {
        if constexpr (CLUSTER) cg::this_cluster().sync();
        return;
    }
    const int shares = csize > 1 ? csize - 1 : 1, share = csize > 1 ? crank - 1 : 0;  // share -1: none
    auto mine = [&](int c) { return share >= 0 && c % shares == share; };
    // Final signals with the optimal homography (getSignals, Identification.cpp:901).
    {
        float Hi[9];
        mat_inv(S.Hopt, Hi);
        __syncthreads();  // the rounds' use of the work area is over
        const int first = crank == 0 ? 0 : share, step = crank == 0 ? 1 : shares;
        for (int c = first + step * warp; c < T.ncuts; c += step * nwarps) {
            float bx, by, w;
            apply_h(Hi, T.stop[c][0], T.stop[c][1], bx, by, w);
            const float xs = bx * ip.beginSig, ys = by * ip.beginSig;
            const float sx = (bx - xs) / (float(nS) - 1.f), sy = (by - ys) / (float(nS) - 1.f);
            bool bad = false;
#pragma unroll
            for (int q = 0; q < kMaxChunks; ++q) {
                const int k = q * 32 + lane;
                if (k >= nS) continue;
                const float x = xs + float(k) * sx, y = ys + float(k) * sy;
                float xr, yr;
                apply_h(S.Hopt, x, y, xr, yr, w);
                if (inside(roi, xr, yr)) F.sig[c][k] = bilinear(roi, xr, yr);
                else bad = true;
            }
            const uint32_t any = __ballot_sync(0xffffffffu, bad);
            if (lane == 0 && any) atomicOr(&S.oob, 1u << c);
        }
    }
    // Bank row i sees a sample as black when it lies inside an odd number of its
    // rings (1 / ratio <= radius): per ring, all samples from the first one at
    // least that far out flip.
    for (int i = tid; share >= 0 && i < ip.nIds; i += nthreads) {
        uint32_t bits[kMaxSamples / 32] = {};
        for (int r = 0; r < ip.nRatios; ++r) {
            const float inv = __ldg(&bankInv[i * kMaxBankRatios + r]);
            int k = min(max(int((inv - ip.beginSig) / (1.f - ip.beginSig) * (float(nS) - 1.f)), 0), nS);
            while (k > 0 && S.radius[k - 1] >= inv) --k;
            while (k < nS && S.radius[k] < inv) ++k;
#pragma unroll
            for (int w = 0; w < kMaxSamples / 32; ++w)
                bits[w] ^= k <= 32 * w ? 0xffffffffu : k >= 32 * w + 32 ? 0u : 0xffffffffu << (k - 32 * w);
        }
#pragma unroll
        for (int w = 0; w < kMaxSamples / 32; ++w) F.black[i][w] = bits[w];
    }
    __syncthreads();
    const uint32_t valid = ~S.oob & cutMask;  // beyond the first block: of its own cuts
    const int nValid = __popc(valid);
    // Statistics of each cut's signal (Identification.cpp:77-190), a lane per cut
    // (the last warp: the first ones sort meanwhile).
    if (warp == nwarps - 1) {
        const int c = lane;
        if (c < T.ncuts && mine(c) && ((valid >> c) & 1u)) {
            const float* sg = F.sig[c];
            // over samples [30, n): Boost immediate mean / variance (the
            // divisions by the counts correctly rounded by div_small)
            float mean = 0.f, var = 0.f;
#pragma unroll 4
            for (int k = 30; k < nS; ++k) {
                const int cnt = k - 29;
                const float x = sg[k];
                const float fc = float(cnt), fc1 = float(cnt - 1), rc = S.rcp[cnt];
                mean = pm::div_small(__fmaf_rn(mean, fc1, x), fc, rc);
                const float t = __fsub_rn(x, mean);
                const float v = __fadd_rn(pm::div_small(__fmul_rn(var, fc1), fc, rc),
                                          pm::div_small(__fmul_rn(t, t), fc1, S.rcp[cnt - 1]));
                if (cnt > 1) var = v;
            }
            // running means of the samples below the mean and of the others,
            // from the first one below it
            float mub = 0.f, muw = 0.f;
            int nb = 0, nw = 0;
#pragma unroll 4
            for (int k = 0; k < nS; ++k) {
                const float x = sg[k];
                const bool below = x < mean, use = below || nb > 0;
                const int n1 = below ? nb : nw;
                const float mu = below ? mub : muw;
                const float m = pm::div_small(__fmaf_rn(mu, float(n1), x), float(n1 + 1), S.rcp[n1 + 1]);
                mub = use && below ? m : mub;
                muw = use && !below ? m : muw;
                nb += below ? 1 : 0;
                nw += use && !below ? 1 : 0;
            }
            // dis()'s division by 2 var: a float quotient through the double
            // reciprocal is correctly rounded for a normal result (its relative
            // error, 2^-52, is below the 2^-49 that separates a quotient of floats
            // from a float rounding midpoint), so each term is the IEEE quotient.
            const double rvar2 = 1.0 / double(2.0f * var);
            S.stats[c][0] = mub;
            S.stats[c][1] = muw;
            S.stats[c][2] = __int_as_float(__double2hiint(rvar2));
            S.stats[c][3] = __int_as_float(__double2loint(rvar2));
        }
    }
    // Median barcode over the valid cuts (computeMedian, Identification.hpp:
    // 351-371): a thread per sample sorts its values in registers by Batcher's
    // odd-even merge network, absent cuts last.
    if (crank == 0)
        for (int k = tid; k < nS; k += nthreads) {
            float v[kMaxCuts];
#pragma unroll
            for (int c = 0; c < kMaxCuts; ++c) v[c] = c < T.ncuts && ((valid >> c) & 1u) ? F.sig[c][k] : FLT_MAX;
            sort_network<1, 1>(v);
            float hi = 0.f, lo = 0.f;
#pragma unroll
            for (int c = 0; c < kMaxCuts; ++c) {
                hi = c == nValid / 2 ? v[c] : hi;
                lo = c == nValid / 2 - 1 ? v[c] : lo;
            }
            F.barcode[k] = nValid == 0 ? 0.f : (nValid & 1) ? hi : float((double(hi) + double(lo)) / 2.0);
        }
    __syncthreads();
    // Orazio distance per valid cut, a warp per cut, lane = bank id (four rows of
    // 32): a sample adds one of two terms, by the row's black mask, in order.
    // The terms sit in the lanes' registers, sample k's in lane k mod 32.
    for (int c = share + shares * warp; share >= 0 && c < T.ncuts; c += shares * nwarps) {
        if (!((valid >> c) & 1u)) continue;
        const float mub = S.stats[c][0], muw = S.stats[c][1];
        const double rvar2 = __hiloint2double(__float_as_int(S.stats[c][2]), __float_as_int(S.stats[c][3]));
        float dist[kMaxBankIds / 32] = {};
        for (int w = 0; w < nch; ++w) {
            const int k = 32 * w + lane;
            // past the last sample both terms are 0
            const float x = F.sig[c][min(k, nS - 1)];
            const float tw = k < nS ? dis_r(x, true, mub, muw, rvar2) : 0.f;
            const float tb = k < nS ? dis_r(x, false, mub, muw, rvar2) : 0.f;
            uint32_t bits[kMaxBankIds / 32];
#pragma unroll
            for (int q = 0; q < kMaxBankIds / 32; ++q) bits[q] = F.black[32 * q + lane][w];
#pragma unroll
            for (int b = 0; b < 32; ++b) {
                if (b % 4 == 0 && 32 * w + b >= nS) break;
                const float aw = __shfl_sync(0xffffffffu, tw, b), ab = __shfl_sync(0xffffffffu, tb, b);
#pragma unroll
                for (int q = 0; q < kMaxBankIds / 32; ++q) dist[q] += (bits[q] & (1u << b)) ? ab : aw;
            }
        }
        // std::map<float, id> keeps, for equal keys, the id inserted last: the
        // winner is the largest v, ties to the largest id.  v >= 0, so its bit
        // pattern orders like the value; (bits << 32 | id) orders like the map.
        unsigned long long best = 0ull;
#pragma unroll
        for (int q = 0; q < kMaxBankIds / 32; ++q) {
            const int idc = 32 * q + lane;
            const float v = expf(-dist[q]);
            const unsigned long long key = (static_cast<unsigned long long>(__float_as_uint(v)) << 32) | unsigned(idc);
            if (idc < ip.nIds && key > best) best = key;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(0xffffffffu, best, o);
            best = ok > best ? ok : best;
        }
        if (lane == 0) {
            Shared* first = &S;
            if constexpr (CLUSTER) first = cg::this_cluster().map_shared_rank(&S, 0);
            first->winner[c] = int(best & 0xffffffffull);
            first->vwin[c] = __uint_as_float(unsigned(best >> 32));
        }
    }
    if constexpr (CLUSTER) {
        cg::this_cluster().sync();
        if (crank != 0) return;
    } else {
        __syncthreads();
    }
    if (warp == 0) {
        // ID vote (Identification.cpp:1408-1431): most-voted id (first on ties),
        // score = mean probability of its votes; a lane per cut.
        const bool votes = lane < T.ncuts && ((valid >> lane) & 1u);
        const int own = votes ? S.winner[lane] : -1;
        const int n = __popc(__match_any_sync(0xffffffffu, own));
        // the largest count, then the least id
        unsigned key = votes ? (unsigned(n) << 16) | unsigned(0xffff - own) : 0u;
        key = __reduce_max_sync(0xffffffffu, key);
        const int iMax = key ? 0xffff - int(key & 0xffffu) : 0;
        const int maxSize = int(key >> 16);
        float vmin = FLT_MAX, vmax = -FLT_MAX;
        for (int k = lane; k < nS; k += 32) {
            vmin = fminf(vmin, F.barcode[k]);
            vmax = fmaxf(vmax, F.barcode[k]);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
            vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        }
        if (lane == 0) {
            float score = 0.f;
            for (int c = 0; c < T.ncuts; ++c)
                if (((valid >> c) & 1u) && S.winner[c] == iMax) score += S.vwin[c];
            score /= float(maxSize);
            const float residual = sqrtf(S.minRes) / (vmax - vmin);
            R.x = S.cx;
            R.y = S.cy;
            for (int k = 0; k < 9; ++k) R.H[k] = S.Hopt[k];
            R.residual = residual;
            R.nvalid = nValid;
            R.iterations = S.iterations;
            if (residual > 2.7f || !(residual == residual)) {
                R.status = CCTAGB_OPTI_HAS_DIVERGED;
                R.id = -1;
                R.score = 0.f;
            } else {
                R.id = iMax;
                R.score = score;
                R.status = score > ip.minIdentProba ? CCTAGB_ID_RELIABLE : CCTAGB_ID_NOT_RELIABLE;
            }
        }
    }
}


namespace {

// Warps of a cost block: few while several blocks fill an SM, a warp per cut
// while the tasks are fewer than that.
constexpr int kCostWarps = 4;
template <int WARPS>
struct CostShared {
    float C[9], Tp[9], Td[9];
    float H[9], Hi[9], dH[2][9];
    float4 cut[kMaxCuts];         // first plane point and step of each cut
    float4 end[kMaxCuts];         // back-projected cut end, step from the unrounded first point
    float scale[kMaxCuts];        // its scale
    float t[kMaxSamples];         // the samples' plane radii
    float mean[kMaxSamples];
    float dz[kMaxCuts][3];        // d cost / d (Hi p) of each cut's end
    double red[WARPS][10];
    double m[2][9];
    uint32_t oob;
    int bad;
};

// A sample's image point under H, and 1 / w.  The two quotients by one rounded
// reciprocal and a remainder step each (pm::div_small's, for any divisor).  An
// invertible H has a line that it sends to infinity: a sample on it, or so near that
// 1 / w overflows, gets NaN or an infinity, which inside() refuses, so its cut is
// dropped, as with the quotient itself (an infinity, or beyond any image).
__device__ __forceinline__ void cost_point(const float* H, float x, float y, float& qx, float& qy, float& rw)
{
    const float u = H[0] * x + H[1] * y + H[2];
    const float v = H[3] * x + H[4] * y + H[5];
    const float w = H[6] * x + H[7] * y + H[8];
    rw = __frcp_rn(w);
    qx = pm::div_small(u, w, rw);
    qy = pm::div_small(v, w, rw);
}

__device__ void write_cost(float* o, float cost)
{
    o[0] = cost;
    for (int j = 1; j < 12; ++j) o[j] = 0.f;
}

}  // namespace

// Cut-consistency cost of one task at a given center and its adjoints (one
// block per task).  Pass 1 reads every sample (a sample outside the
// rectangle drops its cut, as extractSignalUsingHomography does); pass 2
// sends d cost / d s_ik = 2 n / pairs (s_ik - mean_k) back through the
// bilinear patch to the image position, from there to H directly and to the
// sample's marker-plane position, whose cut end is H^-1 applied to the stop
// point; the inverse's adjoint is -H^-T G H^-T.  The center gradient is the
// H gradient contracted with dH/dcenter (forward derivatives).
//
// Bound by the instructions of the samples once the serial steps of a task (its
// homography by one thread) hide behind the samples of others: so small blocks,
// several on an SM; the pixels of a sample kept from pass 1 for pass 2; the
// sums over the cuts by a lane per matrix entry.  Measured, 4096 tasks of 22
// cuts x 100 samples: blocks of 25 warps that read the pixels twice 419 us,
// 154 us now.
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, WARPS == kCostWarps ? 7 : 1)
    k_cut_cost(const uint8_t* __restrict__ img, size_t pitch, const IdentTask* __restrict__ tasks,
               const float* __restrict__ centers, float* out, IdentParams ip, int sampleCap)
{
    constexpr int kBlock = 32 * WARPS;
    __shared__ CostShared<WARPS> S;
    extern __shared__ float s_cost[];  // the samples, their four pixels and the corner, sampleCap each
    const IdentTask& T = tasks[blockIdx.x];
    const Roi roi = make_roi(img, pitch, T);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nS = ip.nSamples;
    float* const sig = s_cost;
    uint32_t* const pix = reinterpret_cast<uint32_t*>(s_cost + sampleCap);
    uint32_t* const cell = pix + sampleCap;
    const float bs = ip.beginSig;
    const float den = float(nS) - 1.f;
    float* o = out + 12 * size_t(blockIdx.x);
    const uint32_t cutMask = (T.ncuts >= 32) ? 0xffffffffu : ((1u << T.ncuts) - 1u);
    if (tid == 0) {
        canonic_form(T.Q, S.C, S.Tp, S.Td);
        homography_center_derivs(S.C, S.Tp, S.Td, centers[2 * blockIdx.x], centers[2 * blockIdx.x + 1], S.H,
                                 S.dH[0], S.dH[1]);
        S.bad = mat_inv(S.H, S.Hi) ? 0 : 1;
        S.oob = 0u;
    }
    for (int j = tid; j < kMaxCuts * 3; j += kBlock) S.dz[j / 3][j % 3] = 0.f;
    for (int k = tid; k < nS; k += kBlock) S.t[k] = bs + float(k) * (1.f - bs) / den;
    __syncthreads();
    if (S.bad) {
        if (tid == 0) write_cost(o, FLT_MAX);
        return;
    }
    if (tid < T.ncuts) {
        const float px = T.stop[tid][0], py = T.stop[tid][1];
        const float z0 = S.Hi[0] * px + S.Hi[1] * py + S.Hi[2];
        const float z1 = S.Hi[3] * px + S.Hi[4] * py + S.Hi[5];
        const float z2 = S.Hi[6] * px + S.Hi[7] * py + S.Hi[8];
        const float bx = z0 / z2, by = z1 / z2;
        const float xs = __fmul_rn(bx, bs), ys = __fmul_rn(by, bs);
        S.cut[tid] = make_float4(xs, ys, __fsub_rn(bx, xs) / den, __fsub_rn(by, ys) / den);
        S.end[tid] = make_float4(bx, by, __fmaf_rn(-bx, bs, bx) / den, __fmaf_rn(-by, bs, by) / den);
        S.scale[tid] = z2;
    }
    __syncthreads();
    float Hm[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) Hm[j] = S.H[j];
    // pass 1, the samples of all cuts in a row
    for (int c = tid / nS, k = tid - c * nS; c < T.ncuts;) {
        const float4 l = S.cut[c];
        const float x = l.x + float(k) * l.z, y = l.y + float(k) * l.w;
        float xr, yr, rw;
        cost_point(Hm, x, y, xr, yr, rw);
        if (inside(roi, xr, yr)) {
            const int px = int(xr), py = int(yr), at = c * nS + k;
            const uint8_t* p0 = roi.img + px + size_t(py) * roi.pitch;
            const uint8_t* p1 = p0 + roi.pitch;
            const uint32_t b0 = __ldg(p0), b1 = __ldg(p0 + 1), b2 = __ldg(p1), b3 = __ldg(p1 + 1);
            cell[at] = uint32_t(py) << 16 | (uint32_t(px) & 0xffffu);
            pix[at] = b0 | b1 << 8 | b2 << 16 | b3 << 24;
            const float fx = xr - float(px), fy = yr - float(py);
            const float fx1 = 1.0f - fx, fy1 = 1.0f - fy;
            sig[at] = (byte_to_float(b0) * (fx1 * fy1) + byte_to_float(b1) * (fx * fy1) +
                       byte_to_float(b2) * (fx1 * fy) + byte_to_float(b3) * (fx * fy)) / 2;
        } else {
            atomicOr(&S.oob, 1u << c);
        }
        for (k += kBlock; k >= nS; k -= nS) ++c;
    }
    __syncthreads();
    const uint32_t valid = ~S.oob & cutMask;
    const int n = __popc(valid);
    if (n < 2) {
        if (tid == 0) write_cost(o, FLT_MAX);
        return;
    }
    const double pairs = 0.5 * double(n) * double(n - 1);
    double costPart = 0.0;
    for (int k = tid; k < nS; k += kBlock) {
        double s1 = 0.0, s2 = 0.0;
        uint32_t m = valid;
        while (m) {
            const int c = __ffs(m) - 1;
            m &= m - 1;
            const double v = sig[c * nS + k];
            s1 += v;
            s2 += v * v;
        }
        S.mean[k] = float(s1 / double(n));
        costPart += double(n) * s2 - s1 * s1;
    }
    __syncthreads();
    double red[10];
    red[0] = costPart;
#pragma unroll
    for (int j = 1; j < 10; ++j) red[j] = 0.0;
    const float coef = float(2.0 * double(n) / pairs);
    for (int c = warp; c < T.ncuts; c += WARPS) {
        if (!((valid >> c) & 1u)) continue;
        const float4 l = S.end[c];
        float gH[9];  // of the lane's samples of this cut; over the cuts in double
#pragma unroll
        for (int j = 0; j < 9; ++j) gH[j] = 0.f;
        float gbx = 0.f, gby = 0.f;
        for (int k = lane; k < nS; k += 32) {
            // (pass 1 rounds the first point, so a sample may lie in the next patch)
            const float x = __fmaf_rn(l.x, bs, __fmul_rn(float(k), l.z));
            const float y = __fmaf_rn(l.y, bs, __fmul_rn(float(k), l.w));
            float qx, qy, rw;
            cost_point(Hm, x, y, qx, qy, rw);
            float fpx, fpy, gx, gy;
            const int px = floor_small(fmaxf(qx, 0.f), fpx), py = floor_small(fmaxf(qy, 0.f), fpy);
            uint32_t b = pix[c * nS + k];
            if ((uint32_t(py) << 16 | (uint32_t(px) & 0xffffu)) != cell[c * nS + k]) {
                // clamped, so that rounding at the border never reads outside
                const uint8_t* p0 = roi.img + min(max(px, roi.x0), roi.x1 - 2) +
                                    size_t(min(max(py, roi.y0), roi.y1 - 2)) * roi.pitch;
                const uint8_t* p1 = p0 + roi.pitch;
                b = uint32_t(__ldg(p0)) | uint32_t(__ldg(p0 + 1)) << 8 | uint32_t(__ldg(p1)) << 16 |
                    uint32_t(__ldg(p1 + 1)) << 24;
            }
            const float p[4] = {byte_to_float(b & 0xffu), byte_to_float((b >> 8) & 0xffu),
                                byte_to_float((b >> 16) & 0xffu), byte_to_float(b >> 24)};
            (void)bilinear_value_grad(p, qx - fpx, qy - fpy, gx, gy);
            const float lam = coef * (sig[c * nS + k] - S.mean[k]);
            const float fx = lam * gx, fy = lam * gy;
            const float fw = -(fx * qx + fy * qy);
            const float y3[3] = {x, y, 1.f};
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                gH[j] = fmaf(fx * rw, y3[j], gH[j]);
                gH[3 + j] = fmaf(fy * rw, y3[j], gH[3 + j]);
                gH[6 + j] = fmaf(fw * rw, y3[j], gH[6 + j]);
            }
            const float fX = (fx * (Hm[0] - qx * Hm[6]) + fy * (Hm[3] - qy * Hm[6])) * rw;
            const float fY = (fx * (Hm[1] - qx * Hm[7]) + fy * (Hm[4] - qy * Hm[7])) * rw;
            gbx = fmaf(S.t[k], fX, gbx);
            gby = fmaf(S.t[k], fY, gby);
        }
#pragma unroll
        for (int j = 0; j < 9; ++j) red[1 + j] += double(gH[j]);
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            gbx += __shfl_xor_sync(0xffffffffu, gbx, off);
            gby += __shfl_xor_sync(0xffffffffu, gby, off);
        }
        if (lane == 0) {
            const float z2 = S.scale[c];
            S.dz[c][0] = gbx / z2;
            S.dz[c][1] = gby / z2;
            S.dz[c][2] = -(gbx * l.x + gby * l.y) / z2;
        }
    }
#pragma unroll
    for (int j = 0; j < 10; ++j) {
#pragma unroll
        for (int off = 16; off; off >>= 1) red[j] += __shfl_xor_sync(0xffffffffu, red[j], off);
    }
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < 10; ++j) S.red[warp][j] = red[j];
    __syncthreads();
    if (warp != 0) return;
    // the cost and the nine entries of G over the warps, a lane each; the adjoint
    // of Hi from the cut ends, then -Hi^T GHi Hi^T into G
    double sum = 0.0;
    if (lane < 10)
        for (int w = 0; w < WARPS; ++w) sum += S.red[w][lane];
    const int e = min(max(lane - 1, 0), 8), r = e / 3, q = e - 3 * r;
    double g = 0.0;
    for (int c = 0; c < T.ncuts; ++c) {
        const double p = q == 2 ? 1.0 : double(T.stop[c][q]);
        g += double(S.dz[c][r]) * p;
    }
    if (lane >= 1 && lane < 10) S.m[0][e] = g;
    __syncwarp();
    double a = 0.0;  // M = GHi Hi^T
#pragma unroll
    for (int j = 0; j < 3; ++j) a += S.m[0][r * 3 + j] * double(S.Hi[q * 3 + j]);
    if (lane >= 1 && lane < 10) S.m[1][e] = a;
    __syncwarp();
    a = 0.0;  // Hi^T M
#pragma unroll
    for (int j = 0; j < 3; ++j) a += double(S.Hi[j * 3 + r]) * S.m[1][j * 3 + q];
    if (lane >= 1) sum -= a;
    if (lane >= 1 && lane < 10) {
        o[2 + lane] = float(sum);
        S.m[0][e] = sum;
    }
    __syncwarp();
    if (lane < 2) {
        double dc = 0.0;
#pragma unroll
        for (int j = 0; j < 9; ++j) dc += S.m[0][j] * double(S.dH[lane][j]);
        o[1 + lane] = float(dc);
    }
    if (lane == 0) o[0] = float(sum / pairs);
}

namespace {

// ---------------------------------------------------- FP64 check form --
// The same cost and adjoint as k_cut_cost, every step in double precision:
// the canonic form, the trial homography with its center derivatives, the
// back-projected cut ends, the sample positions and the bilinear reads.  It
// exists to check the adjoint's derivation against central differences at a
// precision the FP32 kernel cannot reach (FP32 sample positions alone move
// the cost by ~1e-4 of itself); the refinement kernels do not use it.
struct D2d {
    double v, a, b;
};
__device__ __forceinline__ D2d operator+(D2d p, D2d q) { return D2d{p.v + q.v, p.a + q.a, p.b + q.b}; }
__device__ __forceinline__ D2d operator-(D2d p, D2d q) { return D2d{p.v - q.v, p.a - q.a, p.b - q.b}; }
__device__ __forceinline__ D2d operator*(D2d p, D2d q)
{
    return D2d{p.v * q.v, p.a * q.v + p.v * q.a, p.b * q.v + p.v * q.b};
}
__device__ __forceinline__ D2d operator/(D2d p, D2d q)
{
    const double r = p.v / q.v;
    return D2d{r, (p.a - r * q.a) / q.v, (p.b - r * q.b) / q.v};
}
__device__ __forceinline__ D2d sqrt_d2(D2d p)
{
    const double r = sqrt(p.v);
    return D2d{r, p.a / (2.0 * r), p.b / (2.0 * r)};
}
__device__ __forceinline__ D2d cst_d2(double v) { return D2d{v, 0.0, 0.0}; }

__device__ void canonic_form_d(const float* Qf, double* C, double* Tp, double* Td)
{
    const double q1 = Qf[0], q2 = Qf[1], q3 = Qf[2], q4 = Qf[4], q5 = Qf[5], q6 = Qf[8];
    const double par1 = q1, par2 = 2 * q2, par3 = q4, par4 = 2 * q3, par5 = 2 * q5;
    const double th = 0.5 * atan2(par2, par1 - par3);
    const double ct = cos(th), st = sin(th);
    const double s2 = st * st, c2 = ct * ct, cs = st * ct;
    const double Au = par4 * ct + par5 * st, Av = -par4 * st + par5 * ct;
    const double Auu = par1 * c2 + par3 * s2 + par2 * cs, Avv = par1 * s2 + par3 * c2 - par2 * cs;
    const double tu = -Au / (2 * Auu), tv = -Av / (2 * Avv);
    const double uc = tu * ct - tv * st, vc = tu * st + tv * ct;
    const double t1 = ct * (ct * q1 + q2 * st) + st * (ct * q2 + q4 * st);
    const double t2 = ct * (ct * q2 + q4 * st) - st * (ct * q1 + q2 * st);
    const double t3 = ct * q3 + q5 * st + uc * (ct * q1 + q2 * st) + vc * (ct * q2 + q4 * st);
    const double t4 = ct * (ct * q4 - q2 * st) - st * (ct * q2 - q1 * st);
    const double t5 = ct * q5 - q3 * st + uc * (ct * q2 - q1 * st) + vc * (ct * q4 - q2 * st);
    const double t6 = q6 + uc * (q3 + q1 * uc + q2 * vc) + vc * (q5 + q2 * uc + q4 * vc) + q3 * uc + q5 * vc;
    const double c[9] = {t1, t2, t3, t2, t4, t5, t3, t5, t6};
    const double tp[9] = {ct, st, -ct * uc - st * vc, -st, ct, st * uc - ct * vc, 0, 0, ct * ct + st * st};
    const double td[9] = {ct, -st, uc, st, ct, vc, 0, 0, 1};
    for (int k = 0; k < 9; ++k) {
        C[k] = c[k];
        Tp[k] = tp[k];
        Td[k] = td[k];
    }
}

// homography_from_center in double, with d/d(x, y).
__device__ void homography_center_derivs_d(const double* C, const double* Tp, const double* Td, double x, double y,
                                           double* H, double* dHx, double* dHy)
{
    const D2d X{x, 1.0, 0.0}, Y{y, 0.0, 1.0};
    const D2d u = X * cst_d2(Tp[0]) + Y * cst_d2(Tp[1]) + cst_d2(Tp[2]);
    const D2d v = X * cst_d2(Tp[3]) + Y * cst_d2(Tp[4]) + cst_d2(Tp[5]);
    const D2d w = X * cst_d2(Tp[6]) + Y * cst_d2(Tp[7]) + cst_d2(Tp[8]);
    const D2d xc = u / w, yc = v / w;
    const D2d Q11 = cst_d2(C[0]), Q22 = cst_d2(C[4]), Q33 = cst_d2(C[8]), z = cst_d2(0.0);
    D2d h[9] = {Q33,          Q22 * xc * yc,           z - Q33 * xc,
                z,            z - Q11 * xc * xc - Q33, z - Q33 * yc,
                z - Q11 * xc, Q22 * yc,                z - Q33};
    const D2d d0 = sqrt_d2(Q22 * Q33 / Q11 * (Q11 * xc * xc + Q22 * yc * yc + Q33));
    const D2d d2 = sqrt_d2(z - Q22 * (Q11 * xc * xc + Q33));
    for (int i = 0; i < 3; ++i) {
        h[i * 3 + 0] = h[i * 3 + 0] * d0;
        h[i * 3 + 1] = h[i * 3 + 1] * Q33;
        h[i * 3 + 2] = h[i * 3 + 2] * d2;
    }
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const D2d r = h[j] * cst_d2(Td[i * 3]) + h[3 + j] * cst_d2(Td[i * 3 + 1]) + h[6 + j] * cst_d2(Td[i * 3 + 2]);
            H[i * 3 + j] = r.v;
            dHx[i * 3 + j] = r.a;
            dHy[i * 3 + j] = r.b;
        }
}

__device__ bool mat_inv_d(const double* a, double* r)
{
    const double c00 = a[4] * a[8] - a[5] * a[7];
    const double c01 = a[5] * a[6] - a[3] * a[8];
    const double c02 = a[3] * a[7] - a[4] * a[6];
    const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
    if (det == 0.0 || !isfinite(det)) return false;
    const double id = 1.0 / det;
    r[0] = c00 * id;
    r[1] = (a[2] * a[7] - a[1] * a[8]) * id;
    r[2] = (a[1] * a[5] - a[2] * a[4]) * id;
    r[3] = c01 * id;
    r[4] = (a[0] * a[8] - a[2] * a[6]) * id;
    r[5] = (a[2] * a[3] - a[0] * a[5]) * id;
    r[6] = c02 * id;
    r[7] = (a[1] * a[6] - a[0] * a[7]) * id;
    r[8] = (a[0] * a[4] - a[1] * a[3]) * id;
    return true;
}

__device__ __forceinline__ bool inside_d(const Roi& R, double x, double y)
{
    return x >= double(R.x0) && x < double(R.x1 - 1) && y >= double(R.y0) && y < double(R.y1 - 1);
}

// Identification.hpp:197-219 and its gradient, in double.
__device__ __forceinline__ double bilinear_d(const Roi& R, double x, double y, double& gx, double& gy)
{
    const int px = int(x), py = int(y);
    const uint8_t* p0 = R.img + px + size_t(py) * R.pitch;
    const double fx = x - double(px), fy = y - double(py);
    const double p1 = __ldg(p0), p2 = __ldg(p0 + 1), p3 = __ldg(p0 + R.pitch), p4 = __ldg(p0 + R.pitch + 1);
    gx = ((p2 - p1) * (1.0 - fy) + (p4 - p3) * fy) * 0.5;
    gy = ((p3 - p1) * (1.0 - fx) + (p4 - p2) * fx) * 0.5;
    return (p1 * (1.0 - fx) * (1.0 - fy) + p2 * fx * (1.0 - fy) + p3 * (1.0 - fx) * fy + p4 * fx * fy) * 0.5;
}

struct CostSharedD {
    double C[9], Tp[9], Td[9];
    double H[9], Hi[9], dH[2][9];
    double sig[kMaxCuts][kMaxSamples];
    double mean[kMaxSamples];
    double dz[kMaxCuts][3];
    double red[kThreads / 32][10];
    uint32_t oob;
    int bad;
};

}  // namespace

// k_cut_cost in double precision (one block per task).
__global__ void __launch_bounds__(kThreads) k_cut_cost_f64(const uint8_t* __restrict__ img, size_t pitch,
                                                           const IdentTask* __restrict__ tasks,
                                                           const float* __restrict__ centers, float* out,
                                                           IdentParams ip)
{
    __shared__ CostSharedD S;
    const IdentTask& T = tasks[blockIdx.x];
    const Roi roi = make_roi(img, pitch, T);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nS = ip.nSamples;
    const double bs = ip.beginSig;
    const double den = double(nS) - 1.0;
    float* o = out + 12 * size_t(blockIdx.x);
    const uint32_t cutMask = (T.ncuts >= 32) ? 0xffffffffu : ((1u << T.ncuts) - 1u);
    if (tid == 0) {
        canonic_form_d(T.Q, S.C, S.Tp, S.Td);
        homography_center_derivs_d(S.C, S.Tp, S.Td, centers[2 * blockIdx.x], centers[2 * blockIdx.x + 1], S.H,
                                   S.dH[0], S.dH[1]);
        S.bad = mat_inv_d(S.H, S.Hi) ? 0 : 1;
        S.oob = 0u;
    }
    if (tid < kMaxCuts * 3) S.dz[tid / 3][tid % 3] = 0.0;
    __syncthreads();
    if (S.bad) {
        if (tid == 0) write_cost(o, FLT_MAX);
        return;
    }
    for (int c = warp; c < T.ncuts; c += kWarps) {
        const double px = T.stop[c][0], py = T.stop[c][1];
        const double z0 = S.Hi[0] * px + S.Hi[1] * py + S.Hi[2];
        const double z1 = S.Hi[3] * px + S.Hi[4] * py + S.Hi[5];
        const double z2 = S.Hi[6] * px + S.Hi[7] * py + S.Hi[8];
        const double bx = z0 / z2, by = z1 / z2;
        const double xs = bx * bs, ys = by * bs;
        const double sx = (bx - xs) / den, sy = (by - ys) / den;
        bool bad = false;
        for (int k = lane; k < nS; k += 32) {
            const double x = xs + double(k) * sx, y = ys + double(k) * sy;
            const double u = S.H[0] * x + S.H[1] * y + S.H[2];
            const double v = S.H[3] * x + S.H[4] * y + S.H[5];
            const double w = S.H[6] * x + S.H[7] * y + S.H[8];
            const double qx = u / w, qy = v / w;
            double gx, gy;
            if (inside_d(roi, qx, qy)) S.sig[c][k] = bilinear_d(roi, qx, qy, gx, gy);
            else bad = true;
        }
        if (__ballot_sync(0xffffffffu, bad) && lane == 0) atomicOr(&S.oob, 1u << c);
    }
    __syncthreads();
    const uint32_t valid = ~S.oob & cutMask;
    const int n = __popc(valid);
    if (n < 2) {
        if (tid == 0) write_cost(o, FLT_MAX);
        return;
    }
    const double pairs = 0.5 * double(n) * double(n - 1);
    double costPart = 0.0;
    for (int k = tid; k < nS; k += kThreads) {
        double s1 = 0.0, s2 = 0.0;
        uint32_t m = valid;
        while (m) {
            const int c = __ffs(m) - 1;
            m &= m - 1;
            const double v = S.sig[c][k];
            s1 += v;
            s2 += v * v;
        }
        S.mean[k] = s1 / double(n);
        costPart += double(n) * s2 - s1 * s1;
    }
    __syncthreads();
    double gH[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double coef = 2.0 * double(n) / pairs;
    const double* Hm = S.H;
    for (int c = warp; c < T.ncuts; c += kWarps) {
        if (!((valid >> c) & 1u)) continue;
        const double px = T.stop[c][0], py = T.stop[c][1];
        const double z0 = S.Hi[0] * px + S.Hi[1] * py + S.Hi[2];
        const double z1 = S.Hi[3] * px + S.Hi[4] * py + S.Hi[5];
        const double z2 = S.Hi[6] * px + S.Hi[7] * py + S.Hi[8];
        const double bx = z0 / z2, by = z1 / z2;
        const double xs = bx * bs, ys = by * bs;
        const double sx = (bx - xs) / den, sy = (by - ys) / den;
        double gbx = 0.0, gby = 0.0;
        for (int k = lane; k < nS; k += 32) {
            const double x = xs + double(k) * sx, y = ys + double(k) * sy;
            const double u = Hm[0] * x + Hm[1] * y + Hm[2];
            const double v = Hm[3] * x + Hm[4] * y + Hm[5];
            const double w = Hm[6] * x + Hm[7] * y + Hm[8];
            const double rw = 1.0 / w;
            const double qx = u / w, qy = v / w;
            double gx, gy;
            (void)bilinear_d(roi, qx, qy, gx, gy);
            const double lam = coef * (S.sig[c][k] - S.mean[k]);
            const double fx = lam * gx, fy = lam * gy;
            const double fw = -(fx * qx + fy * qy);
            const double y3[3] = {x, y, 1.0};
            for (int j = 0; j < 3; ++j) {
                gH[j] += fx * rw * y3[j];
                gH[3 + j] += fy * rw * y3[j];
                gH[6 + j] += fw * rw * y3[j];
            }
            const double fX = (fx * (Hm[0] - qx * Hm[6]) + fy * (Hm[3] - qy * Hm[6])) * rw;
            const double fY = (fx * (Hm[1] - qx * Hm[7]) + fy * (Hm[4] - qy * Hm[7])) * rw;
            const double t = bs + double(k) * (1.0 - bs) / den;
            gbx += t * fX;
            gby += t * fY;
        }
        for (int off = 16; off; off >>= 1) {
            gbx += __shfl_xor_sync(0xffffffffu, gbx, off);
            gby += __shfl_xor_sync(0xffffffffu, gby, off);
        }
        if (lane == 0) {
            S.dz[c][0] = gbx / z2;
            S.dz[c][1] = gby / z2;
            S.dz[c][2] = -(gbx * bx + gby * by) / z2;
        }
    }
    double red[10];
    red[0] = costPart;
    for (int j = 0; j < 9; ++j) red[1 + j] = gH[j];
    for (int j = 0; j < 10; ++j)
        for (int off = 16; off; off >>= 1) red[j] += __shfl_xor_sync(0xffffffffu, red[j], off);
    if (lane == 0)
        for (int j = 0; j < 10; ++j) S.red[warp][j] = red[j];
    __syncthreads();
    if (tid == 0) {
        double cost = 0.0, G[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int w = 0; w < kWarps; ++w) {
            cost += S.red[w][0];
            for (int j = 0; j < 9; ++j) G[j] += S.red[w][1 + j];
        }
        cost /= pairs;
        double GHi[9] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int c = 0; c < T.ncuts; ++c) {
            const double p3[3] = {T.stop[c][0], T.stop[c][1], 1.0};
            for (int r = 0; r < 3; ++r)
                for (int q = 0; q < 3; ++q) GHi[r * 3 + q] += S.dz[c][r] * p3[q];
        }
        double M[9], Mt[9];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double a = 0.0;
                for (int q = 0; q < 3; ++q) a += GHi[i * 3 + q] * S.Hi[j * 3 + q];
                M[i * 3 + j] = a;
            }
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double a = 0.0;
                for (int q = 0; q < 3; ++q) a += S.Hi[q * 3 + i] * M[q * 3 + j];
                Mt[i * 3 + j] = a;
            }
        double dc[2] = {0.0, 0.0};
        for (int j = 0; j < 9; ++j) {
            G[j] -= Mt[j];
            dc[0] += G[j] * S.dH[0][j];
            dc[1] += G[j] * S.dH[1][j];
        }
        o[0] = float(cost);
        o[1] = float(dc[0]);
        o[2] = float(dc[1]);
        for (int j = 0; j < 9; ++j) o[3 + j] = float(G[j]);
    }
}

void upload_bank(const std::vector<std::vector<float>>& bank, float* d_bank_inv)
{
    std::vector<float> inv(size_t(kMaxBankIds) * kMaxBankRatios, 0.f);
    if (bank.empty() || bank.size() > size_t(kMaxBankIds) || bank[0].size() > size_t(kMaxBankRatios))
        throw Error{CCTAGB_BANK_ERROR, "bank larger than the identification kernel supports"};
    for (size_t i = 0; i < bank.size(); ++i)
        for (size_t r = 0; r < bank[i].size(); ++r) inv[i * kMaxBankRatios + r] = 1.f / bank[i][r];
    CCTAGB_CUDA(cudaMemcpy(d_bank_inv, inv.data(), inv.size() * sizeof(float), cudaMemcpyHostToDevice));
}

void launch_identify(const uint8_t* d_img, size_t pitch, const IdentTask* d_tasks, IdentResult* d_res, int n,
                     const IdentTask* tasks, int maxCuts, const float* d_bank_inv, const IdentParams& ip, cudaStream_t s)
{
    if (n <= 0) return;
    if (ip.gridN * ip.gridN > kMaxTrials || ip.gridN < 3 || (ip.gridN & 1) == 0)
        throw Error{CCTAGB_BAD_ARG, "imagedCenterNGridSample (gnCoarseGrid in Gauss-Newton) must be 3 or 5"};
    if (ip.nSamples > kMaxSamples || ip.nSamples < 32) throw Error{CCTAGB_BAD_ARG, "sampleCutLength out of range"};
    if (ip.refineMode != CCTAGB_REFINE_GRID && ip.refineMode != CCTAGB_REFINE_GAUSS_NEWTON)
        throw Error{CCTAGB_BAD_ARG, "unknown refineMode"};
    if (ip.refineMode == CCTAGB_REFINE_GAUSS_NEWTON && (ip.gnIterations < 1 || ip.gnIterations > 100))
        throw Error{CCTAGB_BAD_ARG, "gnIterations must be in [1, 100]"};
    if (ip.refineMode == CCTAGB_REFINE_GAUSS_NEWTON && (ip.coarseRounds < 1 || ip.coarseRounds > 64))
        throw Error{CCTAGB_BAD_ARG, "gnCoarseRounds must be in [1, 64]"};
    // Measured, against a block of 25 warps per marker (a cluster of 4 below 38
    // markers) that read the image and one trial per warp: 28 markers of a 1080p
    // frame 261 -> 120 us, 80 of a 3840x2160 clutter frame 588 -> 346 us, 1024
    // candidates of 8-150 px radius 3.15 -> 1.48 ms (1.95 ms in the caller's
    // order), by Gauss-Newton 4096 of them 2.61 -> 1.65 ms (4 to 6 blocks per SM,
    // with room for larger markers' pixels, 3 % slower).
    int dev = 0, sms = 0, smemBlock = 0, smemSm = 0;
    CCTAGB_CUDA(cudaGetDevice(&dev));
    CCTAGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    CCTAGB_CUDA(cudaDeviceGetAttribute(&smemBlock, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    CCTAGB_CUDA(cudaDeviceGetAttribute(&smemSm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    const bool gn = ip.refineMode == CCTAGB_REFINE_GAUSS_NEWTON;
    // Dynamic shared memory: the lines or the Gauss-Newton samples, then the
    // markers' pixels (1 KB per block is the driver's; markers without cuts, as
    // numCutsInIdentStep <= 0 leaves them, take none).
    const int cuts = std::min(std::max(maxCuts, 0), kMaxCuts);
    size_t work = grid_work(ip.gridN * ip.gridN, cuts);
    auto room = [&](int perSm) {
        const size_t all = std::min(size_t(smemBlock), size_t(smemSm) / size_t(perSm));
        return (all - align16(sizeof(Shared)) - work - 1024) & ~size_t(15);
    };
    struct {
        size_t largest = 0, some = 0;  // largest marker's pixels, of those that leave kIdentSpareL1
        int beyond = 0, half = 0;      // markers whose pixels exceed `one`, `two` bytes
    } px;
    auto look = [&](size_t one, size_t two) {
        for (int i = 0; i < n; ++i) {
            const size_t b = align16(size_t(ident_box(tasks[i].a, tasks[i].b, tasks[i].angle)));
            px.largest = std::max(px.largest, b);
            if (b + kIdentSpareL1 <= one) px.some = std::max(px.some, b);
            px.beyond += b > one ? 1 : 0;
            px.half += b > two ? 1 : 0;
        }
    };
    IdentLaunch a{n, sms, ip.gridN * ip.gridN, ip.nSamples, gn, ip.layout == CCTAGB_IDENT_BLOCK, 0, 0};
    if (!gn) {
        look(room(1), room(2));
        a.beyond = px.beyond;
        a.beyondHalf = px.half;
    }
    IdentLayout l = ident_layout(a);
    const int cluster = l.cluster, perSm = l.perSm, warps = l.warps;
    if (gn) {
        if (warps > kMaxChunks)
            work = std::max({work, kGnWork,
                             cluster == 1 && perSm == 1 ? align16(3 * sizeof(float) * size_t(cuts * ip.nSamples)) : 0});
        look(room(perSm), room(perSm));
        // reads take less of a marker's time than in the grid: room is kept while a
        // third of the markers use it (4096 of 8-200 px, 68 % beyond: 2.00 ms with,
        // 1.94 without; 400 of 8-150 px, 52 % beyond: 322 and 333 us), but a launch
        // of one wave lasts as long as its largest marker (92 of 200 and 400 px 217
        // and 193 us)
        if (3LL * px.beyond > 2LL * n || (px.beyond && cluster == 1 && n <= sms)) l.pixels = IdentPixels::kNone;
    }
    const size_t box = l.pixels == IdentPixels::kNone   ? 0
                       : l.pixels == IdentPixels::kSome ? px.some
                                                        : std::min(px.largest, room(perSm));
    const size_t smem = std::max(work + box, sizeof(FinalWork));
    auto* kernel = cluster > 1                 ? k_identify<true, false>
                   : warps == kIdentTrialWarps ? k_identify<false, true>
                                               : k_identify<false, false>;
    CCTAGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     smemBlock - int(align16(sizeof(Shared)))));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(n * cluster));
    cfg.blockDim = dim3(unsigned(32 * warps));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(cluster);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    CCTAGB_CUDA(cudaLaunchKernelEx(&cfg, kernel, d_img, pitch, d_tasks, d_res, d_bank_inv, ip, int(work), int(box)));
}

int ident_box(float a, float b, float angle)
{
    // half extents of the ellipse, and room for the margin of find_box and the
    // rows' padding
    const float c = std::cos(angle), s = std::sin(angle);
    const float hx = std::sqrt(a * a * c * c + b * b * s * s), hy = std::sqrt(a * a * s * s + b * b * c * c);
    const double w = 2.0 * hx + 20.0, h = 2.0 * hy + 10.0;
    return w * h < double(1 << 20) ? int(w * h) : 1 << 20;  // also for NaN: as much as there is
}

void launch_cut_cost(const uint8_t* d_img, size_t pitch, const IdentTask* d_tasks, const float* d_centers,
                     float* d_out, int n, int maxCuts, const IdentParams& ip, cudaStream_t s, bool fp64)
{
    if (n <= 0) return;
    if (ip.nSamples > kMaxSamples || ip.nSamples < 32) throw Error{CCTAGB_BAD_ARG, "sampleCutLength out of range"};
    if (fp64) {
        k_cut_cost_f64<<<n, kThreads, 0, s>>>(d_img, pitch, d_tasks, d_centers, d_out, ip);
    } else {
        // A block per SM has no other's samples to hide its serial steps behind: a
        // warp per cut then.  Measured per call, 25 warps against 4: 50 against 61 us
        // for one task, 68 against 73 for 148, 82 either way for 222, 106 against 96
        // for 444, 640 against 428 for 4096.
        int dev = 0, sms = 0;
        CCTAGB_CUDA(cudaGetDevice(&dev));
        CCTAGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        const int cap = std::min(std::max(maxCuts, 1), kMaxCuts) * ip.nSamples;
        const size_t smem = 3 * sizeof(float) * size_t(cap);
        auto launch = [&](auto* kernel, int threads) {
            CCTAGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(3 * sizeof(float) * kMaxCuts * kMaxSamples)));
            kernel<<<n, threads, smem, s>>>(d_img, pitch, d_tasks, d_centers, d_out, ip, cap);
        };
        if (n <= sms) launch(k_cut_cost<kWarps>, kThreads);
        else launch(k_cut_cost<kCostWarps>, 32 * kCostWarps);
    }
    CCTAGB_CUDA(cudaGetLastError());
}

}  // namespace cctagb
