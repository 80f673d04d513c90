// Image stage of the CCTag hot path on sm_100a: pyramid, 9x9 DoG derivatives,
// Canny NMS + hysteresis, thinning, raster-order edge compaction, Bresenham
// gradient walk, vote, voter lists and seeds.  Every launch covers all pyramid
// levels at once (the block index is split into level and tile), no launch
// needs a host synchronisation, so a frame is one capturable launch sequence.
//
// Bit-exactness with the reference CPU path (file:line in the CCTag project):
//  * derivatives: same 72-tap FMA chain as cv::filter2D, cvRecode.cpp:74-92
//  * magnitude / NMS / hysteresis: cvRecode.cpp:174-409 (final edge set is the
//    8-connected components of NMS candidates that hold a strong pixel)
//  * thinning: thinning.cpp:12-51 (Lam-Lee-Suen tables, temp border = 0)
//  * edge order: raster order, Canny.cpp:15-31
//  * walk: Bresenham.cpp:18-209, vote: Vote.cpp:58-247 (no FMA contraction,
//    IEEE division and square root, same accumulation order)
#include <algorithm>
#include <cstdint>

#include "common.hpp"
#include "cctag_b200/portable/pmath.hpp"

namespace cctagb {

// kerneldX of cvRecode.cpp:74-83
__constant__ float cK[9][9] = {
    {-0.000000143284235f, -0.000003558691641f, -0.000028902492951f, -0.000064765993382f, 0.f, 0.000064765993382f, 0.000028902492951f, 0.000003558691641f, 0.000000143284235f},
    {-0.000004744922188f, -0.000117847682078f, -0.000957119116802f, -0.002144755142391f, 0.f, 0.002144755142391f, 0.000957119116802f, 0.000117847682078f, 0.000004744922188f},
    {-0.000057804985902f, -0.001435678675203f, -0.011660097860113f, -0.026128466569370f, 0.f, 0.026128466569370f, 0.011660097860113f, 0.001435678675203f, 0.000057804985902f},
    {-0.000259063973527f, -0.006434265427174f, -0.052256933138740f, -0.117099663048638f, 0.f, 0.117099663048638f, 0.052256933138740f, 0.006434265427174f, 0.000259063973527f},
    {-0.000427124283626f, -0.010608310271112f, -0.086157117207395f, -0.193064705260108f, 0.f, 0.193064705260108f, 0.086157117207395f, 0.010608310271112f, 0.000427124283626f},
    {-0.000259063973527f, -0.006434265427174f, -0.052256933138740f, -0.117099663048638f, 0.f, 0.117099663048638f, 0.052256933138740f, 0.006434265427174f, 0.000259063973527f},
    {-0.000057804985902f, -0.001435678675203f, -0.011660097860113f, -0.026128466569370f, 0.f, 0.026128466569370f, 0.011660097860113f, 0.001435678675203f, 0.000057804985902f},
    {-0.000004744922188f, -0.000117847682078f, -0.000957119116802f, -0.002144755142391f, 0.f, 0.002144755142391f, 0.000957119116802f, 0.000117847682078f, 0.000004744922188f},
    {-0.000000143284235f, -0.000003558691641f, -0.000028902492951f, -0.000064765993382f, 0.f, 0.000064765993382f, 0.000028902492951f, 0.000003558691641f, 0.000000143284235f}};

// Lam-Lee-Suen sub-iteration tables as bitsets (index = the 3x3 neighbourhood
// with the weights of thinning.cpp: (x-1,y-1)=1 ... (x+1,y+1)=256): bit set
// where the pixel stays.  Derived from the thinning conditions at compile time.
struct ThinTables {
    uint32_t bits[2][16];
};
constexpr ThinTables make_thin_tables()
{
    ThinTables t{};
    for (int pass = 1; pass <= 2; ++pass)
        for (int idx = 0; idx < 512; ++idx) {
            if (!(idx & 16)) continue;
            int x[10] = {0, (idx & 128) ? 1 : 0, (idx & 64) ? 1 : 0, (idx & 8) ? 1 : 0, (idx & 1) ? 1 : 0,
                         (idx & 2) ? 1 : 0, (idx & 4) ? 1 : 0, (idx & 32) ? 1 : 0, (idx & 256) ? 1 : 0, 0};
            x[9] = x[1];
            int xh = 0, n1 = 0, n2 = 0;
            for (int i = 1; i <= 4; ++i) {
                xh += (x[2 * i - 1] == 0 && (x[2 * i] == 1 || x[2 * i + 1] == 1)) ? 1 : 0;
                n1 += x[2 * i - 1] | x[2 * i];
                n2 += x[2 * i] | x[2 * i + 1];
            }
            const int mn = n1 < n2 ? n1 : n2;
            const bool g1 = xh == 1, g2 = mn >= 2 && mn <= 3;
            const bool g3 = pass == 1 ? (((x[2] | x[3] | (1 - x[8])) & x[1]) == 0)
                                      : (((x[6] | x[7] | (1 - x[4])) & x[5]) == 0);
            if (!(g1 && g2 && g3)) t.bits[pass - 1][idx >> 5] |= 1u << (idx & 31);
        }
    return t;
}
__constant__ ThinTables cThinTab = make_thin_tables();

// ------------------------------------------------------------------ utils --
__device__ __forceinline__ int level_of_block(const Levels& lv, int b, int LevelView::*tiles, int& local)
{
    int l = 0;
    while (l < lv.n - 1 && b >= lv.l[l].*tiles) {
        b -= lv.l[l].*tiles;
        ++l;
    }
    local = b;
    return l;
}

__device__ __forceinline__ int16_t sat_round16(float s)
{
    float r = rintf(s);
    r = fminf(32767.f, fmaxf(-32768.f, r));
    return int16_t(r);
}

// Gradient magnitude, rintf(sqrtf(dx^2 + dy^2)) as cvRecode.cpp:200-211.
__device__ __forceinline__ int magnitude(int16_t gx, int16_t gy)
{
    const float fx = float(gx), fy = float(gy);
    return int(rintf(__fsqrt_rn(__fadd_rn(__fmul_rn(fx, fx), __fmul_rn(fy, fy)))));
}

// ---------------------------------------------------------------- pyramid --
// ImagePyramid.cpp:23-52, Level.cpp:57-81.  Exact 2x reductions (every level
// of a frame whose sides are multiples of 8) are the rounded 2x2 mean, as
// cv::resize's area fast path; one thread builds an 8x8 block of level 0 into
// levels 1..3.
__global__ void k_pyramid3(Levels lv)
{
    const int base = blockIdx.z * (lv.n / lv.frames);  // this frame's level 0
    const LevelView& L0 = lv.l[base];
    const int W3 = L0.W >> 3, H3 = L0.H >> 3;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W3 || y >= H3) return;
    uint32_t p[8][8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint2 v = *reinterpret_cast<const uint2*>(L0.src + size_t(8 * y + r) * L0.W + 8 * x);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            p[r][c] = (v.x >> (8 * c)) & 0xff;
            p[r][c + 4] = (v.y >> (8 * c)) & 0xff;
        }
    }
    uint32_t q1[4][4], q2[2][2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c)
            q1[r][c] = (p[2 * r][2 * c] + p[2 * r][2 * c + 1] + p[2 * r + 1][2 * c] + p[2 * r + 1][2 * c + 1] + 2) >> 2;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c)
            q2[r][c] = (q1[2 * r][2 * c] + q1[2 * r][2 * c + 1] + q1[2 * r + 1][2 * c] + q1[2 * r + 1][2 * c + 1] + 2) >> 2;
    const uint32_t q3 = (q2[0][0] + q2[0][1] + q2[1][0] + q2[1][1] + 2) >> 2;
    const LevelView& L1 = lv.l[base + 1];
    const LevelView& L2 = lv.l[base + 2];
    const LevelView& L3 = lv.l[base + 3];
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<uint32_t*>(L1.src + size_t(4 * y + r) * L1.W + 4 * x) =
            q1[r][0] | (q1[r][1] << 8) | (q1[r][2] << 16) | (q1[r][3] << 24);
#pragma unroll
    for (int r = 0; r < 2; ++r)
        *reinterpret_cast<uint16_t*>(L2.src + size_t(2 * y + r) * L2.W + 2 * x) = uint16_t(q2[r][0] | (q2[r][1] << 8));
    L3.src[size_t(y) * L3.W + x] = uint8_t(q3);
}

// One level from the previous one, any size: exact 2x -> 2x2 rounded mean,
// otherwise cv::resize INTER_LINEAR fixed point (11-bit coefficients and the
// vectorised vertical pass of OpenCV: 16-bit high products, rounding shift 2).
__device__ __forceinline__ void resize_coef(int d, int dn, int sn, int& s, int& c0)
{
    const double scale = double(sn) / dn;
    float f = float((d + 0.5) * scale - 0.5);
    s = int(floorf(f));
    f -= float(s);
    if (s < 0) { f = 0.f; s = 0; }
    if (s >= sn - 1) { f = 0.f; s = sn - 1; }
    c0 = int(rintf(__fmul_rn(1.f - f, 2048.f)));
}

__global__ void k_resize_level(const uint8_t* __restrict__ src, int sw, int sh, uint8_t* __restrict__ dst, int dw, int dh)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    if (sw == 2 * dw && sh == 2 * dh) {
        const uint8_t* p = src + size_t(2 * y) * sw + 2 * x;
        dst[size_t(y) * dw + x] = uint8_t((p[0] + p[1] + p[sw] + p[sw + 1] + 2) >> 2);
        return;
    }
    int sx, cx0, sy, cy0;
    resize_coef(x, dw, sw, sx, cx0);
    resize_coef(y, dh, sh, sy, cy0);
    const int cx1 = 2048 - cx0, cy1 = 2048 - cy0;
    const int sx1 = min(sx + 1, sw - 1), sy1 = min(sy + 1, sh - 1);
    const int r0 = src[size_t(sy) * sw + sx] * cx0 + src[size_t(sy) * sw + sx1] * cx1;
    const int r1 = src[size_t(sy1) * sw + sx] * cx0 + src[size_t(sy1) * sw + sx1] * cx1;
    int v = ((((r0 >> 4) * cy0) >> 16) + (((r1 >> 4) * cy1) >> 16) + 2) >> 2;
    dst[size_t(y) * dw + x] = uint8_t(min(255, max(0, v)));
}

// ------------------------------------------------------------- derivatives --
// dx and dy of every level: cv::filter2D's FP32 sums over the 72 nonzero taps in
// row-major order, rounded to int16.  The kernel is the outer product of a
// smoothing column G (G[4] = 1) and an antisymmetric row D, up to the last
// digits of its printed constants, so the sums are first formed separably, with
// exact integer sums and differences of the symmetric taps, 35 operations a
// pixel instead of 144.  That value and the reference's chain differ by less
// than kDerivErr, so where it is further than that from a rounding boundary
// both round to the same integer; the other pixels (0.3 % on noisy frames) are
// listed and their chains evaluated as written.
//
// kDerivErr, for pixels in [0, 255] and with u = 2^-24: a rounding adds at most
// u times its result.  The chain's partial sums (bounded by 255 times the larger
// of their positive and negative weights) add up to 4.1e-4 for dx and 4.9e-4 for
// dy; the separable form's row sums, bounded by 74 and 639, and their weighted
// sums by 186, to 1.1e-4 and 1.7e-4; the factors' products differ from the
// constants by 2.2e-6 in all.
//
// A warp takes 64 columns (two per lane) and kDvRows rows, walking down with the
// last nine row sums in registers; products and sums of the two columns go in
// pairs (fma.rn.f32x2).  Four columns per lane need fewer loads but 138
// registers: 10 warps on an SM, which left it waiting for the tile's loads
// (3840x2160 frame and its pyramid: 88 us; two columns 52 us; the chains for
// every pixel, with the suppression in the same kernel, 145 us).
constexpr float kDerivErr = 7.5e-4f;
constexpr int kDvCols = 64, kDvWarps = 4, kDvRows = 16;
constexpr int kDvTileRows = kDvWarps * kDvRows;
constexpr int kDvPitch = kDvCols + 8;
constexpr int kDvList = 512;  // unsure pixels listed per tile; above that the whole tile is redone

using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pair2(float lo, float hi)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void split2(f32x2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// The reference's chains for the pixel whose 9x9 window starts at s.
__device__ __noinline__ void deriv_chain(const float* s, float& ax, float& ay)
{
    ax = ay = 0.f;
#pragma unroll 1
    for (int i = 0; i < 9; ++i)
#pragma unroll
        for (int j = 0; j < 9; ++j) {
            const float v = s[i * kDvPitch + j];
            if (j != 4) ax = __fmaf_rn(cK[i][j], v, ax);
            if (i != 4) ay = __fmaf_rn(cK[j][i], v, ay);
        }
}

__global__ void __launch_bounds__(32 * kDvWarps) k_derivs(Levels lv)
{
    __shared__ __align__(16) float s_src[kDvTileRows + 8][kDvPitch];
    __shared__ uint16_t s_list[kDvList];
    __shared__ int s_unsure;
    int tile;
    const int l = level_of_block(lv, blockIdx.x, &LevelView::dv_tiles, tile);
    const LevelView& L = lv.l[l];
    const int W = L.W, H = L.H;
    const int x0 = (tile % L.dv_tx) * kDvCols, y0 = (tile / L.dv_tx) * kDvTileRows;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_unsure = 0;
    if (blockIdx.x == 0)  // the counters of the launch's levels start at 0
        for (int i = t; i < lv.n * int(sizeof(LevelCounters) / 4); i += 32 * kDvWarps)
            reinterpret_cast<int32_t*>(lv.cnt)[i] = 0;
    // the tile with its halo of 4, the image's border pixels repeated; inside
    // the image and on word boundaries a word at a time, several in flight
    constexpr int kWords = kDvPitch / 4, kStage = (kDvTileRows + 8) * kWords;
    auto put = [&](int i, uint32_t v) {
        const int r = i / kWords, q = i - r * kWords;
        *reinterpret_cast<float4*>(&s_src[r][4 * q]) =
            make_float4(float(v & 0xffu), float((v >> 8) & 0xffu), float((v >> 16) & 0xffu), float(v >> 24));
    };
    auto row_of = [&](int i) { return L.src + size_t(min(H - 1, max(0, y0 - 4 + i / kWords))) * W; };
    if (x0 >= 4 && x0 + kDvCols + 4 <= W && W % 4 == 0 && (reinterpret_cast<size_t>(L.src) & 3) == 0) {
        constexpr int kAhead = 6;
        for (int i0 = t; i0 < kStage; i0 += kAhead * 32 * kDvWarps) {
            uint32_t v[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                const int i = i0 + k * 32 * kDvWarps;
                if (i < kStage)
                    v[k] = __ldg(reinterpret_cast<const uint32_t*>(row_of(i) + x0 - 4 + 4 * (i % kWords)));
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (i0 + k * 32 * kDvWarps < kStage) put(i0 + k * 32 * kDvWarps, v[k]);
        }
    } else {
        constexpr int kAhead = 3;
        for (int i0 = t; i0 < kStage; i0 += kAhead * 32 * kDvWarps) {
            uint32_t v[kAhead][4];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                const int i = min(i0 + k * 32 * kDvWarps, kStage - 1);
                const uint8_t* row = row_of(i);
                const int x = x0 - 4 + 4 * (i % kWords);
#pragma unroll
                for (int q = 0; q < 4; ++q) v[k][q] = __ldg(row + min(W - 1, max(0, x + q)));
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k)
                if (i0 + k * 32 * kDvWarps < kStage)
                    put(i0 + k * 32 * kDvWarps, v[k][0] | v[k][1] << 8 | v[k][2] << 16 | v[k][3] << 24);
        }
    }
    __syncthreads();
    // D[8 - j] and G[j], j = 0..3 (cK's center row, and its columns over it)
    const float D[4] = {0.000427124283626f, 0.010608310271112f, 0.086157117207395f, 0.193064705260108f};
    const float G[4] = {0.000335462624f, 0.0111089963f, 0.135335281f, 0.606530666f};
    f32x2 D2[4], G2[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        D2[j] = pair2(D[j], D[j]);
        G2[j] = pair2(G[j], G[j]);
    }
    const f32x2 magic = pair2(12582912.f, 12582912.f), nmagic = pair2(-12582912.f, -12582912.f);
    const f32x2 minus1 = pair2(-1.f, -1.f);
    f32x2 wd[9], wg[9];  // the last nine rows' sums (slot = row mod 9)
    const int yw = y0 + warp * kDvRows;
    const int rows = min(kDvRows, H - yw) + 8;
    // four-byte stores where the rows (and the caller's planes) allow them
    const bool wide = W % 2 == 0 && ((reinterpret_cast<size_t>(L.dx) | reinterpret_cast<size_t>(L.dy)) & 3) == 0;
    const int xq = x0 + 2 * lane;
    for (int r9 = 0; r9 < rows; r9 += 9) {
#pragma unroll
        for (int u = 0; u < 9; ++u) {
            const int r = r9 + u;
            if (r >= rows) break;
            const float2* p = reinterpret_cast<const float2*>(&s_src[warp * kDvRows + r][2 * lane]);
            float v[10];
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const float2 q = p[j];
                v[2 * j] = q.x;
                v[2 * j + 1] = q.y;
            }
            f32x2 d = 0, g = pair2(v[4], v[5]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const f32x2 df = pair2(v[8 - j] - v[j], v[9 - j] - v[1 + j]);
                const f32x2 sm = pair2(v[8 - j] + v[j], v[9 - j] + v[1 + j]);
                d = j == 0 ? mul2(D2[0], df) : fma2(D2[j], df, d);
                g = fma2(G2[j], sm, g);
            }
            wd[u] = d;
            wg[u] = g;
            if (r < 8) continue;
            // output row r - 8: slots u + 1 .. u + 9 (mod 9) hold its nine rows
            f32x2 x = wd[(u + 5) % 9], y = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int a = (u + 1 + j) % 9, b = (u + 9 - j) % 9;
                x = fma2(G2[j], add2(wd[a], wd[b]), x);
                const f32x2 df = fma2(minus1, wg[a], wg[b]);
                y = j == 0 ? mul2(D2[0], df) : fma2(D2[j], df, y);
            }
            // rounded to the nearest integer (in the low bits of the sum with
            // 1.5 * 2^23), and the distance to it
            const f32x2 mx = add2(x, magic), my = add2(y, magic);
            const f32x2 ex = fma2(minus1, add2(mx, nmagic), x), ey = fma2(minus1, add2(my, nmagic), y);
            const uint32_t ox = __byte_perm(uint32_t(mx), uint32_t(mx >> 32), 0x5410);
            const uint32_t oy = __byte_perm(uint32_t(my), uint32_t(my >> 32), 0x5410);
            float a0, a1, b0, b1;
            split2(ex, a0, a1);
            split2(ey, b0, b1);
            const int yo = yw + r - 8;
            const size_t o = size_t(yo) * W + xq;
            if (wide) {
                if (xq < W) {
                    *reinterpret_cast<uint32_t*>(L.dx + o) = ox;
                    *reinterpret_cast<uint32_t*>(L.dy + o) = oy;
                }
            } else {
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (xq + k < W) {
                        L.dx[o + k] = int16_t(ox >> (16 * k));
                        L.dy[o + k] = int16_t(oy >> (16 * k));
                    }
            }
            const float w0 = fmaxf(fabsf(a0), fabsf(b0)), w1 = fmaxf(fabsf(a1), fabsf(b1));
            if (fmaxf(w0, w1) > 0.5f - kDerivErr) {
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if ((k ? w1 : w0) > 0.5f - kDerivErr && xq + k < W) {
                        const int i = atomicAdd(&s_unsure, 1);
                        if (i < kDvList) s_list[i] = uint16_t((yo - y0) * kDvCols + 2 * lane + k);
                    }
            }
        }
    }
    __syncthreads();  // and the stores above come before those below
    const bool all = s_unsure > kDvList;
    const int n = all ? kDvTileRows * kDvCols : s_unsure;
    for (int i = t; i < n; i += 32 * kDvWarps) {
        const int p = all ? i : s_list[i];
        const int r = p / kDvCols, c = p % kDvCols;
        if (x0 + c >= W || y0 + r >= H) continue;
        float ax, ay;
        deriv_chain(&s_src[r][c], ax, ay);
        const size_t o = size_t(y0 + r) * W + x0 + c;
        L.dx[o] = sat_round16(ax);
        L.dy[o] = sat_round16(ay);
    }
}

// ------------------------------------------------------------- hysteresis --
// The reference's stack hysteresis (cvRecode.cpp:362-394) keeps exactly the
// 8-connected components of NMS candidates that contain a strong pixel.  Here
// the image is cut into 32x32 tiles, one warp each, lane r holding row r of
// the tile as 32-bit masks (candidates C, strong S):
//  1. k_nms_tiles: non-maximum suppression (C, S), the closure R of S within C
//     inside the tile, and the other components of C that touch the tile border,
//     labelled per border position;
//  2. k_hyst_unions / k_hyst_roots: those weak border components joined across
//     tile borders by a lock-free union-find over (tile, component) ids
//     (parent <= self, roots linked by atomicMin, so any schedule gives the
//     same sets) or marked where they meet a pixel of R, and each set with a
//     marked member marked strong at its root;
//  3. k_hyst_final: per tile, R plus the border pixels of strong sets, closed
//     within C again: the hysteresis result H, one bit per pixel.
// A pixel is in H exactly when its component holds a strong pixel: a path to
// one either stays in the tile (step 1) or leaves it through a border pixel
// of its tile component, whose set is then strong (steps 2-3).
constexpr int kUfCap = 1 << 22;
constexpr int kTile = 32;          // hysteresis tile side
constexpr int kBorderPos = 128;    // border positions of a tile (4 x 32, some unused)
constexpr int kTileComps = 64;     // border components per tile (at most 62: runs on a 124-pixel cycle)

__device__ __forceinline__ int uf_find(const int32_t* L, int p)
{
    int q = *(volatile const int32_t*)&L[p];
    int guard = 0;
    while (q != p && guard++ < kUfCap) {
        p = q;
        q = *(volatile const int32_t*)&L[p];
    }
    return p;
}

__device__ __forceinline__ void uf_union(int32_t* L, int a, int b, int32_t* err)
{
    for (int it = 0; it < kUfCap; ++it) {
        // both walks to the roots side by side
        int pa = *(volatile const int32_t*)&L[a], pb = *(volatile const int32_t*)&L[b];
        for (int guard = 0; (pa != a || pb != b) && guard < kUfCap; ++guard) {
            a = pa;
            b = pb;
            pa = *(volatile const int32_t*)&L[a];
            pb = *(volatile const int32_t*)&L[b];
        }
        if (a == b) return;
        if (a > b) { const int tmp = a; a = b; b = tmp; }
        const int old = atomicMin(&L[b], a);
        if (old == b) return;
        b = old;
    }
    atomicOr(err, kErrUnionFind);
}

// The closure of `seed` (a subset of c) within c, 8-connected, over the
// warp's tile (lane = row).  A round takes the neighbour rows' pixels and goes
// on along the row's runs: upwards to their ends (adding pixels of a run to it
// carries through it), downwards seven pixels (c2: pixels whose lower neighbour
// is one too, c4: whose three lower neighbours are).  Each round adds a pixel or
// ends the loop, so it ends within the tile's 1024 pixels.
__device__ __forceinline__ uint32_t tile_closure(uint32_t seed, uint32_t c, int lane)
{
    const uint32_t c2 = c & (c >> 1), c4 = c2 & (c2 >> 2);
    uint32_t r = seed & c;
    for (int it = 0; it <= kTile * kTile; ++it) {
        uint32_t up = __shfl_up_sync(0xffffffffu, r, 1);
        uint32_t dn = __shfl_down_sync(0xffffffffu, r, 1);
        if (lane == 0) up = 0u;
        if (lane == kTile - 1) dn = 0u;
        const uint32_t v = r | up | dn;
        uint32_t nb = (v | (v << 1) | (v >> 1)) & c;
        nb |= ((nb + c) ^ c) & c;
        nb |= c2 & (nb >> 2);
        nb |= c4 & (nb >> 4);
        if (!__any_sync(0xffffffffu, nb != r)) break;
        r = nb;
    }
    return r;
}

// Border position of tile pixel (x, y) (tile coordinates), -1 inside:
// row 0 -> x, row 31 -> 32 + x, column 0 -> 64 + y, column 31 -> 96 + y.
__device__ __forceinline__ int border_pos(int x, int y)
{
    if (y == 0) return x;
    if (y == kTile - 1) return kTile + x;
    if (x == 0) return 2 * kTile + y;
    if (x == kTile - 1) return 3 * kTile + y;
    return -1;
}

// Warp w of the launch: its level and tile (tiles of all levels back to back).
__device__ __forceinline__ int level_of_tile(const Levels& lv, int g, int& tile)
{
    int l = 0;
    while (l < lv.n - 1 && g >= lv.l[l].uf_tiles) {
        g -= lv.l[l].uf_tiles;
        ++l;
    }
    tile = g;
    return l;
}

__device__ __forceinline__ uint32_t* plane_c(const LevelView& L) { return L.hbits; }
__device__ __forceinline__ uint32_t* plane_r(const LevelView& L) { return L.hbits + size_t(L.WW) * L.H; }
__device__ __forceinline__ uint32_t* plane_h(const LevelView& L) { return L.hbits + 2 * size_t(L.WW) * L.H; }

constexpr int kHystWarps = 4;

// Magnitude and direction of a pixel as the suppression reads them.  GIVEN:
// derivatives of any size (the caller's), in the reference's own arithmetic;
// else those of k_derivs, whose magnitude is below 263: their squares' sum is
// exact and its root is never near a half, so the approximate root rounds to
// the same integer, and the direction tests are exact in floats.
template <bool GIVEN>
struct Gradient {
    float m;     // magnitude, an integer
    int sector;  // 0 horizontal, 1 vertical, 2 and 3 the diagonals (signs equal, different)
};
template <bool GIVEN>
__device__ __forceinline__ Gradient<GIVEN> gradient_of(int gx, int gy)
{
    Gradient<GIVEN> g;
    const int diag = (gx ^ gy) < 0 ? 3 : 2;
    if (GIVEN) {
        g.m = float(magnitude(int16_t(gx), int16_t(gy)));
        const int TG22 = int(0.4142135623730950488016887242097 * (1 << 15) + 0.5);
        const unsigned ax = unsigned(abs(gx)), ay = unsigned(abs(gy));
        const int tg22x = int(ax * unsigned(TG22));
        const int tg67x = int(unsigned(tg22x) + ((ax + ax) << 15));
        const int gy15 = int(ay << 15);
        g.sector = gy15 < tg22x ? 0 : gy15 > tg67x ? 1 : diag;
    } else {
        // small integers to floats through the bits of 1.5 * 2^23 + n
        const float fx = fabsf(__fsub_rn(__int_as_float(0x4B400000 + gx), 12582912.f));
        const float fy = fabsf(__fsub_rn(__int_as_float(0x4B400000 + gy), 12582912.f));
        float r;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__fmaf_rn(fx, fx, __fmul_rn(fy, fy))));
        g.m = __fsub_rn(__fadd_rn(r, 12582912.f), 12582912.f);
        // TG22 = 13573 = tan(22.5 deg) * 2^15; tan(67.5 deg) = tan(22.5 deg) + 2
        const float y15 = __fmul_rn(fy, 32768.f);
        g.sector = y15 < __fmul_rn(fx, 13573.f) ? 0 : y15 > __fmul_rn(fx, 13573.f + 65536.f) ? 1 : diag;
    }
    return g;
}

// Non-maximum suppression (cvRecode.cpp:258-323) and step 1 of the hysteresis,
// a block of WARPS warps per tile: each suppresses its rows (lane = column),
// then all hold the tile's masks (lane = row).  The pixels of R need no
// component: what they touch across the border is strong.  So only the weak
// components that touch the border are flooded, one by one, in rounds that fill
// runs of a row, each warp from its sides of the tile; a component's label is
// its first border position, the same from every side, numbered at the end.
// A tile is one long chain of instructions: with few tiles four warps shorten
// it, with many one warp takes fewer instructions in all.  Measured, one warp
// and four (suppression included): 640x480 21 and 10 us, 1080p and its pyramid
// (2,725 tiles) 33 and 31 us, 3840x2160 clutter 85 and 98 us, sixteen 1080p
// frames 315 and 432 us.  With a flood per border component, strong ones too, a
// pixel per round, the hysteresis alone took 22 us of the small frame, 26 of the
// 1080p frame; a union-find over the runs of the tile 35 us and 58 us.
constexpr int kNmsFewTiles = 148 * 20;

template <bool GIVEN, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) k_nms_tiles(Levels lv, VoteParamsDev vp)
{
    constexpr int kRows = kTile / WARPS;             // of a warp
    constexpr int kGroup = WARPS == 4 ? kRows + 2 : 8;  // rows whose loads are in flight together
    static_assert(WARPS == 4 || WARPS == 1, "sides of the tile per warp");
    __shared__ float s_side[WARPS][2][kRows + 2];  // magnitudes left and right of the tile
    __shared__ uint32_t s_c[kTile], s_st[kTile];
    __shared__ uint8_t s_lab[kBorderPos], s_rank[kBorderPos];
    const unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int tile;
    const int l = level_of_block(lv, blockIdx.x, &LevelView::uf_tiles, tile);
    const LevelView& L = lv.l[l];
    const int W = L.W, H = L.H;
    const int tx = tile % L.uf_tx, ty = tile / L.uf_tx;
    const int x0 = tx * kTile, y0 = ty * kTile;
    const int rows = min(kTile, H - y0), cols = min(kTile, W - x0);
    const int yw = y0 + warp * kRows - 1;  // the first of the warp's rows, with one above and below
    for (int i = lane; i < 2 * (kRows + 2); i += 32) {
        const int side = i >= kRows + 2 ? 1 : 0, r = i - side * (kRows + 2);
        const int x = side ? x0 + kTile : x0 - 1;
        float m = 0.f;
        if (unsigned(yw + r) < unsigned(H) && unsigned(x) < unsigned(W)) {
            const size_t p = size_t(yw + r) * W + x;
            m = gradient_of<GIVEN>(L.dx[p], L.dy[p]).m;
        }
        s_side[warp][side][r] = m;
    }
    for (int i = threadIdx.x; i < kBorderPos; i += 32 * WARPS) s_lab[i] = 0xff;
    __syncwarp();
    float ul = 0.f, uc = 0.f, ur = 0.f, cl = 0.f, cc = 0.f, cr = 0.f;
    int sector = 0;
    const float low = float(vp.low), high = float(vp.high);
    const bool in = lane < cols;
    for (int r0 = 0; r0 < kRows + 2; r0 += kGroup) {
        int gx[kGroup], gy[kGroup];
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            gx[u] = gy[u] = 0;
            if (r0 + u < kRows + 2 && unsigned(yw + r0 + u) < unsigned(H) && in) {
                const size_t p = size_t(yw + r0 + u) * W + x0 + lane;
                gx[u] = L.dx[p];
                gy[u] = L.dy[p];
            }
        }
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
            const int r = r0 + u;
            if (r >= kRows + 2) break;
            Gradient<GIVEN> q = gradient_of<GIVEN>(gx[u], gy[u]);
            if (unsigned(yw + r) >= unsigned(H) || !in) q.m = 0.f;
            float dl = __shfl_up_sync(kAll, q.m, 1), dr = __shfl_down_sync(kAll, q.m, 1);
            if (lane == 0) dl = s_side[warp][0][r];
            if (lane == kTile - 1) dr = s_side[warp][1][r];
            if (r >= 2) {  // cvRecode.cpp:258-323 for the row above
                const float n1 = sector == 0 ? cl : sector == 1 ? uc : sector == 2 ? ul : ur;
                const float n2 = sector == 0 ? cr : sector == 1 ? q.m : sector == 2 ? dr : dl;
                const int row = warp * kRows + r - 2;
                const bool cand = in && row < rows && cc > low && cc > n1 && (sector >= 2 ? cc > n2 : cc >= n2);
                const uint32_t cm = __ballot_sync(kAll, cand), sm = __ballot_sync(kAll, cand && cc > high);
                if (lane == 0) {
                    s_c[row] = cm;
                    s_st[row] = sm;
                }
            }
            ul = cl;
            uc = cc;
            ur = cr;
            cl = dl;
            cc = q.m;
            cr = dr;
            sector = q.sector;
        }
    }
    __syncthreads();
    const uint32_t c = s_c[lane];
    const uint32_t R = tile_closure(s_st[lane], c, lane);
    const bool firstRow = lane == 0, lastRow = lane == kTile - 1;
    const uint32_t bmask = firstRow || lastRow ? c : c & 0x80000001u;
    uint32_t todo = bmask & ~R;
    if (WARPS == 4)
        todo &= warp == 0 ? (firstRow ? ~0u : 0u) : warp == 1 ? (lastRow ? ~0u : 0u) : warp == 2 ? 1u : 0x80000000u;
    for (unsigned have; (have = __ballot_sync(kAll, todo != 0u)) != 0u;) {
        const int sl = __ffs(have) - 1;
        const uint32_t m = tile_closure(lane == sl ? todo & (0u - todo) : 0u, c, lane);
        todo &= ~m;
        const uint32_t bm = m & bmask;
        const int own = bm ? min(border_pos(__ffs(bm) - 1, lane), border_pos(31 - __clz(bm), lane)) : 255;
        const int label = __reduce_min_sync(kAll, unsigned(own));
        for (uint32_t q = bm; q; q &= q - 1) s_lab[border_pos(__ffs(q) - 1, lane)] = uint8_t(label);
    }
    __syncthreads();
    if (warp == 0) {
        int n = 0;
        for (int w = 0; w < kBorderPos / 32; ++w) {
            const int p = 32 * w + lane;
            const unsigned m = __ballot_sync(kAll, s_lab[p] == p);
            s_rank[p] = uint8_t(n + __popc(m & ((1u << lane) - 1u)));
            n += __popc(m);
        }
        if (n > kTileComps && lane == 0) atomicOr(&lv.cnt[l].err, kErrUnionFind);  // cannot happen (<= 62)
        if (lane < rows) {
            const size_t w = size_t(y0 + lane) * L.WW + tx;
            plane_c(L)[w] = c;
            plane_r(L)[w] = R;
        }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < kBorderPos; p += 32 * WARPS) {
        const int lab = s_lab[p];
        L.blab[size_t(tile) * kBorderPos + p] = lab == 0xff ? uint8_t(0xff) : s_rank[lab];
    }
    for (int k = threadIdx.x; k < kTileComps; k += 32 * WARPS) {
        const size_t id = size_t(tile) * kTileComps + k;
        L.tcomp[id] = int32_t(id);
        L.tflag[id] = 0;
    }
}

// Step 2: pairs of neighbours across tile borders, two warps per tile: its first
// row with the row above (lane = column, three neighbours each), its first
// column with the column to the left (lane = row).  Every 8-neighbour pair that
// straddles a tile border meets here.  Two weak components are joined, once for
// neighbouring pixels of the same two; a weak one next to a pixel of R is marked
// strong.  All words and labels are loaded first, side by side: the kernel is a
// chain of loads and atomics (17 us of a 1080p frame with each pixel's bit, then
// its label, then its neighbours' loaded in turn and every pair joined, 11 us now).
__global__ void __launch_bounds__(64) k_hyst_unions(Levels lv)
{
    int tile;
    const int l = level_of_block(lv, blockIdx.x, &LevelView::uf_tiles, tile);
    const LevelView& L = lv.l[l];
    const int tx = tile % L.uf_tx, ty = tile / L.uf_tx, tilesY = L.uf_tiles / L.uf_tx;
    const int y0 = ty * kTile;
    const int lane = threadIdx.x & 31;
    const bool row = threadIdx.x < 32;
    if (row ? ty == 0 : tx == 0) return;
    const uint32_t* C = plane_c(L);
    const uint32_t* R = plane_r(L);
    const uint8_t* lab = L.blab + size_t(tile) * kBorderPos;
    auto word = [&](const uint32_t* plane, int wx, int y) {
        return wx >= 0 && wx < L.WW && y >= 0 && y < L.H ? __ldg(plane + size_t(y) * L.WW + wx) : 0u;
    };
    // component at border position `pos` of the tile (dx, dy) tiles away
    auto comp = [&](int dx, int dy, int pos) {
        const int qx = tx + dx, qy = ty + dy;
        if (qx < 0 || qx >= L.uf_tx || qy < 0 || qy >= tilesY) return 0;
        const int t = tile + dy * L.uf_tx + dx;
        return t * kTileComps + int(__ldg(L.blab + size_t(t) * kBorderPos + pos));
    };
    // own pixel and the three across the border: candidate, in R, component
    bool oc, orr, nc[3], nr[3];
    int oa, nb[3];
    if (row) {
        const uint32_t c0 = word(C, tx, y0), r0 = word(R, tx, y0);
        const uint32_t um = word(C, tx - 1, y0 - 1), uc = word(C, tx, y0 - 1), up = word(C, tx + 1, y0 - 1);
        const uint32_t sm = word(R, tx - 1, y0 - 1), sc = word(R, tx, y0 - 1), sp = word(R, tx + 1, y0 - 1);
        const int up0 = comp(0, -1, border_pos(lane, kTile - 1));
        const int upL = comp(-1, -1, border_pos(kTile - 1, kTile - 1)), upR = comp(1, -1, border_pos(0, kTile - 1));
        oa = tile * kTileComps + int(__ldg(lab + border_pos(lane, 0)));
        oc = c0 >> lane & 1u;
        orr = r0 >> lane & 1u;
        nc[1] = uc >> lane & 1u;
        nr[1] = sc >> lane & 1u;
        nb[1] = up0;
        nc[0] = lane > 0 ? uc >> (lane - 1) & 1u : um >> 31;
        nr[0] = lane > 0 ? sc >> (lane - 1) & 1u : sm >> 31;
        nc[2] = lane < 31 ? uc >> (lane + 1) & 1u : up & 1u;
        nr[2] = lane < 31 ? sc >> (lane + 1) & 1u : sp & 1u;
        nb[0] = __shfl_up_sync(0xffffffffu, up0, 1);
        nb[2] = __shfl_down_sync(0xffffffffu, up0, 1);
        if (lane == 0) nb[0] = upL;
        if (lane == 31) nb[2] = upR;
    } else {
        const int y = y0 + lane;
        const uint32_t c0 = word(C, tx, y), r0 = word(R, tx, y);
        const uint32_t lc = word(C, tx - 1, y) >> 31, lr = word(R, tx - 1, y) >> 31;
        const uint32_t ac = word(C, tx - 1, y0 - 1) >> 31, ar = word(R, tx - 1, y0 - 1) >> 31;
        const uint32_t dc = word(C, tx - 1, y0 + kTile) >> 31, dr = word(R, tx - 1, y0 + kTile) >> 31;
        const int left = comp(-1, 0, border_pos(kTile - 1, lane));
        const int above = comp(-1, -1, border_pos(kTile - 1, kTile - 1)), below = comp(-1, 1, border_pos(kTile - 1, 0));
        oa = tile * kTileComps + int(__ldg(lab + border_pos(0, lane)));
        oc = c0 & 1u;
        orr = r0 & 1u;
        nc[1] = lc;
        nr[1] = lr;
        nb[1] = left;
        const uint32_t uc = __shfl_up_sync(0xffffffffu, lc, 1), ur = __shfl_up_sync(0xffffffffu, lr, 1);
        const uint32_t wc = __shfl_down_sync(0xffffffffu, lc, 1), wr = __shfl_down_sync(0xffffffffu, lr, 1);
        nb[0] = __shfl_up_sync(0xffffffffu, left, 1);
        nb[2] = __shfl_down_sync(0xffffffffu, left, 1);
        nc[0] = lane > 0 ? uc : ac;
        nr[0] = lane > 0 ? ur : ar;
        nc[2] = lane < 31 ? wc : dc;
        nr[2] = lane < 31 ? wr : dr;
        if (lane == 0) nb[0] = above;
        if (lane == 31) nb[2] = below;
    }
    // weak-weak pairs, without those this lane or the one before has already
    bool join[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        join[d] = false;
        if (!oc || !nc[d] || (orr && nr[d])) continue;
        if (orr) L.tflag[nb[d]] = 1;
        else if (nr[d]) L.tflag[oa] = 1;
        else join[d] = true;
    }
    join[0] = join[0] && !(join[1] && nb[0] == nb[1]);
    join[2] = join[2] && !(join[1] && nb[2] == nb[1]) && !(join[0] && nb[2] == nb[0]);
    const int pa = __shfl_up_sync(0xffffffffu, join[1] ? oa : -1, 1), pb = __shfl_up_sync(0xffffffffu, nb[1], 1);
    if (lane > 0 && pa == oa && pb == nb[1]) join[1] = false;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (join[d]) uf_union(L.tcomp, oa, nb[d], &lv.cnt[l].err);
}

// Each set with a marked member is marked strong at its root; four components
// per thread.
__global__ void __launch_bounds__(256) k_hyst_roots(Levels lv, int total_tiles)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    constexpr int kPer = kTileComps / 4;  // threads per tile
    if (i >= total_tiles * kPer) return;
    int tile;
    const int l = level_of_tile(lv, i / kPer, tile);
    const LevelView& L = lv.l[l];
    const int id = tile * kTileComps + 4 * (i % kPer);
    const int4 f = *reinterpret_cast<const int4*>(L.tflag + id);
    const int own[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (own[k] & 1) atomicOr(&L.tflag[uf_find(L.tcomp, id + k)], 2);
}

__global__ void __launch_bounds__(32 * kHystWarps) k_hyst_final(Levels lv, int total_tiles)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.x * kHystWarps + warp;
    if (g >= total_tiles) return;
    int tile;
    const int l = level_of_tile(lv, g, tile);
    const LevelView& L = lv.l[l];
    const int tx = tile % L.uf_tx, ty = tile / L.uf_tx;
    const int y0 = ty * kTile;
    const int rows = min(kTile, L.H - y0);
    uint32_t c = 0u, R = 0u;
    if (lane < rows) {
        const size_t w = size_t(y0 + lane) * L.WW + tx;
        c = plane_c(L)[w];
        R = plane_r(L)[w];
    }
    // which of the tile's components belong to a strong set (two per lane,
    // the finds side by side; unused components are their own roots, flag 0)
    const int base = tile * kTileComps;
    const bool s0 = L.tflag[uf_find(L.tcomp, base + lane)] & 2;
    const bool s1 = L.tflag[uf_find(L.tcomp, base + 32 + lane)] & 2;
    const uint64_t strongSets =
        uint64_t(__ballot_sync(0xffffffffu, s0)) | (uint64_t(__ballot_sync(0xffffffffu, s1)) << 32);
    // border pixels of those components seed the closure
    __shared__ uint32_t s_lab[kHystWarps][kBorderPos / 4];
    s_lab[warp][lane] = reinterpret_cast<const uint32_t*>(L.blab + size_t(tile) * kBorderPos)[lane];
    __syncwarp();
    const uint8_t* lab = reinterpret_cast<const uint8_t*>(s_lab[warp]);
    const uint32_t bmask = (lane == 0 || lane == kTile - 1) ? c : (c & (1u | (1u << (kTile - 1))));
    uint32_t seed = 0u, bm = strongSets ? (bmask & ~R) : 0u;
    while (bm) {
        const int b = __ffs(bm) - 1;
        bm &= bm - 1;
        if ((strongSets >> lab[border_pos(b, lane)]) & 1ull) seed |= 1u << b;
    }
    const uint32_t H = __any_sync(0xffffffffu, seed != 0u) ? tile_closure(R | seed, c, lane) : R;
    if (lane < rows) plane_h(L)[size_t(y0 + lane) * L.WW + tx] = H;
}

// ------------------------------------------------ final edges + thinning --
// thin() (thinning.cpp:12-51): two Lam-Lee-Suen sub-iterations over the
// hysteresis result, interior pixels only, the image border keeping its
// Canny value.  Evaluated bit-parallel: a warp takes one 32-pixel word column
// and 28 output rows, lane r holding row y0 - 2 + r as a 64-bit window
// (x0 - 16 .. x0 + 47) built from three words of the H plane.  The neighbour
// masks are the window shifted by one bit and the rows above and below
// (shuffles); each sub-iteration's "delete" condition is the conjunction of
// G1 (exactly one of four 0 -> 1 transitions), G2 (2 <= min(n1, n2) <= 3) and
// the sub-iteration's G3, in bitwise form -- the same function as the
// reference's 512-entry tables (checked entry by entry in the tests).  Rows
// and columns two away from the output are enough for the two passes.
constexpr int kThinRows = 28;
constexpr int kThinWarps = 4;

__device__ __forceinline__ uint64_t atl2(uint64_t a, uint64_t b, uint64_t c, uint64_t d)
{
    return ((a | b) & (c | d)) | (a & b) | (c & d);
}

// Pixels of plane P that one sub-iteration keeps (pass 1 or 2), as a mask;
// up / dn are the rows above and below.
__device__ __forceinline__ uint64_t thin_keep(uint64_t P, uint64_t up, uint64_t dn, int pass)
{
    const uint64_t x1 = P >> 1, x2 = up >> 1, x3 = up, x4 = up << 1;  // E, NE, N, NW
    const uint64_t x5 = P << 1, x6 = dn << 1, x7 = dn, x8 = dn >> 1;  // W, SW, S, SE
    const uint64_t b1 = ~x1 & (x2 | x3), b2 = ~x3 & (x4 | x5), b3 = ~x5 & (x6 | x7), b4 = ~x7 & (x8 | x1);
    const uint64_t g1 = (b1 | b2 | b3 | b4) & ~atl2(b1, b2, b3, b4);
    const uint64_t a1 = x1 | x2, a2 = x3 | x4, a3 = x5 | x6, a4 = x7 | x8;
    const uint64_t c1 = x2 | x3, c2 = x4 | x5, c3 = x6 | x7, c4 = x8 | x1;
    const uint64_t g2 = atl2(a1, a2, a3, a4) & atl2(c1, c2, c3, c4) & ~((a1 & a2 & a3 & a4) & (c1 & c2 & c3 & c4));
    const uint64_t g3 = pass == 1 ? ~((x2 | x3 | ~x8) & x1) : ~((x6 | x7 | ~x4) & x5);
    return P & ~(g1 & g2 & g3);
}

// Bits of the window (bit i = column x0 - 16 + i) whose column lies in [lo, hi].
__device__ __forceinline__ uint64_t col_range(int x0, int lo, int hi)
{
    const int a = max(lo - (x0 - 16), 0), b = min(hi - (x0 - 16), 63);
    if (b < a) return 0ull;
    const uint64_t upto = b == 63 ? ~0ull : ((1ull << (b + 1)) - 1ull);
    return upto & ~((1ull << a) - 1ull);
}

__global__ void __launch_bounds__(32 * kThinWarps) k_final_thin(Levels lv, int total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int g = blockIdx.x * kThinWarps + warp;
    if (g >= total) return;
    int l = 0;
    while (l < lv.n - 1 && g >= lv.l[l].thin_tiles) {
        g -= lv.l[l].thin_tiles;
        ++l;
    }
    const LevelView& L = lv.l[l];
    const int W = L.W, H = L.H, WW = L.WW;
    const int wx = g % WW, y0 = (g / WW) * kThinRows;
    const int x0 = wx * 32;
    const int y = y0 - 2 + lane;
    uint64_t P = 0ull;
    if (y >= 0 && y < H) {
        const uint32_t* row = plane_h(L) + size_t(y) * WW;
        const uint32_t wl = wx > 0 ? row[wx - 1] : 0u, wc = row[wx], wr = wx + 1 < WW ? row[wx + 1] : 0u;
        P = uint64_t((wl >> 16) | (wc << 16)) | (uint64_t((wc >> 16) | (wr << 16)) << 32);
    }
    const bool rowInterior = y >= 1 && y <= H - 2;
    const uint64_t interior = rowInterior ? col_range(x0, 1, W - 2) : 0ull;
    uint64_t up = __shfl_up_sync(0xffffffffu, P, 1), dn = __shfl_down_sync(0xffffffffu, P, 1);
    const uint64_t T = thin_keep(P, up, dn, 1) & interior;
    up = __shfl_up_sync(0xffffffffu, T, 1);
    dn = __shfl_down_sync(0xffffffffu, T, 1);
    const uint64_t inImage = (y >= 0 && y < H) ? col_range(x0, 0, W - 1) : 0ull;
    const uint64_t out = (thin_keep(T, up, dn, 2) & interior) | (P & inImage & ~interior);
    if (lane >= 2 && lane < 2 + kThinRows && y < H) {
        const uint32_t word = uint32_t(out >> 16);
        L.bitmap[size_t(y) * WW + wx] = word;
        if (word && L.row_count) atomicAdd(&L.row_count[y], __popc(word));
    }
}

// ------------------------------------------------------------------ scans --
__device__ __forceinline__ int warp_incl_scan(int v)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= o) v += n;
    }
    return v;
}

// Exclusive block scan (blockDim.x multiple of 32, <= 1024); returns the block total in *total.
__device__ __forceinline__ int block_excl_scan(int v, int* s_warp, int* total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int inc = warp_incl_scan(v);
    if (lane == 31) s_warp[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const int w = lane < nw ? s_warp[lane] : 0;
        const int wi = warp_incl_scan(w);
        if (lane < nw) s_warp[lane] = wi - w;
        if (lane == nw - 1) s_warp[32] = wi;
    }
    __syncthreads();
    const int res = inc - v + s_warp[wid];
    *total = s_warp[32];
    __syncthreads();
    return res;
}

// One block per level: row_off = exclusive scan of row_count; E clamped to the
// capacity (overflow flagged); row_count is cleared for the next frame.
__global__ void __launch_bounds__(1024) k_row_scan(Levels lv)
{
    __shared__ int s_warp[33];
    const int l = blockIdx.x;
    const LevelView& L = lv.l[l];
    int carry = 0;
    for (int base = 0; base < L.H; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < L.H ? L.row_count[i] : 0;
        int total;
        const int ex = block_excl_scan(v, s_warp, &total);
        if (i < L.H) {
            L.row_off[i] = carry + ex;
            L.row_count[i] = 0;
        }
        carry += total;
    }
    if (threadIdx.x == 0) {
        L.row_off[L.H] = carry;
        int E = carry;
        if (E > L.cap) {
            atomicOr(&lv.cnt[l].err, kErrEdgeOverflow);
            E = L.cap;
        }
        lv.cnt[l].E = E;
    }
}

// One block (4 warps) per image row: raster-order edge list, per-point state
// reset, and per bitmap word the word with the index of its first edge point
// (an edge pixel's index is that plus the word's set bits below it).
// EdgePointCollection::add_point, Types.cpp:40-61.
__global__ void __launch_bounds__(128) k_emit(Levels lv, int rows_total)
{
    __shared__ int s_warp[4];
    int y = blockIdx.x, l = 0;
    while (l < lv.n - 1 && y >= lv.l[l].H) { y -= lv.l[l].H; ++l; }
    const LevelView& L = lv.l[l];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int per = (L.WW + 3) / 4;
    const int w0 = wid * per, w1 = min(L.WW, w0 + per);
    const uint32_t* row = L.bitmap + size_t(y) * L.WW;
    int cnt = 0;
    for (int w = w0 + lane; w < w1; w += 32) cnt += __popc(row[w]);
#pragma unroll
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0) s_warp[wid] = cnt;
    __syncthreads();
    int base = L.row_off[y];
    for (int k = 0; k < wid; ++k) base += s_warp[k];
    uint2* bi = L.bitidx + size_t(y) * L.WW;
    for (int w = w0; w < w1; ++w) {
        const uint32_t m = row[w];
        if (lane == 0) bi[w] = make_uint2(m, uint32_t(base));
        if (!m) continue;
        if ((m >> lane) & 1u) {
            const int idx = base + __popc(m & ((1u << lane) - 1u));
            if (idx < L.cap) {
                const int x = (w << 5) + lane;
                const size_t p = size_t(y) * L.W + x;
                L.exy[idx] = x | (y << 16);
                L.grad[idx] = int32_t(uint16_t(L.dx[p])) | (int32_t(L.dy[p]) << 16);
                L.nvotes[idx] = 0;
                L.fill[idx] = 0;
            }
        }
        base += __popc(m);
    }
}

// ------------------------------------------------------ gradient walk --
// Bresenham.cpp:18-209: from an edge point, follow the gradient (dir = -1
// backward, +1 forward) for up to distSearch steps and return the index of the
// first edge point met, or -1.
//
// Bound by the instructions of the steps (71 % of the issue slots, 19 of 32
// lanes at work, with one loop over all steps of a walk).  Most walks stop
// within three steps: those are taken by a lane per point for both directions
// at once, which share the line's error terms, with all their probes in flight.
// The others run the full distance or stop anywhere: a lane takes the next of
// the warp's chunk as soon as its current one stops, two steps per iteration,
// their probes loaded before the first is tested (steps past the walk's end are
// computed and dropped).  A position is one word, x + 65536 y, so a step is one
// addition (the sides are at most 16384); a coordinate of a walk never turns
// back, so the side probe, which has one coordinate of this step's and one of
// the last step's position, is inside wherever the step is.  The steps and
// probes of every walk are those of the reference in the same order, so the
// results do not depend on the schedule.  Measured: 1080p frame (380 k points
// on four levels) 54 -> 32 us, 3840x2160 clutter 174 -> 110 us.
constexpr int kWalkWarps = 8;
constexpr int kWalkChunk = 512;  // walks (two per point) a warp takes at once, at most

__device__ __forceinline__ int sgn_i(int v) { return (v > 0) - (v < 0); }

// A walk step: the position moves by the major step m, and by the minor step as
// well when the error reaches half a pixel (the return value).
__device__ __forceinline__ bool walk_step(float& e, float a)
{
    e = __fadd_rn(e, a);
    const bool c = e >= 0.5f;
    if (c) e = __fadd_rn(e, -1.f);
    return c;
}

// The pixel's bit of a bitidx word, and its edge point's index.
__device__ __forceinline__ bool walk_hit(uint2 w, int at) { return __funnelshift_r(w.x, 0u, at) & 1u; }
__device__ __forceinline__ int walk_index(uint2 w, int at, int E)
{
    const int idx = int(w.y) + __popc(w.x & ((1u << (at & 31)) - 1u));
    return idx < E ? idx : -1;  // -1 past a clamped edge count
}

__global__ void __launch_bounds__(32 * kWalkWarps) k_walk(Levels lv, VoteParamsDev vp)
{
    __shared__ float s_a[kWalkWarps][kWalkChunk / 2], s_e[kWalkWarps][kWalkChunk / 2];
    __shared__ uint8_t s_g[kWalkWarps][kWalkChunk / 2];
    __shared__ int s_res[kWalkWarps][kWalkChunk];        // a walk's position after three steps, then its result
    __shared__ uint16_t s_list[kWalkWarps][kWalkChunk];  // the walks that go on from there
    const unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int gw = blockIdx.x * kWalkWarps + wid, NW = gridDim.x * kWalkWarps;
    const int nmax = vp.distSearch;
    // chunk size: the launch's walks spread over its warps (a multiple of 32,
    // 32 .. kWalkChunk), the same in every block
    long long walks = 0;
    for (int l = 0; l < lv.n; ++l) walks += 2LL * lv.cnt[l].E;
    long long per = (walks / NW + 31) / 32 * 32;
    const int chunk = per < 32 ? 32 : per > kWalkChunk ? kWalkChunk : int(per);
    int first = 0;  // global number of the level's first chunk
    for (int l = 0; l < lv.n; ++l) {
        const LevelView& L = lv.l[l];
        const int E = lv.cnt[l].E;
        const int W = L.W, H = L.H, WW = L.WW;
        const uint2* __restrict__ bits = L.bitidx;
        const int nch = (2 * E + chunk - 1) / chunk;
        int c = (gw - first % NW + NW) % NW;
        first += nch;
        auto inside = [&](int at) { return unsigned(at & 0xffff) < unsigned(W) && unsigned(at >> 16) < unsigned(H); };
        auto word = [&](int at) { return __ldg(bits + ((at >> 16) * WW + ((at & 0xffff) >> 5))); };
        for (; c < nch; c += NW) {
            const int t0 = c * chunk, t1 = min(2 * E, t0 + chunk);
            const int p0 = t0 >> 1, np = (t1 - t0) >> 1;
            int ns = 0;
            for (int i0 = 0; i0 < np; i0 += 32) {
                const int i = i0 + lane;
                const bool in = i < np;
                int res[2] = {-1, -1}, at[2] = {0, 0};
                bool more[2] = {false, false};
                if (in) {
                    const int xy = L.exy[p0 + i], g = L.grad[p0 + i];
                    const int gxi = int16_t(g & 0xffff), gyi = g >> 16;
                    const float gx = float(gxi), gy = float(gyi);
                    const bool ym = fabsf(gy) > fabsf(gx);
                    const int smaj = sgn_i(ym ? gyi : gxi), smin = sgn_i(ym ? gxi : gyi);
                    // |dmin / dmaj|, the same for both directions, as is the error
                    const float a = fabsf(__fdiv_rn(ym ? gx : gy, ym ? gy : gx));
                    // After the first step the reference re-orients the walk
                    // along the gradient at its start point (Bresenham.cpp:
                    // 74-81): the direction already is dir * g, its product
                    // with g is dir * |g|^2, so the direction stays dir * g
                    // (0 when g is 0) and the steps are unchanged.  No probe
                    // after the first step, and no side probe after the second.
                    const int m = ym ? smaj * 65536 : smaj, n = ym ? smin : smin * 65536;
                    float e = 0.f;
                    const int d1 = m + (walk_step(e, a) ? n : 0);
                    const int d2 = d1 + m + (walk_step(e, a) ? n : 0);
                    const int d3 = d2 + m + (walk_step(e, a) ? n : 0);
                    s_a[wid][i] = a;
                    s_e[wid][i] = e;
                    s_g[wid][i] = uint8_t((ym ? 1 : 0) | (smaj + 1) << 1 | (smin + 1) << 3);
                    uint2 w2[2], w3[2], ws[2];
                    bool in2[2], in3[2];
#pragma unroll
                    for (int d = 0; d < 2; ++d) {
                        const int dir = d ? 1 : -1;
                        in2[d] = inside(xy + dir * d2);
                        in3[d] = inside(xy + dir * d3);
                        w2[d] = w3[d] = ws[d] = make_uint2(0u, 0u);
                        if (in2[d]) w2[d] = word(xy + dir * d2);
                        if (in3[d]) {
                            w3[d] = word(xy + dir * d3);
                            ws[d] = word(xy + dir * (d3 - m));
                        }
                    }
#pragma unroll
                    for (int d = 0; d < 2; ++d) {
                        const int dir = d ? 1 : -1;
                        if (!in2[d]) continue;
                        if (walk_hit(w2[d], xy + dir * d2)) {
                            res[d] = walk_index(w2[d], xy + dir * d2, E);
                        } else if (2 <= nmax && in3[d]) {
                            at[d] = xy + dir * d3;
                            if (walk_hit(w3[d], at[d])) res[d] = walk_index(w3[d], at[d], E);
                            else if (walk_hit(ws[d], at[d] - dir * m)) res[d] = walk_index(ws[d], at[d] - dir * m, E);
                            else more[d] = true;
                        }
                    }
                }
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    if (in) s_res[wid][2 * i + d] = more[d] ? at[d] : res[d];
                    const unsigned b = __ballot_sync(kAll, more[d]);
                    if (more[d]) s_list[wid][ns + __popc(b & below)] = uint16_t(2 * i + d);
                    ns += __popc(b);
                }
            }
            __syncwarp();
            int q = 0, t = 0, at = 0, n = 0, m = 0, mn = 0;  // major step; major and minor step
            float e = 0.f, a = 0.f;
            bool act = false;
            while (true) {
                const unsigned idle = __ballot_sync(kAll, !act);
                if (!act) {
                    const int k = q + __popc(idle & below);
                    if (k < ns) {
                        t = s_list[wid][k];
                        act = true;
                        const int i = t >> 1, st = s_g[wid][i], dir = (t & 1) ? 1 : -1;
                        const int maj = dir * ((st >> 1 & 3) - 1), min_ = dir * ((st >> 3) - 1);
                        m = st & 1 ? maj * 65536 : maj;
                        mn = m + (st & 1 ? min_ : min_ * 65536);
                        at = s_res[wid][t];
                        a = s_a[wid][i];
                        e = s_e[wid][i];
                        n = 3;
                    }
                }
                q += __popc(idle);
                if (!__any_sync(kAll, act)) break;
                if (!act) continue;
                // the walk ends before a step once n > nmax
                const int a0 = at + (walk_step(e, a) ? mn : m), a1 = a0 + (walk_step(e, a) ? mn : m);
                const bool in0 = inside(a0) && n <= nmax, in1 = inside(a1) && n < nmax;
                uint2 w0 = make_uint2(0u, 0u), w1 = w0, v0 = w0, v1 = w0;
                if (in0) {
                    w0 = word(a0);
                    v0 = word(a0 - m);
                }
                if (in1) {
                    w1 = word(a1);
                    v1 = word(a1 - m);
                }
                const bool f0 = walk_hit(w0, a0), g0 = walk_hit(v0, a0 - m);
                const bool f1 = walk_hit(w1, a1), g1 = walk_hit(v1, a1 - m);
                if (!in1 || f0 || g0 || f1 || g1) {
                    int res = -1;
                    if (f0) res = walk_index(w0, a0, E);
                    else if (g0) res = walk_index(v0, a0 - m, E);
                    else if (f1) res = walk_index(w1, a1, E);
                    else if (g1) res = walk_index(v1, a1 - m, E);
                    s_res[wid][t] = res;
                    act = false;
                }
                at = a1;
                n += 2;
            }
            __syncwarp();
            for (int i = lane; i < np; i += 32) {
                L.before[p0 + i] = s_res[wid][2 * i];
                L.after[p0 + i] = s_res[wid][2 * i + 1];
            }
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------ vote --
// Vote.cpp:101-243: follow before/after links across the 2*nCrowns-1 ring
// edges with the gradient-angle and distance-ratio tests.
__device__ __forceinline__ float pt_dist(int xya, int xyb)
{
    const int ddx = (xyb & 0xffff) - (xya & 0xffff), ddy = (xyb >> 16) - (xya >> 16);
    return __fsqrt_rn(__fadd_rn(float(ddx * ddx), float(ddy * ddy)));
}

__device__ __forceinline__ float neg_dot(int ga, int gb)
{
    const int d = int(int16_t(ga & 0xffff)) * int(int16_t(gb & 0xffff)) + (ga >> 16) * (gb >> 16);
    return -float(d);
}

__global__ void k_vote(Levels lv, VoteParamsDev vp)
{
    const int stride = gridDim.x * blockDim.x;
    constexpr int kMaxSeg = 16;
    for (int l = 0; l < lv.n; ++l) {
        const LevelView& L = lv.l[l];
        const int E = lv.cnt[l].E;
        for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < E; p += stride) {
            float vd[kMaxSeg];
            int nd = 0;
            float total = 0.f;
            int chosen = -1;
            int current = L.before[p];
            const int gp = L.grad[p];
            const int xyp = L.exy[p];
            auto ratio_ok = [&]() {
                bool ok = true;
                for (int i = 0; i < nd; ++i)
                    for (int j = i + 1; j < nd; ++j)
                        ok = ok && (vd[i] <= __fmul_rn(vd[j], vp.ratioVoting)) && (vd[j] <= __fmul_rn(vd[i], vp.ratioVoting));
                return ok;
            };
            if (current >= 0 && neg_dot(gp, L.grad[current]) >= vp.angleVoting && 2 * vp.nCrowns - 1 <= kMaxSeg) {
                float d = pt_dist(xyp, L.exy[current]);
                vd[nd++] = d;
                total = __fadd_rn(total, d);
                for (int i = 1; i < vp.nCrowns; ++i) {
                    chosen = -1;
                    int target = L.after[current];
                    if (target < 0) break;
                    if (!(neg_dot(L.grad[target], L.grad[current]) >= vp.angleVoting)) break;
                    d = pt_dist(L.exy[target], L.exy[current]);
                    vd[nd++] = d;
                    total = __fadd_rn(total, d);
                    if (nd > 1 && !ratio_ok()) break;
                    current = target;
                    target = L.before[current];
                    if (target < 0) break;
                    if (!(neg_dot(L.grad[target], L.grad[current]) >= vp.angleVoting)) break;
                    d = pt_dist(L.exy[target], L.exy[current]);
                    vd[nd++] = d;
                    total = __fadd_rn(total, d);
                    if (!ratio_ok()) break;
                    current = target;
                    chosen = current;
                }
            }
            L.chosen[p] = chosen;
            L.total[p] = chosen >= 0 ? total : 0.f;
            if (chosen >= 0) atomicAdd(&L.nvotes[chosen], 1);
        }
    }
}

// ----------------------------------------------------- voter lists (CSR) --
// Chunked exclusive scan of nvotes[0, E) into voff: level blockIdx.y, one block
// per chunk, up to kScanBlocksPerLevel of them, of a multiple of 1024 points
// (four per thread and load).  A large level then has a chunk per SM (with 32
// chunks per level and one point per load, a 3840x2160 clutter frame's 1.2 M
// points of level 0 took 189 us in the two kernels, 18 us now).
constexpr int kScanBlocks = kScanBlocksPerLevel;
constexpr int kScanThreads = 256;
constexpr int kScanStep = 4 * kScanThreads;  // points per iteration of a block

__device__ __forceinline__ int scan_chunk(int E)
{
    const int per = (E + kScanBlocks - 1) / kScanBlocks;
    return max((per + kScanStep - 1) / kScanStep, 1) * kScanStep;
}

// Points [i, i + 4) of a, 0 from n on; i is a multiple of 4.
__device__ __forceinline__ int4 load4(const int32_t* a, int i, int n)
{
    if (i + 4 <= n) return *reinterpret_cast<const int4*>(a + i);
    return make_int4(i < n ? a[i] : 0, i + 1 < n ? a[i + 1] : 0, i + 2 < n ? a[i + 2] : 0, 0);
}

__global__ void __launch_bounds__(kScanThreads) k_vscan_partial(Levels lv, int32_t* partial)
{
    __shared__ int s_sum;
    const int l = blockIdx.y;
    const LevelView& L = lv.l[l];
    const int E = lv.cnt[l].E;
    const int chunk = scan_chunk(E);
    const int b0 = min(E, int(blockIdx.x) * chunk), b1 = min(E, b0 + chunk);
    if (b0 >= b1) return;  // its partial sum is not read
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    int s = 0;
    for (int i = b0 + 4 * int(threadIdx.x); i < b1; i += kScanStep) {
        const int4 v = load4(L.nvotes, i, b1);
        s += v.x + v.y + v.z + v.w;
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, s);
    __syncthreads();
    if (threadIdx.x == 0) partial[l * kScanBlocks + blockIdx.x] = s_sum;
}

__global__ void __launch_bounds__(kScanThreads) k_vscan_final(Levels lv, const int32_t* partial)
{
    __shared__ int s_warp[33];
    __shared__ int s_base;
    const int l = blockIdx.y;
    const LevelView& L = lv.l[l];
    const int E = lv.cnt[l].E;
    const int chunk = scan_chunk(E);
    const int b0 = min(E, int(blockIdx.x) * chunk), b1 = min(E, b0 + chunk);
    if (b0 >= b1) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            L.voff[0] = 0;
            lv.cnt[l].V = 0;
        }
        return;
    }
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    int before = int(threadIdx.x) < int(blockIdx.x) ? partial[l * kScanBlocks + threadIdx.x] : 0;
    static_assert(kScanBlocks <= kScanThreads, "one partial sum per thread");
    before = __reduce_add_sync(0xffffffffu, before);
    if ((threadIdx.x & 31) == 0 && before) atomicAdd(&s_base, before);
    __syncthreads();
    int carry = s_base;
    for (int i0 = b0; i0 < b1; i0 += kScanStep) {
        const int i = i0 + 4 * int(threadIdx.x);
        const int4 v = load4(L.nvotes, i, b1);
        int total;
        const int ex = carry + block_excl_scan(v.x + v.y + v.z + v.w, s_warp, &total);
        const int4 o = make_int4(ex, ex + v.x, ex + v.x + v.y, ex + v.x + v.y + v.z);
        if (i + 4 <= b1) {
            *reinterpret_cast<int4*>(L.voff + i) = o;
        } else {
            if (i < b1) L.voff[i] = o.x;
            if (i + 1 < b1) L.voff[i + 1] = o.y;
            if (i + 2 < b1) L.voff[i + 2] = o.z;
        }
        carry += total;
    }
    if (b1 == E && threadIdx.x == 0) {
        L.voff[E] = carry;
        lv.cnt[l].V = carry;
    }
}

__global__ void k_vfill(Levels lv)
{
    const int stride = gridDim.x * blockDim.x;
    for (int l = 0; l < lv.n; ++l) {
        const LevelView& L = lv.l[l];
        const int E = lv.cnt[l].E;
        for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < E; p += stride) {
            const int c = L.chosen[p];
            if (c < 0) continue;
            const int slot = atomicAdd(&L.fill[c], 1);
            L.vlist[L.voff[c] + slot] = p;
        }
    }
}

// One step of the running mean of the field-line lengths in ascending voter
// order (Vote.cpp:232): (mean * k + length) / (k + 1), the division correctly
// rounded by div_small up to 256 voters (the lengths are sums of distances of
// distinct pixels: 0 or normal); rcp = 1 / (k + 1), rounded.
__device__ __forceinline__ float flow_step(float mean, int k, float length, float rcp)
{
    const float x = __fadd_rn(__fmul_rn(mean, float(k)), length), d = float(k + 1);
    return k < 256 ? pm::div_small(x, d, rcp) : __fdiv_rn(x, d);
}

// Seed registration (Vote.cpp:236-241) of the lanes that have one, one atomic
// per warp; every lane of the warp calls it.
__device__ __forceinline__ void push_seed(const LevelView& L, LevelCounters& cnt, bool seed, int c, int key, int votes)
{
    const unsigned m = __ballot_sync(0xffffffffu, seed);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    int s = 0;
    if (lane == __ffs(m) - 1) s = atomicAdd(&cnt.S, __popc(m));
    s = __shfl_sync(0xffffffffu, s, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
    if (!seed) return;
    if (s < L.seedcap) {
        L.seed_idx[s] = c;
        L.seed_key[s] = key;
        L.seed_votes[s] = votes;
    } else {
        atomicOr(&cnt.err, kErrSeedOverflow);
    }
}

// Voter lists in ascending order, flow lengths and seeds.  Nearly all lists are
// short (of a 1080p frame's 285 k points 4 % have votes, 21 more than 8): a
// thread per point sorts up to kThreadList voters in registers, with all loads
// of a list in flight; the warp takes its longer lists up to kWarpList
// together; the rest are queued for a block each.  What took the time before
// was the few long lists: one thread's chain of a load and a division per voter
// (1080p frame: 21 + 54 us for the two kernels, 17 + 16 us now; 3840x2160
// clutter: 58 + 34, 36 + 4 us).
constexpr int kThreadList = 8;
constexpr int kWarpList = 64;

// Ascending sort of 8 values (Batcher's network of 19 exchanges).
__device__ __forceinline__ void sort8(int (&v)[8])
{
    auto ex = [&](int a, int b) {
        const int lo = min(v[a], v[b]), hi = max(v[a], v[b]);
        v[a] = lo;
        v[b] = hi;
    };
    ex(0, 1); ex(2, 3); ex(4, 5); ex(6, 7);
    ex(0, 2); ex(1, 3); ex(4, 6); ex(5, 7);
    ex(1, 2); ex(5, 6);
    ex(0, 4); ex(1, 5); ex(2, 6); ex(3, 7);
    ex(2, 4); ex(3, 5);
    ex(1, 2); ex(3, 4); ex(5, 6);
}

constexpr int kListWarps = 8;

__global__ void __launch_bounds__(32 * kListWarps) k_vlists(Levels lv, VoteParamsDev vp)
{
    __shared__ int s_sorted[kListWarps][kWarpList];
    const int stride = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int l = 0; l < lv.n; ++l) {
        const LevelView& L = lv.l[l];
        LevelCounters& cnt = lv.cnt[l];
        const int E = cnt.E;
        for (int c0 = blockIdx.x * blockDim.x + warp * 32; c0 < E; c0 += stride) {
            const int c = c0 + lane;
            const bool in = c < E;
            const int off = in ? L.voff[c] : 0, n = in ? L.voff[c + 1] - off : 0;
            bool seed = false;
            int key = 0;
            if (in && n <= kThreadList) {
                float fl = 0.f;
                if (n) {
                    int v[kThreadList];
                    float t[kThreadList];
#pragma unroll
                    for (int k = 0; k < kThreadList; ++k) v[k] = k < n ? L.vlist[off + k] : 0x7fffffff;
                    sort8(v);
#pragma unroll
                    for (int k = 0; k < kThreadList; ++k) t[k] = k < n ? L.total[v[k]] : 0.f;
#pragma unroll
                    for (int k = 0; k < kThreadList; ++k) {
                        if (k < n) {
                            L.vlist[off + k] = v[k];
                            fl = flow_step(fl, k, t[k], __frcp_rn(float(k + 1)));
                        }
                        if (k == max(vp.minVotes - 1, 0)) key = v[k];
                    }
                    seed = n >= vp.minVotes;
                }
                L.flow[c] = fl;
            }
            for (unsigned m = __ballot_sync(0xffffffffu, n > kThreadList); m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const int cs = c0 + src, on = __shfl_sync(0xffffffffu, off, src), ns = __shfl_sync(0xffffffffu, n, src);
                if (ns > kWarpList) {
                    if (lane == 0) L.bigq[atomicAdd(&cnt.bigq, 1)] = cs;
                    continue;
                }
                // two voters per lane; an element's rank is the number below it
                const int a = lane < ns ? L.vlist[on + lane] : 0x7fffffff;
                const int b = lane + 32 < ns ? L.vlist[on + lane + 32] : 0x7fffffff;
                int ra = 0, rb = 0;
                for (int k = 0; k < ns; ++k) {
                    const int x = __shfl_sync(0xffffffffu, k < 32 ? a : b, k & 31);
                    ra += x < a ? 1 : 0;
                    rb += x < b ? 1 : 0;
                }
                if (lane < ns) s_sorted[warp][ra] = a;
                if (lane + 32 < ns) s_sorted[warp][rb] = b;
                __syncwarp();
                float ta = 0.f, tb = 0.f;
                if (lane < ns) {
                    const int v = s_sorted[warp][lane];
                    L.vlist[on + lane] = v;
                    ta = L.total[v];
                }
                if (lane + 32 < ns) {
                    const int v = s_sorted[warp][lane + 32];
                    L.vlist[on + lane + 32] = v;
                    tb = L.total[v];
                }
                const float qa = __frcp_rn(float(lane + 1)), qb = __frcp_rn(float(lane + 33));
                float fl = 0.f;
#pragma unroll 4
                for (int k = 0; k < ns; ++k)
                    fl = flow_step(fl, k, __shfl_sync(0xffffffffu, k < 32 ? ta : tb, k & 31),
                                   __shfl_sync(0xffffffffu, k < 32 ? qa : qb, k & 31));
                if (lane == src) {
                    L.flow[cs] = fl;
                    seed = ns >= vp.minVotes;
                    if (seed) key = s_sorted[warp][max(vp.minVotes - 1, 0)];
                }
                __syncwarp();
            }
            push_seed(L, cnt, seed, c, key, n);
        }
    }
}

// Very long voter lists: one block per list, rank sort (voter indices are
// distinct), the lengths staged for the running mean.
constexpr int kBigSmem = 4096;

__global__ void __launch_bounds__(256) k_vlists_big(Levels lv, VoteParamsDev vp)
{
    __shared__ int32_t s_in[kBigSmem];
    __shared__ int32_t s_out[kBigSmem];
    for (int l = 0; l < lv.n; ++l) {
        const LevelView& L = lv.l[l];
        const int nq = lv.cnt[l].bigq;
        for (int qi = blockIdx.x; qi < nq; qi += gridDim.x) {
            const int c = L.bigq[qi];
            int32_t* list = L.vlist + L.voff[c];
            const int n = L.voff[c + 1] - L.voff[c];
            if (n <= kBigSmem) {
                for (int k = threadIdx.x; k < n; k += blockDim.x) s_in[k] = list[k];
                __syncthreads();
                for (int k = threadIdx.x; k < n; k += blockDim.x) {
                    const int v = s_in[k];
                    int rank = 0;
                    for (int j = 0; j < n; ++j) rank += s_in[j] < v;
                    s_out[rank] = v;
                }
                __syncthreads();
                for (int k = threadIdx.x; k < n; k += blockDim.x) list[k] = s_out[k];
            } else {
                // rank from global memory in place is impossible, so the ranks
                // are staged through the fill array (free after k_vfill)
                for (int k = threadIdx.x; k < n; k += blockDim.x) {
                    const int v = list[k];
                    int rank = 0;
                    for (int j = 0; j < n; ++j) rank += list[j] < v;
                    L.fill[L.voff[c] + rank] = v;
                }
                __syncthreads();
                for (int k = threadIdx.x; k < n; k += blockDim.x) list[k] = L.fill[L.voff[c] + k];
            }
            __syncthreads();
            float fl = 0.f;  // of thread 0, over the staged lengths
            float* s_len = reinterpret_cast<float*>(s_in);
            float* s_rcp = reinterpret_cast<float*>(s_out);
            for (int k0 = 0; k0 < n; k0 += kBigSmem) {
                const int m = min(n - k0, kBigSmem);
                for (int k = threadIdx.x; k < m; k += blockDim.x) {
                    s_len[k] = L.total[list[k0 + k]];
                    s_rcp[k] = __frcp_rn(float(k0 + k + 1));
                }
                __syncthreads();
                if (threadIdx.x == 0)
#pragma unroll 8
                    for (int k = 0; k < m; ++k) fl = flow_step(fl, k0 + k, s_len[k], s_rcp[k]);
                __syncthreads();
            }
            if (threadIdx.x < 32) {
                if (threadIdx.x == 0) L.flow[c] = fl;
                const bool seed = threadIdx.x == 0 && n >= vp.minVotes;
                push_seed(L, lv.cnt[l], seed, c, seed ? list[max(vp.minVotes - 1, 0)] : 0, n);
            }
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------- launchers --
static int total_of(const Levels& lv, int LevelView::*f)
{
    int s = 0;
    for (int l = 0; l < lv.n; ++l) s += lv.l[l].*f;
    return s;
}

void upload_constants(const float*, int, int)
{
    // The tables are initialised statically with the module (cK, cThinTab);
    // nothing is uploaded, so a context that reloads the module after a
    // device reset sees them too.
}

// fused: every frame has 4 levels and sides that are multiples of 8 (one
// k_pyramid3 launch, blockIdx.z = frame); else one resize launch per level.
static void launch_pyramid(const Levels& lv, cudaStream_t s, bool fused)
{
    const int lpf = lv.n / lv.frames;
    if (lpf < 2) return;
    if (fused && lpf == 4) {
        int w8 = 0, h8 = 0;
        for (int f = 0; f < lv.frames; ++f) {
            w8 = std::max(w8, lv.l[f * lpf].W / 8);
            h8 = std::max(h8, lv.l[f * lpf].H / 8);
        }
        const dim3 blk(32, 8);
        const dim3 grd((w8 + 31) / 32, (h8 + 7) / 8, lv.frames);
        k_pyramid3<<<grd, blk, 0, s>>>(lv);
        return;
    }
    for (int f = 0; f < lv.frames; ++f)
        for (int k = 1; k < lpf; ++k) {
            const LevelView& a = lv.l[f * lpf + k - 1];
            const LevelView& b = lv.l[f * lpf + k];
            const dim3 blk(32, 8);
            const dim3 grd((b.W + 31) / 32, (b.H + 7) / 8);
            k_resize_level<<<grd, blk, 0, s>>>(a.src, a.W, a.H, b.src, b.W, b.H);
        }
}

const char* stage_name(int k)
{
    static const char* names[kStageCount] = {"pyramid", "deriv_nms", "hyst_merge", "hyst_compress", "final_thin",
                                             "row_scan", "emit", "walk", "vote", "voter_scan", "voter_fill",
                                             "voter_sort"};
    return (k >= 0 && k < kStageCount) ? names[k] : "?";
}

static void mark(cudaEvent_t* ev, int k, cudaStream_t s)
{
    if (ev) CCTAGB_CUDA(cudaEventRecord(ev[k], s));
}

// Holds the stream for about `us` microseconds (bounded loop) so that the
// host can queue every stage behind it; used only by the per-stage timing
// mode, which launches without a graph.
__global__ void k_gate(int us)
{
    for (int i = 0; i < us; ++i) __nanosleep(1000);
}

void launch_gate(cudaStream_t s, int us) { k_gate<<<1, 1, 0, s>>>(us); }

// The segments of p back to back into dst: a flat grid-stride loop over the
// total, each thread advancing its segment cursor as its index grows.
__global__ void __launch_bounds__(256) k_pack_words(PackSegs p, int32_t* __restrict__ dst)
{
    const long long total = p.off[p.n];
    const long long stride = (long long)gridDim.x * blockDim.x;
    int g = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        while (i >= p.off[g + 1]) ++g;  // i < off[n], so g < n
        dst[i] = __ldg(p.src[g] + (i - p.off[g]));
    }
}

int launch_pack(const PackSegs& p, int32_t* dst, cudaStream_t s)
{
    if (p.n <= 0 || p.n > kMaxPackSegs) return 0;
    const long long total = p.off[p.n];
    if (total <= 0) return 0;
    const int blocks = int(std::min<long long>((total + 255) / 256, 148 * 4));
    k_pack_words<<<blocks, 256, 0, s>>>(p, dst);
    CCTAGB_CUDA(cudaGetLastError());
    return 1;
}

static void launch_edges(const Levels& lv, const VoteParamsDev& vp, cudaStream_t s, int write_derivs,
                         cudaEvent_t* ev)
{
    const int tiles = total_of(lv, &LevelView::uf_tiles);
    const int hb = (tiles + kHystWarps - 1) / kHystWarps;
    if (write_derivs) {
        k_derivs<<<total_of(lv, &LevelView::dv_tiles), 32 * kDvWarps, 0, s>>>(lv);
        if (tiles <= kNmsFewTiles) k_nms_tiles<false, 4><<<tiles, 128, 0, s>>>(lv, vp);
        else k_nms_tiles<false, 1><<<tiles, 32, 0, s>>>(lv, vp);
    } else {
        if (tiles <= kNmsFewTiles) k_nms_tiles<true, 4><<<tiles, 128, 0, s>>>(lv, vp);
        else k_nms_tiles<true, 1><<<tiles, 32, 0, s>>>(lv, vp);
    }
    mark(ev, kStDerivNms + 1, s);
    k_hyst_unions<<<tiles, 64, 0, s>>>(lv);
    mark(ev, kStHystMerge + 1, s);
    k_hyst_roots<<<(tiles * (kTileComps / 4) + 255) / 256, 256, 0, s>>>(lv, tiles);
    k_hyst_final<<<hb, 32 * kHystWarps, 0, s>>>(lv, tiles);
    mark(ev, kStHystCompress + 1, s);
    const int tt = total_of(lv, &LevelView::thin_tiles);
    k_final_thin<<<(tt + kThinWarps - 1) / kThinWarps, 32 * kThinWarps, 0, s>>>(lv, tt);
    mark(ev, kStFinalThin + 1, s);
    k_row_scan<<<lv.n, 1024, 0, s>>>(lv);
    mark(ev, kStRowScan + 1, s);
    int rows = 0;
    for (int l = 0; l < lv.n; ++l) rows += lv.l[l].H;
    k_emit<<<rows, 128, 0, s>>>(lv, rows);
    mark(ev, kStEmit + 1, s);
}

void launch_image_stage(const Levels& lv, const VoteParamsDev& vp, cudaStream_t s, bool fused_pyramid,
                        cudaEvent_t* ev)
{
    mark(ev, 0, s);
    launch_pyramid(lv, s, fused_pyramid);
    mark(ev, kStPyramid + 1, s);
    launch_edges(lv, vp, s, 1, ev);
    const int G = 148 * 8;
    static const int walkBlocks = [] {
        int per = 0;
        CCTAGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_walk, 32 * kWalkWarps, 0));
        return 148 * (per > 0 ? per : 1);
    }();
    k_walk<<<walkBlocks, 32 * kWalkWarps, 0, s>>>(lv, vp);  // the blocks resident at once
    mark(ev, kStWalk + 1, s);
    k_vote<<<G, 256, 0, s>>>(lv, vp);
    mark(ev, kStVote + 1, s);
    k_vscan_partial<<<dim3(kScanBlocks, lv.n), kScanThreads, 0, s>>>(lv, lv.partial);
    k_vscan_final<<<dim3(kScanBlocks, lv.n), kScanThreads, 0, s>>>(lv, lv.partial);
    mark(ev, kStVoterScan + 1, s);
    k_vfill<<<G, 256, 0, s>>>(lv);
    mark(ev, kStVoterFill + 1, s);
    k_vlists<<<G, 32 * kListWarps, 0, s>>>(lv, vp);
    k_vlists_big<<<148, 256, 0, s>>>(lv, vp);
    mark(ev, kStVoterSort + 1, s);
    CCTAGB_CUDA(cudaGetLastError());
}

void launch_canny_only(const Levels& lv, const VoteParamsDev& vp, cudaStream_t s)
{
    CCTAGB_CUDA(cudaMemsetAsync(lv.cnt, 0, sizeof(LevelCounters) * lv.n, s));
    launch_edges(lv, vp, s, 0, nullptr);
    CCTAGB_CUDA(cudaGetLastError());
}

// Edge bytes of a level's bitmap, four pixels per thread (a word each where the
// rows are word-aligned), and the level's error bits.
__global__ void k_bitmap_to_bytes(Levels lv, uint8_t* out, int32_t* status)
{
    const LevelView& L = lv.l[0];
    const int quads = (L.W + 3) / 4;
    const bool wide = L.W % 4 == 0 && (reinterpret_cast<size_t>(out) & 3) == 0;
    if (status && blockIdx.x == 0 && threadIdx.x == 0) *status = lv.cnt->err;
    const size_t n = size_t(quads) * L.H;
    for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
        const int y = int(i / quads), x = 4 * int(i - size_t(y) * quads);
        const uint32_t b = L.bitmap[size_t(y) * L.WW + (x >> 5)] >> (x & 31);
        // bit k to byte k
        const uint32_t v = ((b & 1u) | (b & 2u) << 7 | (b & 4u) << 14 | (b & 8u) << 21) * 0xffu;
        uint8_t* o = out + size_t(y) * L.W + x;
        if (wide) {
            *reinterpret_cast<uint32_t*>(o) = v;
        } else {
            for (int k = 0; k < 4 && x + k < L.W; ++k) o[k] = uint8_t(v >> (8 * k));
        }
    }
}

__global__ void k_scatter_counters(const LevelCounters* __restrict__ src, CounterTargets t)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < t.n) *t.dst[i] = src[i];
}

void launch_scatter_counters(const LevelCounters* src, const CounterTargets& t, cudaStream_t s)
{
    k_scatter_counters<<<1, kMaxLaunchLevels, 0, s>>>(src, t);
    CCTAGB_CUDA(cudaGetLastError());
}

// Edge stage of one level from its gray image (derivatives, NMS, hysteresis,
// thinning, edge bitmap) without the compaction; lv.l[0].row_count is null.
void launch_edge_level(const Levels& lv, const VoteParamsDev& vp, cudaStream_t s, uint8_t* edges_out,
                       int32_t* status_out)
{
    const LevelView& L = lv.l[0];
    k_derivs<<<L.dv_tiles, 32 * kDvWarps, 0, s>>>(lv);
    const int hb = (L.uf_tiles + kHystWarps - 1) / kHystWarps;
    k_nms_tiles<false, 4><<<L.uf_tiles, 128, 0, s>>>(lv, vp);  // at most 1,281 tiles
    k_hyst_unions<<<L.uf_tiles, 64, 0, s>>>(lv);
    k_hyst_roots<<<(L.uf_tiles * (kTileComps / 4) + 255) / 256, 256, 0, s>>>(lv, L.uf_tiles);
    k_hyst_final<<<hb, 32 * kHystWarps, 0, s>>>(lv, L.uf_tiles);
    k_final_thin<<<(L.thin_tiles + kThinWarps - 1) / kThinWarps, 32 * kThinWarps, 0, s>>>(lv, L.thin_tiles);
    const size_t quads = size_t((L.W + 3) / 4) * L.H;
    k_bitmap_to_bytes<<<int(std::min<size_t>((quads + 255) / 256, 148 * 8)), 256, 0, s>>>(lv, edges_out, status_out);
    CCTAGB_CUDA(cudaGetLastError());
}

}  // namespace cctagb
