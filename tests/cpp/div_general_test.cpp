// div_small (pmath.hpp) against IEEE float division for divisors of any sign and
// value, as a homography's denominator takes them: random pairs, every dividend
// of a binade for the divisors next to the powers of two and in between (where
// the rounded reciprocal is furthest off), and divisors so small that their
// reciprocal overflows, which never give a finite result.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "cctag_b200/portable/pmath.hpp"

static float from_bits(uint32_t b)
{
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}

int main()
{
    long long bad = 0;
    auto same = [&](float x, float d) {
        volatile float dv = d;
        volatile float ref = x / dv;
        const float y = 1.0f / dv, got = cctagb::pm::div_small(x, d, y);
        if (got != ref && ++bad < 10) std::printf("%a / %a: got %a want %a\n", x, d, got, (float)ref);
    };
    uint64_t s = 1;
    auto next = [&] {  // xorshift64*
        s ^= s >> 12;
        s ^= s << 25;
        s ^= s >> 27;
        return s * 2685821657736338717ull;
    };
    // |x| and |d| in [2^-20, 2^20): quotients and remainders stay normal
    for (int i = 0; i < 40000000; ++i) {
        const uint64_t u = next(), v = next();
        const float x = from_bits(uint32_t(u & 0x807fffffu) | uint32_t(107 + (u >> 32) % 40) << 23);
        const float d = from_bits(uint32_t(v & 0x807fffffu) | uint32_t(107 + (v >> 32) % 40) << 23);
        same(x, d);
    }
    // |x| = 0 and pixel coordinates over denominators of about one
    for (int i = 0; i < 10000000; ++i) {
        const uint64_t u = next();
        const float x = i % 1000 == 0 ? 0.f : float(int32_t(u)) * 0x1p-17f;
        same(x, from_bits(uint32_t(u >> 32 & 0x807fffffu) | uint32_t(126 + (u >> 60) % 3) << 23));
    }
    for (uint32_t m : {0u, 1u, 2u, 3u, 5u, 0x3fffffu, 0x400000u, 0x400001u, 0x555555u, 0x2aaaaau, 0x7ffffau, 0x7ffffbu,
                       0x7ffffcu, 0x7ffffdu, 0x7ffffeu, 0x7fffffu}) {
        const float d = from_bits(0x3f800000u | m);
        for (uint32_t k = 0; k < 1u << 23; ++k) same(from_bits(0x3f800000u | k), d);
    }
    // 1 / d overflows: zero and the denormals below 2^-128
    for (uint32_t b = 0; b < 1u << 21; b += b < 4096 ? 1 : 997)
        for (uint32_t sign : {0u, 0x80000000u})
            for (float x : {0.f, 1.f, -3.5f, 4000.f, 1e-20f}) {
                const float d = from_bits(b | sign);
                volatile float dv = d;
                const float y = 1.0f / dv;
                if (std::isfinite(y)) continue;
                const float got = cctagb::pm::div_small(x, d, y);
                if (std::isfinite(got) && ++bad < 10) std::printf("%a / %a: finite %a\n", x, d, got);
            }
    std::printf("%lld mismatches\n", bad);
    return bad != 0;
}
