// link_convexity_lost (cand_shared.hpp) against the reference's test in terms
// of the sine and cosine (Vote.cpp:329-344), for differences of two angles in
// [0, 2 pi): every float within 4096 of each end of its intervals, and a sweep
// of the whole range, in both directions.
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "cand_shared.hpp"

using namespace cctagb;

static bool reference(float front, float back, bool full, int dir)
{
    const float s = float(dir) * pm::sinf_(back - front), c = pm::cosf_(back - front);
    return full ? s < 0.0f : (s < -0.707f && c > 0.f) || (s < 0.f && c < 0.f);
}

int main()
{
    long long bad = 0;
    auto check = [&](float d) {
        if (!(std::fabs(d) < 6.28318530f)) return;
        for (int dir = -1; dir <= 1; dir += 2)
            for (int full = 0; full < 2; ++full)
                bad += cand::link_convexity_lost(0.f, d, full, dir) != reference(0.f, d, full, dir);
    };
    const float ends[] = {0.f, 0.785247266f, 1.57079637f, 3.14159274f, 4.71238899f, 5.49793768f, 6.28318501f};
    for (float e : ends)
        for (float sign : {1.f, -1.f}) {
            float up = sign * e, down = sign * e;
            for (int i = 0; i < 4096; ++i) {
                check(up);
                check(down);
                up = std::nextafter(up, 8.f);
                down = std::nextafter(down, -8.f);
            }
        }
    for (int i = -2000000; i <= 2000000; ++i) check(float(i) * 3.1415925e-6f);
    if (bad) std::printf("%lld differences\n", bad);
    return bad ? 1 : 0;
}
