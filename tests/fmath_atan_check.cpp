// Host check of slm_atan2f_cr (csrc/fmath_cr.h) against the double function
// rounded to float: `count` pseudo-random arguments near the table's steps, the
// diagonals and the axes, over many magnitudes, and pairs of special values.
// Built with SLM_FM_RCP_ULP = -1, 0 or 1 ulp added to each reciprocal, which is
// what the device's approximation may be off (tests/test_fmath_atan.py).
#include <cstdio>
#include <cstdlib>

#include "fmath_cr.h"

int main(int, char **argv) {
    const unsigned long count = strtoul(argv[1], nullptr, 10);
    unsigned long bad = 0, n = 0;
    unsigned long long s = 0x9E3779B97F4A7C15ull;
    auto nx = [&]() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
    auto check = [&](float y, float x) {
        const float got = slm_atan2f_cr(y, x), want = (float)atan2((double)y, (double)x);
        ++n;
        if (slm_fbits(got) != slm_fbits(want) && !(got != got && want != want) && bad++ < 5) printf("atan2(%a, %a)\n", y, x);
    };
    const float sp[] = {0.0f, -0.0f, 1.0f, -1.0f, INFINITY, -INFINITY, NAN, 1e-40f, -1e-40f, 1e30f, 1e-30f, 0x1p100f, 0x1p99f, 0x1p-61f};
    for (float y : sp)
        for (float x : sp) check(y, x);
    for (unsigned long i = 0; i < count; ++i) {
        float x = slm_bitsf(0x3f800000u + (uint32_t)(nx() & 0x7fffff)), y;
        switch (nx() & 3) {
            case 0: y = x * ((float)(nx() % 33) / 32.0f); break;                                // a step, or halfway
            case 1: y = x * (float)(nx() % 1000001) * 1e-6f; break;
            case 2: y = x * slm_bitsf(0x20000000u + (uint32_t)(nx() % 0x1f800000u)); break;      // 2^-63 .. 1
            default: x = slm_bitsf((uint32_t)nx()); y = slm_bitsf((uint32_t)nx());
        }
        y = slm_bitsf(slm_fbits(y) + (uint32_t)(nx() % 5) - 2u);
        const uint32_t f = (uint32_t)nx();
        if (f & 4) { const float q = x; x = y; y = q; }
        check((f & 1) ? -y : y, (f & 2) ? -x : x);
    }
    printf("%lu %lu\n", bad, n);
    return bad != 0;
}
