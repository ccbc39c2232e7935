// Host check of slm_expf_neg_cr (csrc/fmath_cr.h) against the double function
// rounded to float: every `stride`-th float in (-10.5, 0], and the values where
// the table index changes, one ulp to either side (built and run by
// tests/test_fmath_neg.py).
#include <cstdio>
#include <cstdlib>

#include "fmath_cr.h"

int main(int, char **argv) {
    const unsigned long stride = strtoul(argv[1], nullptr, 10);
    unsigned long bad = 0, n = 0;
    auto check = [&](uint32_t u) {
        const float x = slm_bitsf(u);
        ++n;
        if (slm_fbits(slm_expf_neg_cr(x)) != slm_fbits((float)exp((double)x)) && bad++ < 5) printf("exp(%a)\n", x);
    };
    for (unsigned long u = 0x80000000ul; u <= slm_fbits(-10.5f); u += stride) check((uint32_t)u);
    for (int k = 1; k <= 2 * 640; ++k)  // j / 64 and (j + 1/2) / 64
        for (int d = -1; d <= 1; ++d) check(slm_fbits(-(float)k / 128.0f) + (uint32_t)d);
    check(0u);
    printf("%lu %lu\n", bad, n);
    return bad != 0;
}
