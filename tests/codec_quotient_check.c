/* The encoder's quotient (csrc/codec_fast.cuh) against the defining one: with r0 = RN(1 / u), r1 = RN((1 - u r0) r0) and
 * q = RN(d r0 + RN(d r1)), floor(RN(q + 0.5)) == floor(RN(RN(d / u) + 0.5)) for every d within four ulps of the threshold of a
 * code (and of the first one beyond), for u with every `step`-th mantissa at the middle and at both ends of its range.
 * Prints the number of mismatches; exit status 0 when there are none.  Build: gcc -O2 -march=native -ffp-contract=off. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static inline float u2f(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static inline uint32_t f2u(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }

int main(int argc, char** argv) {
    const uint32_t step = argc > 1 ? (uint32_t)atoi(argv[1]) : 1u;
    const int exponents[3] = {-100, 0, 99};
    unsigned long long bad = 0, cases = 0;
    for (int x = 0; x < 3; ++x)
        for (uint32_t m = 0; m < (1u << 23); m += step) {
            const float u = u2f((uint32_t)(127 + exponents[x]) << 23 | m);
            const float r0 = 1.0f / u, r1 = fmaf(-u, r0, 1.0f) * r0;
            for (int c = 1; c <= 16; ++c) {
                const uint32_t at = f2u((float)(((double)c - 0.5) * (double)u));
                for (int j = -4; j <= 4; ++j, ++cases) {
                    const float d = u2f(at + (uint32_t)j);
                    bad += floorf(fmaf(d, r0, d * r1) + 0.5f) != floorf(d / u + 0.5f);
                }
            }
        }
    printf("quotient mismatches %llu of %llu\n", bad, cases);
    return bad == 0 ? 0 : 1;
}
