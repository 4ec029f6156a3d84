/* Checks that div_recip (smokesim_b200/csrc/k_coarse.cu) returns the bits of
 * IEEE division a / b, y = RN(1/b), for divisors b of the coarse levels (sums
 * of up to six fluid fractions) and dividends in the range its callers use it
 * for, 1e-25 < |a| < 1e25, and for a = +0.  Usage: recip_check [divisors]
 * (2^17 mantissas of a each, signs and exponents varied).  Prints the mismatch
 * count and exits non-zero on any.  Same operations as the device code. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static float div_recip(float a, float b, float y) {
    float q = a * y;
    float r = fmaf(-b, q, a);
    q = fmaf(r, y, q);
    r = fmaf(-b, q, a);
    return fmaf(r, y, q);
}

static uint64_t mix(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

int main(int argc, char** argv) {
    const int divisors = argc > 1 ? atoi(argv[1]) : 256;
    unsigned long long bad = 0, n = 0;
#pragma omp parallel for reduction(+ : bad, n) schedule(dynamic)
    for (int d = 0; d < divisors; ++d) {
        /* the counts, then sums of k fractions 1 - alpha, alpha in half precision in [0.5, 1) or 0 */
        float b = 0.f;
        if (d < 6) b = (float)(d + 1);
        else
            for (int k = 0; k <= (int)(mix(d) % 6); ++k) {
                const uint64_t z = mix(1000ull * d + k);
                b += z & 1 ? 1.f : (float)(1 + (z >> 8) % 1024) / 2048.f;   /* 1 - half in [0.5, 1) */
            }
        const volatile float y = 1.f / b;
        for (uint32_t i = 0; i < (1u << 17); ++i) {
            const uint64_t z = mix(((uint64_t)d << 32) + i);
            const uint32_t e = 127 - 83 + (uint32_t)(z >> 40) % 166;   /* 2^-83 .. 2^82 */
            const uint32_t u = (uint32_t)(z & 0x80000000u) | (e << 23) | ((i << 6) + (uint32_t)(z & 63)) % (1u << 23);
            float a;
            memcpy(&a, &u, 4);
            if (i == 0) a = 0.f;
            if (a != 0.f && !(fabsf(a) > 1e-25f && fabsf(a) < 1e25f)) continue;
            const volatile float ref = a / b;
            const float q = div_recip(a, b, y), rv = ref;
            uint32_t bq, br;
            memcpy(&bq, &q, 4);
            memcpy(&br, &rv, 4);
            ++n;
            if (bq != br) ++bad;
        }
    }
    printf("checked %llu quotients, %llu bit mismatches\n", n, bad);
    return bad ? 1 : 0;
}
