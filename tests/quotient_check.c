/* Checks two quotients of the device code against IEEE division, bit for bit.
 *
 * table  the level-0 half-sweeps' (k_rb_smooth4, smokesim_b200/csrc/k_rb.cu): a / f
 *        for a count f in 1..6 by y = RN(1/f) and one residual correction, f = 6 too;
 *        a dividend below 2^-120 and -0 take div_by_count, +0 does not
 * texel  the ray marcher's (texel, k_render.cu): (p / b) * n - 1/2 with div_recip
 *        (common.cuh) for p / b, b = RN(n / m) the side of the box, for grids of up to
 *        4096 cells an axis and every p from +0 to 1e25
 *
 * Usage: quotient_check [stride] (1 = all bit patterns of a, and 64 divisors for
 * every p).  Prints the mismatch count and exits non-zero on any. */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

static float from_bits(uint32_t u) {
    float a;
    memcpy(&a, &u, 4);
    return a;
}
static uint32_t bits(float a) {
    uint32_t u;
    memcpy(&u, &a, 4);
    return u;
}

static float div_by_count(float a, int f) {
    if (f == 6) {
        if (fabsf(a) < 7.52316385e-37f) return a / 6.f;
        a = a * 0.5f;
        f = 3;
    } else if (a == 0.f) {
        return a;
    }
    const float y = f == 1 ? 1.f : f == 2 ? 0.5f : f == 3 ? (1.0f / 3.0f) : f == 4 ? 0.25f : (1.0f / 5.0f);
    const float q0 = a * y;
    const float r = fmaf(-(float)f, q0, a);
    return fmaf(r, y, q0);
}

static float by_table(float a, int f) {
    if (fabsf(a) < 7.52316385e-37f && bits(a) != 0u) return div_by_count(a, f);
    const float y = 1.f / (float)f;
    const float q0 = a * y;
    return fmaf(fmaf(-(float)f, q0, a), y, q0);
}

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
    const long long stride = argc > 1 ? atoll(argv[1]) : 1;
    unsigned long long bad = 0, n = 0;
    const uint32_t special[] = {0x00000000u, 0x80000000u, 0x00000001u, 0x80000001u, 0x007FFFFFu, 0x807FFFFFu, 0x00800000u,
                                0x80800000u, 0x03800000u, 0x837FFFFFu, 0x03800001u, 0x7F7FFFFFu, 0xFF7FFFFFu};
    for (int f = 1; f <= 6; ++f) {
        for (size_t k = 0; k < sizeof special / sizeof special[0]; ++k) {
            volatile float ref = from_bits(special[k]) / (float)f;
            ++n;
            if (bits(by_table(from_bits(special[k]), f)) != bits(ref)) ++bad;
        }
#pragma omp parallel for reduction(+ : bad, n) schedule(static)
        for (long long i = 0; i <= 0xFFFFFFFFLL; i += stride) {
            const float a = from_bits((uint32_t)i);
            if (isnan(a) || isinf(a)) continue;
            volatile float ref = a / (float)f;
            ++n;
            if (bits(by_table(a, f)) != bits(ref)) ++bad;
        }
    }
    const uint32_t top = bits(1e25f);
#pragma omp parallel for reduction(+ : bad, n) schedule(static)
    for (long long i = 0; i <= (long long)top; i += stride) {
        const float p = from_bits((uint32_t)i);
        for (int d = 0; d < 64; ++d) {
            const uint64_t z = mix((uint64_t)i * 64 + d);
            const int m = 3 + (int)(z % 4094), cells = m + (int)((z >> 32) % (uint64_t)(4097 - m));
            const float b = (float)cells / (float)m;
            const volatile float y = 1.f / b;
            volatile float quot = p / b;
            volatile float want = quot * (float)cells;
            volatile float got = div_recip(p, b, y) * (float)cells;
            ++n;
            if (bits(want - 0.5f) != bits(got - 0.5f)) ++bad;
        }
    }
    printf("checked %llu quotients, %llu bit mismatches\n", n, bad);
    return bad ? 1 : 0;
}
