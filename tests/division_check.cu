// Host check of the branch-free division of the exact collision (k17.cuh refine_rcp, refine_div):
// counts results that differ from the host's IEEE division, for seeds as far off as the hardware's
// reciprocal approximation may be.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "k17.cuh"

static uint64_t state;
static uint64_t next()
{
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
static double number(uint64_t fraction, int exponent)
{
    const uint64_t bits = (uint64_t)(1023 + exponent) << 52 | (fraction & 0xfffffffffffffull);
    double x;
    std::memcpy(&x, &bits, 8);
    return x;
}
// fractions next to the ends of a binade and random ones
static uint64_t fraction()
{
    const uint64_t r = next(), n = next() % 8;
    return r % 4 == 0 ? n : r % 4 == 1 ? 0xfffffffffffffull - n : r % 4 == 2 ? r >> 12 : (r >> 12) & 0xfffff00000000ull;
}

extern "C" long division_mismatches(long cases, uint64_t seed, int exponents)
{
    state = seed;
    long bad = 0;
    for (long i = 0; i < cases; ++i) {
        const double b = number(fraction(), (int)(next() % (2 * exponents + 1)) - exponents);
        const double a = number(fraction(), (int)(next() % (2 * exponents + 1)) - exponents) * ((next() & 1) ? 1 : -1);
        const double off = 1.0 + ((double)(int64_t)next() * 0x1p-63) * 0x1p-18;
        const double y = (1.0 / b) * off;
        bad += vfb::k17detail::refine_rcp(b, y) != 1.0 / b;
        bad += vfb::k17detail::refine_div(a, b, y) != a / b;
    }
    bad += vfb::k17detail::refine_div(0.0, 0.01, 100.0) != 0.0;
    return bad;
}
