// Host check of the FMA collision's limiters (k17.cuh): the largest difference of the populations of one
// collision from the exact form's, over random states; NaN where a result is not finite.
#include <cmath>
#include <cstdint>
#include <limits>

#include "k17.cuh"

template <class T>
static double largest_difference(double qP, double qM, double qD, int cases)
{
    const auto exact = vfb::make_k17_rates<T>(T(1.9), T(qP), T(qM), T(qD), true);
    const auto fma = vfb::make_k17_rates<T>(T(1.9), T(qP), T(qM), T(qD), false);
    uint64_t h = 0x9E3779B97F4A7C15ull;
    double worst = 0;
    for (int i = 0; i < cases; ++i) {
        T f[27], g[27], m[4];
        for (int d = 0; d < 27; ++d) {
            h ^= h << 13;
            h ^= h >> 7;
            h ^= h << 17;
            f[d] = g[d] = T((double)(int64_t)h * 0x1p-63 * 0.02);
        }
        vfb::collide<T, true>(f, exact, T(0), T(0), T(0), m[0], m[1], m[2], m[3]);
        vfb::collide<T, false>(g, fma, T(0), T(0), T(0), m[0], m[1], m[2], m[3]);
        for (int d = 0; d < 27; ++d) {
            const double off = std::fabs((double)f[d] - (double)g[d]);
            if (!std::isfinite(off))
                return std::numeric_limits<double>::quiet_NaN();
            worst = std::fmax(worst, off);
        }
    }
    return worst;
}

extern "C" double limiter_difference(int real_bytes, double qP, double qM, double qD, int cases)
{
    return real_bytes == 8 ? largest_difference<double>(qP, qM, qD, cases) : largest_difference<float>(qP, qM, qD, cases);
}
