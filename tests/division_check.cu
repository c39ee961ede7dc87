// Checks of the exact collision's division (k17.cuh): counts results that differ from the IEEE division.
// division_mismatches: refine_rcp and refine_div on the host, for seeds as far off as the hardware's
// reciprocal approximation may be; density_mismatches: collisions whose populations differ from those with
// the IEEE 1 / rho, on the host, where rho is 0, infinite or of 2^120 and more; whole_mismatches: rcp_rounded and the limited moments (limited) on the
// host, for any operands; device_mismatches: the same on the device, with the hardware's approximation.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <limits>

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

// Any doubles: bit patterns, numbers with the exponents at the limits of the range, common ones, zeros,
// subnormals, infinities, NaN. The fractions are those of fraction() above; h: a hash per number.
static __host__ __device__ uint64_t hash(uint64_t x)
{
    x = (x ^ x >> 30) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ x >> 27) * 0x94d049bb133111ebull;
    return x ^ x >> 31;
}
static __host__ __device__ uint64_t any_bits(uint64_t h)
{
    const uint64_t r = hash(h + 1), n = hash(h + 2) % 8, k = hash(h + 3) % 8;
    uint64_t f = r % 4 == 0 ? n : r % 4 == 1 ? 0xfffffffffffffull - n : r >> 12;
    int e;                                                     // biased exponent
    switch (k) {
    case 0: return r;
    case 1: e = 183 + (int)(n % 5) - 2; break;                 // 2^-840
    case 2: e = 1143 + (int)(n % 5) - 2; break;                // 2^120
    case 3: e = 1 + (int)(r % 2046); break;
    case 4: e = n < 2 ? 0 : n < 4 ? 2047 : 1 + (int)(r % 2046); f = n % 2 ? f : 0; break;
    default: e = 1023 - 20 + (int)(r >> 7) % 40; break;
    }
    return (hash(h + 4) & 1) << 63 | (uint64_t)e << 52 | f;
}
static __host__ __device__ bool same(double x, double y)
{
    uint64_t a, b;
    memcpy(&a, &x, 8);
    memcpy(&b, &y, 8);
    return a == b || (x != x && y != y);
}
static __host__ __device__ double number_of(uint64_t bits)
{
    double x;
    memcpy(&x, &bits, 8);
    return x;
}
// |x| with its exponent folded into [lo, hi)
static __host__ __device__ double folded(double x, int lo, int hi)
{
    uint64_t b;
    memcpy(&b, &x, 8);
    return number_of((b & 0xfffffffffffffull) | (uint64_t)(1023 + lo + (int)((b >> 52 & 0x7ff) % (unsigned)(hi - lo))) << 52);
}
struct Limits {
    double q[3], O[3], o[3], bound;
};
// limiters and rates of case i; wide: any, else those that the collision divides without a branch with
static __host__ Limits limits_of(uint64_t i, bool wide)
{
    Limits l;
    for (int j = 0; j < 3; ++j) {
        const uint64_t h = hash(i * 6 + j + 0x5151);
        l.q[j] = wide && h % 4 == 0 ? number_of(any_bits(h)) : folded(number_of(any_bits(h)), h % 2 ? -12 : -300, h % 2 ? 12 : 100);
        l.O[j] = h % 16 == 0 ? 0.0 : wide && h % 16 == 1 ? number_of(any_bits(h + 9)) : folded(number_of(any_bits(h + 9)), -20, 3);
        if (h % 3 == 0)
            l.O[j] = -l.O[j];
        l.o[j] = 1.0 - l.O[j];
    }
    l.bound = vfb::k17detail::division_bound(l.q, l.O, l.o);
    return l;
}
// seven limited moments together, as the collision forms them, and one reciprocal; wide: any doubles
static __host__ __device__ int one_case(uint64_t i, bool wide, const Limits &l)
{
    double m[7], want[7], O[7], o[7], q[7];
    for (int j = 0; j < 7; ++j) {
        const uint64_t h = hash(i * 7 + j);
        m[j] = number_of(any_bits(h));
        if (!wide || j != (int)(i % 7)) {
            const double size = folded(m[j], h % 4 ? -60 : -840, h % 4 ? 4 : 120);
            m[j] = h % 64 == 0 ? 0.0 : m[j] < 0 ? -size : size;
        }
        q[j] = l.q[j % 3];
        O[j] = l.O[j % 3];
        o[j] = l.o[j % 3];
        want[j] = m[j] + (O[j] + o[j] * fabs(m[j]) / (fabs(m[j]) + q[j])) * -m[j];
    }
    const double b = wide ? m[i % 7] : folded(m[i % 7], -840, 120) * (hash(i) & 1 ? -1 : 1), r = 1.0 / b;
    vfb::k17detail::limited(m, O, o, q, l.bound);
    int bad = !same(vfb::k17detail::rcp_rounded(b), r);
    for (int j = 0; j < 7; ++j)
        bad += !same(m[j], want[j]);
    return bad;
}
extern "C" long whole_mismatches(long cases, int wide)
{
    long bad = 0;
    for (long i = 0; i < cases; ++i)
        bad += one_case((uint64_t)i, wide != 0, limits_of((uint64_t)i, wide != 0));
    return bad;
}
extern "C" long density_mismatches(long cases)
{
    const auto r = vfb::make_k17_rates<double>(1.9, 0.01, 0.01, 0.01, true);
    long bad = 0;
    for (long i = 0; i < cases; ++i) {
        double f[2][27], out[2][4];
        for (int d = 0; d < 27; ++d)                           // few bits: the sums are exact
            f[0][d] = i % 8 == 0 ? 0.0 : std::ldexp((double)(int)(hash(27 * i + d) % 2048) - 1024, -16);
        if (i % 4 < 2)
            f[0][0] = 0.0;
        const double rest = vfb::density_pyramid(f[0]);
        if (i % 4 < 2)
            f[0][0] = -1.0 - rest;                             // rho = 0
        else if (i % 4 == 2)
            f[0][i / 4 % 27] = i % 3 ? std::numeric_limits<double>::infinity() : -std::numeric_limits<double>::infinity();
        else
            f[0][0] = std::ldexp(i % 3 ? 1.5 + (double)(i % 100) / 256 : -1.0 - (double)(i % 100) / 128, 120 + (int)(i / 4 % 904));
        std::memcpy(f[1], f[0], sizeof f[0]);
        vfb::collide<double, true, false>(f[0], r, 0.0, 0.0, 0.0, out[0][0], out[0][1], out[0][2], out[0][3]);
        vfb::collide<double, true, true>(f[1], r, 0.0, 0.0, 0.0, out[1][0], out[1][1], out[1][2], out[1][3]);
        for (int d = 0; d < 27; ++d)
            bad += !same(f[0][d], f[1][d]);
        bad += !same(out[0][0], out[1][0]);
    }
    return bad;
}
constexpr int kSets = 4096;             // of limiters and rates
__global__ void device_kernel(uint64_t cases, bool wide, const Limits *sets, unsigned long long *bad)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cases; i += (uint64_t)gridDim.x * blockDim.x) {
        const int n = one_case(i, wide, sets[i % kSets]);
        if (n)
            atomicAdd(bad, (unsigned long long)n);
    }
}
// -1: a CUDA call failed
extern "C" long device_mismatches(long cases, int wide)
{
    static Limits host[kSets];
    for (int i = 0; i < kSets; ++i)
        host[i] = limits_of((uint64_t)i, wide != 0);
    Limits *sets = nullptr;
    unsigned long long *bad = nullptr, n = 0;
    cudaError_t e = cudaMalloc(&bad, sizeof n);
    if (e == cudaSuccess)
        e = cudaMalloc(&sets, sizeof host);
    if (e == cudaSuccess)
        e = cudaMemset(bad, 0, sizeof n);
    if (e == cudaSuccess)
        e = cudaMemcpy(sets, host, sizeof host, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        device_kernel<<<1024, 128>>>((uint64_t)cases, wide != 0, sets, bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpy(&n, bad, sizeof n, cudaMemcpyDeviceToHost);
    cudaFree(sets);
    cudaFree(bad);
    return e == cudaSuccess ? (long)n : -1;
}
