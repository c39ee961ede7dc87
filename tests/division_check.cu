// Checks of the exact collision's division (k17.cuh): counts results that differ from the IEEE division.
// division_mismatches: refine_rcp and refine_div on the host, for seeds as far off as the hardware's
// reciprocal approximation may be; whole_mismatches: rcp_rounded and div_rounded on the host, for any
// operands; device_mismatches: the same on the device, with the hardware's approximation.
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

// Any doubles: bit patterns, numbers with the exponents at the limits of div_in_range, common ones, zeros,
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
// the quotients of seven pairs together, as the collision forms them, and one reciprocal; wide: any
// doubles, else operands within the range without the compiler's division
static __host__ __device__ int one_case(uint64_t i, bool wide)
{
    double a[7], b[7], q[7];
    for (int j = 0; j < 7; ++j) {
        uint64_t x = any_bits(hash(i * 14 + j)), y = any_bits(hash(i * 14 + 7 + j));
        if (!wide || j != (int)(i % 7)) {                      // 183 .. 1142
            x = (x & 0x800fffffffffffffull) | (uint64_t)(183 + (x >> 52 & 0x7ff) % 960) << 52;
            y = (y & 0x800fffffffffffffull) | (uint64_t)(183 + (y >> 52 & 0x7ff) % 960) << 52;
        }
        a[j] = number_of(x);
        b[j] = number_of(y);
        if (!wide && hash(x) % 64 == 0)
            a[j] = 0.0 * a[j];
    }
    vfb::k17detail::div_rounded(a, b, q);
    int bad = 0;
    for (int j = 0; j < 7; ++j)
        bad += !same(q[j], a[j] / b[j]);
    return bad + !same(vfb::k17detail::rcp_rounded(b[i % 7]), 1.0 / b[i % 7]);
}
extern "C" long whole_mismatches(long cases, int wide)
{
    long bad = 0;
    for (long i = 0; i < cases; ++i)
        bad += one_case((uint64_t)i, wide != 0);
    return bad;
}
__global__ void device_kernel(uint64_t cases, bool wide, unsigned long long *bad)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < cases; i += (uint64_t)gridDim.x * blockDim.x) {
        const int n = one_case(i, wide);
        if (n)
            atomicAdd(bad, (unsigned long long)n);
    }
}
// -1: a CUDA call failed
extern "C" long device_mismatches(long cases, int wide)
{
    unsigned long long *bad = nullptr, n = 0;
    if (cudaMalloc(&bad, sizeof n) != cudaSuccess)
        return -1;
    cudaError_t e = cudaMemset(bad, 0, sizeof n);
    device_kernel<<<1024, 128>>>((uint64_t)cases, wide != 0, bad);
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpy(&n, bad, sizeof n, cudaMemcpyDeviceToHost);
    cudaFree(bad);
    return e == cudaSuccess ? (long)n : -1;
}
