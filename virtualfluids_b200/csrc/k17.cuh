// K17 cumulant collision of one D3Q27 node, register resident.
//
// Algorithm: src/lbm/collision/K17CompressibleNavierStokes.h:88-591 (TurbulenceModel::None),
// with the chimera transforms of src/lbm/ChimeraTransformation.h:58-121 and the pyramid
// macroscopic sums of src/lbm/MacroscopicQuantities.h:55-137. The floating-point expression
// trees are kept as in the reference so that a build without FMA contraction (-fmad=false)
// reproduces the reference's host arithmetic bit for bit; the default build contracts
// products into FMAs.
//
// Differences in *work*, not in results:
//  * the omega-only rates (five rational functions and 1/omega - 1/2) are computed once on the
//    host and passed in (K17Rates);
//  * with the relaxation rates O4 = O5 = O6 = 1 that the reference hard-codes, the pre-collision
//    4th, 5th and 6th order cumulants are multiplied by zero (4th) or relaxed to exactly zero
//    (5th, 6th), so they are not computed here; for finite inputs this changes no value.
#pragma once
#include <cmath>

#include "lattice.cuh"

namespace vfb {

template <class T>
struct K17Rates {
    T omega;
    T OxyyPxzz, OxyyMxzz, Oxyz; // 3rd order rates (K17...h:251-255)
    T factorA, factorB;         // 4th order diffusion parameters (K17...h:272-273)
    T neg_iwm;                  // -(1/omega - 1/2)
    T qP, qM, qD;               // quadric limiters (Parameter.cpp:69 default 0.01); FMA form: at most 2^100
    // omega-only subexpressions of the collision, each rounded as the reference rounds it in place
    T mhw;                      // 1/2 * (-omega) (exact)
    T w32;                      // omega * 3/2
    T m3w;                      // -3 * omega
    T c3a;                      // 3 * (1 + 1/2 * (-omega))
    T omOxyz, omOP, omOM;       // 1 - Oxyz, 1 - OxyyPxzz, 1 - OxyyMxzz
    // folded constants of the FMA form (k17_collide_fast)
    T omo;                      // 1 - omega
    T mc3h;                     // -3 (1 - omega / 2)
    T hP, hM, cD;               // 1/2 (1 - OxyyPxzz) qP, 1/2 (1 - OxyyMxzz) qM, (1 - Oxyz) qD
    T kA, kB;                   // neg_iwm 2/3 factorA, neg_iwm 1/3 factorB (-3 omega)
    T divBound;                 // the exact form's division without a branch (limited)
};

namespace k17detail {
// The bound of |m| + q below which limited() divides without a branch: 2^120 where the limiters q and the
// rates O and o = 1 - O are ordinary, else 0.
inline double division_bound(const double (&q)[3], const double (&O)[3], const double (&o)[3])
{
    bool fine = true;
    for (int i = 0; i < 3; ++i)
        fine = fine && q[i] >= 0x1p-300 && q[i] <= 0x1p100 && (o[i] == 0 || (std::fabs(o[i]) >= 0x1p-50 && std::fabs(o[i]) <= 0x1p50))
            && (O[i] == 0 || std::fabs(O[i]) >= 0x1p-100);
    return fine ? 0x1p120 : 0.0;
}
inline float division_bound(const float (&)[3], const float (&)[3], const float (&)[3]) { return 0.0f; }
} // namespace k17detail

// host computation of the omega-only rates, expression for expression as the reference. The FMA form takes
// limiters of at most 2^100: beside that |m| is rounded away (the limiter is off), and 1 / (|m| + q) stays
// normal and the product of seven denominators in a double finite.
template <class T>
inline K17Rates<T> make_k17_rates(T omega, T qP, T qM, T qD, bool exact)
{
    const T most = T(0x1p100);
    if (!exact) {
        qP = qP > most ? most : qP;
        qM = qM > most ? most : qM;
        qD = qD > most ? most : qD;
    }
    K17Rates<T> r;
    const T w = omega;
    r.omega = w;
    r.OxyyPxzz = T(8) * (T(-2) + w) * (T(1) + T(2) * w) / (T(-8) - T(14) * w + T(7) * w * w);
    r.OxyyMxzz = T(8) * (T(-2) + w) * (T(-7) + T(4) * w) / (T(56) - T(50) * w + T(9) * w * w);
    r.Oxyz = T(24) * (T(-2) + w) * (T(-2) - T(7) * w + T(3) * w * w) / (T(48) + T(152) * w - T(130) * w * w + T(29) * w * w * w);
    r.factorA = (T(4) + T(2) * w - T(3) * w * w) / (T(2) - T(7) * w + T(5) * w * w);
    r.factorB = (T(4) + T(28) * w - T(14) * w * w) / (T(6) - T(21) * w + T(15) * w * w);
    r.neg_iwm = -(T(1) / w - T(0.5));
    r.qP = qP;
    r.qM = qM;
    r.qD = qD;
    r.mhw = T(0.5) * (-w);
    r.w32 = w * (T(3) / T(2));
    r.m3w = -T(3) * w;
    r.c3a = T(3) * (T(1) + T(0.5) * (-w));
    r.omOxyz = T(1) - r.Oxyz;
    r.omOP = T(1) - r.OxyyPxzz;
    r.omOM = T(1) - r.OxyyMxzz;
    r.divBound = k17detail::division_bound({ qP, qM, qD }, { r.OxyyPxzz, r.OxyyMxzz, r.Oxyz }, { r.omOP, r.omOM, r.omOxyz });
    r.omo = T(1) - w;
    r.mc3h = T(-3) * (T(1) - T(0.5) * w);
    r.hP = T(0.5) * r.omOP * qP;
    r.hM = T(0.5) * r.omOM * qM;
    r.cD = r.omOxyz * qD;
    r.kA = r.neg_iwm * (T(2) / T(3)) * r.factorA;
    r.kB = r.neg_iwm * (T(1) / T(3)) * r.factorB * r.m3w;
    return r;
}

namespace k17detail {

template <class T>
__host__ __device__ __forceinline__ void fwd_k(T &a, T &b, T &c, T v, T v2, T kinv, T k)
{
    const T s2 = a + c;
    const T s1 = c - a;
    T s0 = s2 + b;
    a = s0;
    s0 *= kinv;
    s0 += T(1);
    b = (s1 * kinv - s0 * v) * k;
    c = ((s2 - T(2) * s1 * v) * kinv + v2 * s0) * k;
}
template <class T>
__host__ __device__ __forceinline__ void bwd_k(T &a, T &b, T &c, T v, T v2, T kinv, T k)
{
    const T h = T(0.5);
    const T r0 = (((c - b) * h + b * v) * kinv + (a * kinv + T(1)) * (v2 - v) * h) * k;
    const T r1 = (((a - c) - T(2) * b * v) * kinv + (a * kinv + T(1)) * (-v2)) * k;
    c = (((c + b) * h + b * v) * kinv + (a * kinv + T(1)) * (v2 + v) * h) * k;
    a = r0;
    b = r1;
}
template <class T>
__host__ __device__ __forceinline__ void fwd(T &a, T &b, T &c, T v, T v2)
{
    const T s1 = (a + c) + b;
    const T s2 = c - a;
    c = (c + a) + (v2 * s1 - T(2) * v * s2);
    b = s2 - v * s1;
    a = s1;
}
template <class T>
__host__ __device__ __forceinline__ void bwd(T &a, T &b, T &c, T v, T v2)
{
    const T h = T(0.5);
    const T ra = (c + a * (v2 - v)) * h + b * (v - h);
    const T rb = ((a - c) - a * v2) - T(2) * b * v;
    c = (c + a * (v2 + v)) * h + b * (v + h);
    b = rb;
    a = ra;
}

// The transforms of the exact collision. They round exactly as fwd_k / bwd_k / bwd above, with
// fewer operations:
//  * 2 s v is formed as s (2 v), 2 v once per axis: (2 s) v and s (2 v) are the same real number,
//    rounded once;
//  * X (v^2 -+ v) 1/2 is formed as X ((v^2 -+ v) 1/2), the halved factor once per axis: halving is
//    exact, so both round X (v^2 -+ v) / 2 once. This holds for every operand whose products stay
//    out of the subnormal range (|X (v^2 -+ v)| >= 2^-1021 or zero); a velocity component of a
//    state made of finite populations of magnitude above 1e-300 never comes near it;
//  * x h + y (h = 1/2) is one fma(x, h, y): the product is exact, so the fused operation rounds
//    once where the reference rounds the exact product and then the sum.
template <class T>
__host__ __device__ __forceinline__ void fwd_kx(T &a, T &b, T &c, T v, T v2, T twov, T kinv, T k)
{
    const T s2 = a + c;
    const T s1 = c - a;
    T s0 = s2 + b;
    a = s0;
    s0 *= kinv;
    s0 += T(1);
    b = (s1 * kinv - s0 * v) * k;
    c = ((s2 - s1 * twov) * kinv + v2 * s0) * k;
}
template <class T>
__host__ __device__ __forceinline__ void bwd_kx(T &a, T &b, T &c, T v, T v2, T twov, T v2mv_h, T v2pv_h, T kinv, T k)
{
    const T h = T(0.5);
    const T a1 = a * kinv + T(1);
    const T bv = b * v;
    const T r0 = (fma(c - b, h, bv) * kinv + a1 * v2mv_h) * k;
    const T r1 = (((a - c) - b * twov) * kinv + a1 * (-v2)) * k;
    c = (fma(c + b, h, bv) * kinv + a1 * v2pv_h) * k;
    a = r0;
    b = r1;
}
template <class T>
__host__ __device__ __forceinline__ void bwdx(T &a, T &b, T &c, T v, T v2, T twov)
{
    const T h = T(0.5);
    const T ra = fma(c + a * (v2 - v), h, b * (v - h));
    const T rb = ((a - c) - a * v2) - b * twov;
    c = fma(c + a * (v2 + v), h, b * (v + h));
    b = rb;
    a = ra;
}

// chimera constants, as the reference writes them (c36o1, c1o36, c9o4, c4o9, ...)
template <class T> __host__ __device__ __forceinline__ T kinv_z(int a, int b)
{
    return (a != 1 && b != 1) ? T(36) : (a == 1 && b == 1) ? T(9) / T(4) : T(9);
}
template <class T> __host__ __device__ __forceinline__ T k_z(int a, int b)
{
    return (a != 1 && b != 1) ? T(1) / T(36) : (a == 1 && b == 1) ? T(4) / T(9) : T(1) / T(9);
}
template <class T> __host__ __device__ __forceinline__ T kinv_y(int a, int c)
{
    return a != 1 ? (c == 0 ? T(6) : T(18)) : (c == 0 ? T(3) / T(2) : T(9) / T(2));
}
template <class T> __host__ __device__ __forceinline__ T k_y(int a, int c)
{
    return a != 1 ? (c == 0 ? T(1) / T(6) : T(1) / T(18)) : (c == 0 ? T(2) / T(3) : T(2) / T(9));
}

// Correctly rounded 1 / b and a / b in double. Within the range below without a branch. Method:
// Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34 (1990); Cornea, Harrison, Tang, "Scientific Computing on Itanium-based Systems" (2002), ch. 8:
//  * y1 is within one unit in the last place of 1 / b: the hardware's approximation refined by one
//    cubic step (its error, below 2^-18, to the third power is far below the rounding of y1);
//  * then y2 = y1 + y1 (1 - b y1), one rounding, is the rounded reciprocal, except where b's 52
//    fraction bits are all ones: y2 may be a power of two there, and the rounded reciprocal is
//    the next double (its last bit set);
//  * with y2 the rounded reciprocal, q1 = q0 - y2 (b q0 - a), one rounding, is the rounded quotient
//    (the remainder is exact; in this sign a zero keeps that of the quotient).
// It holds for |b| in [2^-840, 2^120) and, with it, |a| in [2^-890, 2^170) or zero (b > 0 then): the
// quotient is normal, and the remainder, a multiple of 2^-106 |a|, above the smallest double.
__host__ __device__ __forceinline__ double refine_rcp(double b, double y)
{
    const double e = ::fma(-b, y, 1.0);
    y = ::fma(y, ::fma(e, e, e), y);
    y = ::fma(y, ::fma(-b, y, 1.0), y);
#ifdef __CUDA_ARCH__
    const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
    return __hiloint2double(__double2hiint(y), __double2loint(y) | ((lo & (hi | 0xfff00000u)) == 0xffffffffu ? 1 : 0));
#else
    uint64_t bits, r;
    __builtin_memcpy(&bits, &b, 8);
    __builtin_memcpy(&r, &y, 8);
    r |= (~bits & 0xfffffffffffffull) == 0 ? 1 : 0;
    __builtin_memcpy(&y, &r, 8);
    return y;
#endif
}
__host__ __device__ __forceinline__ double refine_div(double a, double b, double y)
{
    y = refine_rcp(b, y);
    const double q = a * y;
    return ::fma(-::fma(b, q, -a), y, q);
}

__host__ __device__ __forceinline__ unsigned upper_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    uint64_t bits;
    __builtin_memcpy(&bits, &x, 8);
    return (unsigned)(bits >> 32);
#endif
}
// an approximation of 1 / b: the hardware's, on the host one of 20 bits
__host__ __device__ __forceinline__ double rcp_seed(double b)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
#else
    double y = 1.0 / b;
    uint64_t bits;
    __builtin_memcpy(&bits, &y, 8);
    bits &= ~0xffffffffull;
    __builtin_memcpy(&y, &bits, 8);
    return y;
#endif
}

// 1 / b for any b
__host__ __device__ __forceinline__ double rcp_rounded(double b)
{
    const bool fine = (upper_word(b) & 0x7fffffffu) - ((1023u - 840u) << 20) < (960u << 20);
    return fine ? refine_rcp(b, rcp_seed(b)) : 1.0 / b;
}
__host__ __device__ __forceinline__ float rcp_rounded(float b) { return 1.0f / b; }
// 1 / rho of the collision, without a branch (rho = 1 + drho is 0 or at least 2^-53 away from it). It is NaN
// for a rho of 0 or infinity and 0 about 2^1022 and above; with the IEEE reciprocals there, too, all 27
// populations come out NaN. The branch of rcp_rounded, on which all that follows waits, costs 1.6 % of the
// exact collision: it is taken where the velocity is an output.
__host__ __device__ __forceinline__ double rcp_density(double rho) { return refine_rcp(rho, rcp_seed(rho)); }
__host__ __device__ __forceinline__ float rcp_density(float rho) { return 1.0f / rho; }

// The third order moments m, limited: m + (O + o |m| / (|m| + q)) (-m), the IEEE quotients. One test for
// all of them sends any operand out of the range of refine_div to the compiler's division: |m| + q at
// the bound, infinite or NaN, or 0 < |m| < 2^-840 (a limiter of 1e40, a moment of 1e-260). An |m| below
// 2^-1042 counts as zero in it, which changes nothing: its quotient, below 2^-690, vanishes beside O,
// or, where O is 0, beside 1 in m's own product.
// The compiler's division has such a branch in each of the seven, between which no arithmetic moves: four
// exact FP64 steps of 256^3 took 6.90 ms with it and 6.63 ms with no branch at all. This one costs 0.8 %.
template <int N>
__host__ __device__ __forceinline__ void limited(double (&m)[N], const double (&O)[N], const double (&o)[N],
                                                 const double (&q)[N], double bound)
{
    bool fine = true;
    double w[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
        fine &= (upper_word(fabs(m[i]) + q[i]) < upper_word(bound)) & (2u * upper_word(m[i]) - 2u >= 2u * ((1023u - 840u) << 20) - 2u);
    if (fine) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            w[i] = refine_div(o[i] * fabs(m[i]), fabs(m[i]) + q[i], rcp_seed(fabs(m[i]) + q[i]));
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            w[i] = o[i] * fabs(m[i]) / (fabs(m[i]) + q[i]);
    }
#pragma unroll
    for (int i = 0; i < N; ++i)
        m[i] += (O[i] + w[i]) * (-m[i]);
}
template <int N>
__host__ __device__ __forceinline__ void limited(float (&m)[N], const float (&O)[N], const float (&o)[N],
                                                 const float (&q)[N], float)
{
#pragma unroll
    for (int i = 0; i < N; ++i)
        m[i] += (O[i] + o[i] * fabsf(m[i]) / (fabsf(m[i]) + q[i])) * (-m[i]);
}

} // namespace k17detail

// pyramid density (MacroscopicQuantities.h:55), f in direction order
template <class T>
__host__ __device__ __forceinline__ T density_pyramid(const T *f)
{
    const T corners = ((f[19] + f[26]) + (f[24] + f[21])) + ((f[20] + f[25]) + (f[22] + f[23]));
    const T edges = (((f[18] + f[17]) + (f[16] + f[15])) + ((f[14] + f[13]) + (f[12] + f[11]))) + ((f[10] + f[9]) + (f[8] + f[7]));
    const T faces = ((f[2] + f[1]) + (f[4] + f[3])) + (f[6] + f[5]);
    return ((corners + edges) + f[0]) + faces;
}
template <class T>
__host__ __device__ __forceinline__ T momentum_x(const T *f)
{
    return ((((f[19] - f[26]) + (f[21] - f[24])) + ((f[25] - f[20]) + (f[23] - f[22])))
          + (((f[13] - f[14]) + (f[11] - f[12])) + ((f[9] - f[10]) + (f[7] - f[8]))))
          + (f[1] - f[2]);
}
template <class T>
__host__ __device__ __forceinline__ T momentum_y(const T *f)
{
    return ((((f[19] - f[26]) + (f[24] - f[21])) + ((f[20] - f[25]) + (f[23] - f[22])))
          + (((f[17] - f[18]) + (f[15] - f[16])) + ((f[10] - f[9]) + (f[7] - f[8]))))
          + (f[3] - f[4]);
}
template <class T>
__host__ __device__ __forceinline__ T momentum_z(const T *f)
{
    return ((((f[19] - f[26]) + (f[21] - f[24])) + ((f[20] - f[25]) + (f[22] - f[23])))
          + (((f[18] - f[17]) + (f[15] - f[16])) + ((f[14] - f[13]) + (f[11] - f[12]))))
          + (f[5] - f[6]);
}

// In place on f[27] (direction order). fx, fy, fz: half the acceleration, already scaled.
// Returns drho and the velocity including the half force (MacroscopicValues); VELOCITY: the caller keeps it.
template <class T, bool EXACT, bool VELOCITY = false>
__host__ __device__ __forceinline__ void k17_collide(T *f, const K17Rates<T> &r, T fx, T fy, T fz, T &drho_out, T &vx_out,
                                            T &vy_out, T &vz_out)
{
    using namespace k17detail;
    const T drho = density_pyramid(f);
    const T oneOverRho = VELOCITY ? rcp_rounded(drho + T(1)) : rcp_density(drho + T(1));
    T vx = momentum_x(f) * oneOverRho;
    T vy = momentum_y(f) * oneOverRho;
    T vz = momentum_z(f) * oneOverRho;
    vx += fx;
    vy += fy;
    vz += fz;
    const T vx2 = vx * vx, vy2 = vy * vy, vz2 = vz * vz;
    const T twovx = T(2) * vx, twovy = T(2) * vy, twovz = T(2) * vz;

    T m[27];
#pragma unroll
    for (int d = 0; d < 27; ++d)
        m[m3(d)] = f[d];
#define M(a, b, c) m[(a) * 9 + (b) * 3 + (c)]

#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            fwd_kx(M(a, b, 0), M(a, b, 1), M(a, b, 2), vz, vz2, twovz, kinv_z<T>(a, b), k_z<T>(a, b));
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; c += 1) {
            if (c == 1)
                fwd(M(a, 0, 1), M(a, 1, 1), M(a, 2, 1), vy, vy2);
            else
                fwd_kx(M(a, 0, c), M(a, 1, c), M(a, 2, c), vy, vy2, twovy, kinv_y<T>(a, c), k_y<T>(a, c));
        }
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (b == 0 && c == 0)
                fwd_kx(M(0, 0, 0), M(1, 0, 0), M(2, 0, 0), vx, vx2, twovx, T(1), T(1));
            else if (b == 2 && c == 2) // K17...h:222: K^-1 = 3, K = 1/9 on this line
                fwd_kx(M(0, 2, 2), M(1, 2, 2), M(2, 2, 2), vx, vx2, twovx, T(3), T(1) / T(9));
            else if ((b == 2 && c == 0) || (b == 0 && c == 2))
                fwd_kx(M(0, b, c), M(1, b, c), M(2, b, c), vx, vx2, twovx, T(3), T(1) / T(3));
            else
                fwd(M(0, b, c), M(1, b, c), M(2, b, c), vx, vx2);
        }

    const T c13 = T(1) / T(3), c19 = T(1) / T(9), c23 = T(2) / T(3), c127 = T(1) / T(27), h = T(0.5);
    const T omega = r.omega;

    // second and third order linear combinations (K17...h:323-335)
    T mxxPyyPzz = M(2, 0, 0) + M(0, 2, 0) + M(0, 0, 2);
    T mxxMyy = M(2, 0, 0) - M(0, 2, 0);
    T mxxMzz = M(2, 0, 0) - M(0, 0, 2);
    T mxxyPyzz = M(2, 1, 0) + M(0, 1, 2);
    T mxxyMyzz = M(2, 1, 0) - M(0, 1, 2);
    T mxxzPyyz = M(2, 0, 1) + M(0, 2, 1);
    T mxxzMyyz = M(2, 0, 1) - M(0, 2, 1);
    T mxyyPxzz = M(1, 2, 0) + M(1, 0, 2);
    T mxyyMxzz = M(1, 2, 0) - M(1, 0, 2);

    // velocity gradients times rho (K17...h:347-352), OxxPyyPzz = 1
    // (the omega-only factors -3 omega, 1/2 (-omega), omega 3/2 come rounded from the host)
    const T Dxy = r.m3w * M(1, 1, 0);
    const T Dxz = r.m3w * M(1, 0, 1);
    const T Dyz = r.m3w * M(0, 1, 1);
    const T dxux = fma(M(0, 0, 0) - mxxPyyPzz, h, r.mhw * (mxxMyy + mxxMzz));
    const T dyuy = dxux + r.w32 * mxxMyy;
    const T dzuz = dxux + r.w32 * mxxMzz;

    // second order relaxation with correction (K17...h:375-387)
    mxxPyyPzz += T(1) * (M(0, 0, 0) - mxxPyyPzz) - T(3) * (T(1) - h * T(1)) * (vx2 * dxux + vy2 * dyuy + vz2 * dzuz);
    mxxMyy += omega * (-mxxMyy) - r.c3a * (vx2 * dxux - vy2 * dyuy);
    mxxMzz += omega * (-mxxMzz) - r.c3a * (vx2 * dxux - vz2 * dzuz);
    M(0, 1, 1) += omega * (-M(0, 1, 1));
    M(1, 0, 1) += omega * (-M(1, 0, 1));
    M(1, 1, 0) += omega * (-M(1, 1, 0));

    // third order with the quartic limiter (K17...h:397-410)
    T third[7] = { M(1, 1, 1), mxxyPyzz, mxxyMyzz, mxxzPyyz, mxxzMyyz, mxyyPxzz, mxyyMxzz };
    const T O[7] = { r.Oxyz, r.OxyyPxzz, r.OxyyMxzz, r.OxyyPxzz, r.OxyyMxzz, r.OxyyPxzz, r.OxyyMxzz };
    const T o[7] = { r.omOxyz, r.omOP, r.omOM, r.omOP, r.omOM, r.omOP, r.omOM };
    const T q[7] = { r.qD, r.qP, r.qM, r.qP, r.qM, r.qP, r.qM };
    limited(third, O, o, q, r.divBound);
    M(1, 1, 1) = third[0];
    mxxyPyzz = third[1];
    mxxyMyzz = third[2];
    mxxzPyyz = third[3];
    mxxzMyyz = third[4];
    mxyyPxzz = third[5];
    mxyyMxzz = third[6];

    // back from the linear combinations (K17...h:424-433)
    M(2, 0, 0) = c13 * (mxxMyy + mxxMzz + mxxPyyPzz);
    M(0, 2, 0) = c13 * (fma(T(-2), mxxMyy, mxxMzz) + mxxPyyPzz);
    M(0, 0, 2) = c13 * (fma(T(-2), mxxMzz, mxxMyy) + mxxPyyPzz);
    M(2, 1, 0) = (mxxyMyzz + mxxyPyzz) * h;
    M(0, 1, 2) = (-mxxyMyzz + mxxyPyzz) * h;
    M(2, 0, 1) = (mxxzMyyz + mxxzPyyz) * h;
    M(0, 2, 1) = (-mxxzMyyz + mxxzPyyz) * h;
    M(1, 2, 0) = (mxyyMxzz + mxyyPxzz) * h;
    M(1, 0, 2) = (-mxyyMxzz + mxyyPxzz) * h;

    // post-collision 4th order cumulants: modified equilibrium (K17...h:443-448)
    const T cm022 = r.neg_iwm * (dyuy + dzuz) * c23 * r.factorA;
    const T cm202 = r.neg_iwm * (dxux + dzuz) * c23 * r.factorA;
    const T cm220 = r.neg_iwm * (dyuy + dxux) * c23 * r.factorA;
    const T cm112 = r.neg_iwm * Dxy * c13 * r.factorB;
    const T cm121 = r.neg_iwm * Dxz * c13 * r.factorB;
    const T cm211 = r.neg_iwm * Dyz * c13 * r.factorB;
    // 5th and 6th order post-collision cumulants are zero
    const T z = T(0);

    // central moments from post-collision cumulants (K17...h:469-505)
    M(2, 1, 1) = cm211 + c13 * ((T(3) * M(2, 0, 0) + T(1)) * M(0, 1, 1) + T(6) * M(1, 1, 0) * M(1, 0, 1)) * oneOverRho;
    M(1, 2, 1) = cm121 + c13 * ((T(3) * M(0, 2, 0) + T(1)) * M(1, 0, 1) + T(6) * M(1, 1, 0) * M(0, 1, 1)) * oneOverRho;
    M(1, 1, 2) = cm112 + c13 * ((T(3) * M(0, 0, 2) + T(1)) * M(1, 1, 0) + T(6) * M(1, 0, 1) * M(0, 1, 1)) * oneOverRho;
    // products with a power of two are exact: (2 m) m = 2 (m m), and a sum with it is one fma
    const T sq110 = M(1, 1, 0) * M(1, 1, 0), sq101 = M(1, 0, 1) * M(1, 0, 1), sq011 = M(0, 1, 1) * M(0, 1, 1);
    M(2, 2, 0) = cm220 + ((fma(T(2), sq110, M(2, 0, 0) * M(0, 2, 0)) * T(9) + T(3) * (M(2, 0, 0) + M(0, 2, 0))) * oneOverRho - (drho * oneOverRho)) * c19;
    M(2, 0, 2) = cm202 + ((fma(T(2), sq101, M(2, 0, 0) * M(0, 0, 2)) * T(9) + T(3) * (M(2, 0, 0) + M(0, 0, 2))) * oneOverRho - (drho * oneOverRho)) * c19;
    M(0, 2, 2) = cm022 + ((fma(T(2), sq011, M(0, 0, 2) * M(0, 2, 0)) * T(9) + T(3) * (M(0, 0, 2) + M(0, 2, 0))) * oneOverRho - (drho * oneOverRho)) * c19;

    const T t122 = c13 * (T(3) * fma(T(2), M(1, 0, 1) * M(0, 2, 1) + M(1, 1, 0) * M(0, 1, 2), fma(T(4), M(0, 1, 1) * M(1, 1, 1), M(0, 0, 2) * M(1, 2, 0) + M(0, 2, 0) * M(1, 0, 2))) + (M(1, 2, 0) + M(1, 0, 2))) * oneOverRho;
    const T t212 = c13 * (T(3) * fma(T(2), M(0, 1, 1) * M(2, 0, 1) + M(1, 1, 0) * M(1, 0, 2), fma(T(4), M(1, 0, 1) * M(1, 1, 1), M(0, 0, 2) * M(2, 1, 0) + M(2, 0, 0) * M(0, 1, 2))) + (M(2, 1, 0) + M(0, 1, 2))) * oneOverRho;
    const T t221 = c13 * (T(3) * fma(T(2), M(1, 0, 1) * M(1, 2, 0) + M(0, 1, 1) * M(2, 1, 0), fma(T(4), M(1, 1, 0) * M(1, 1, 1), M(2, 0, 0) * M(0, 2, 1) + M(0, 2, 0) * M(2, 0, 1))) + (M(0, 2, 1) + M(2, 0, 1))) * oneOverRho;
    M(1, 2, 2) = EXACT ? z + t122 : t122;
    M(2, 1, 2) = EXACT ? z + t212 : t212;
    M(2, 2, 1) = EXACT ? z + t221 : t221;

    const T b222 = fma(T(-2), M(1, 2, 0) * M(1, 0, 2) + M(2, 1, 0) * M(0, 1, 2) + M(2, 0, 1) * M(0, 2, 1),
                       fma(T(-4), M(0, 1, 1) * M(2, 1, 1) + M(1, 0, 1) * M(1, 2, 1) + M(1, 1, 0) * M(1, 1, 2),
                           fma(T(-4), M(1, 1, 1) * M(1, 1, 1), -(M(2, 0, 0) * M(0, 2, 2) + M(0, 2, 0) * M(2, 0, 2) + M(0, 0, 2) * M(2, 2, 0))))) * oneOverRho
                 + fma(T(16), M(1, 1, 0) * M(1, 0, 1) * M(0, 1, 1),
                       fma(T(4), sq101 * M(0, 2, 0) + sq011 * M(2, 0, 0) + sq110 * M(0, 0, 2),
                           T(2) * (M(2, 0, 0) * M(0, 2, 0) * M(0, 0, 2)))) * oneOverRho * oneOverRho
                 - c13 * (M(0, 2, 2) + M(2, 0, 2) + M(2, 2, 0)) * oneOverRho - c19 * (M(2, 0, 0) + M(0, 2, 0) + M(0, 0, 2)) * oneOverRho
                 + (fma(T(2), sq101 + sq011 + sq110, M(0, 0, 2) * M(0, 2, 0) + M(0, 0, 2) * M(2, 0, 0) + M(0, 2, 0) * M(2, 0, 0))
                    + c13 * (M(0, 0, 2) + M(0, 2, 0) + M(2, 0, 0))) * oneOverRho * oneOverRho * c23
                 + c127 * ((drho * drho - drho) * oneOverRho * oneOverRho);
    M(2, 2, 2) = EXACT ? z - b222 : -b222;

    // first moments change sign (K17...h:512-514)
    M(1, 0, 0) = -M(1, 0, 0);
    M(0, 1, 0) = -M(0, 1, 0);
    M(0, 0, 1) = -M(0, 0, 1);

    const T x2mvh = (vx2 - vx) * h, x2pvh = (vx2 + vx) * h, y2mvh = (vy2 - vy) * h, y2pvh = (vy2 + vy) * h;
    const T z2mvh = (vz2 - vz) * h, z2pvh = (vz2 + vz) * h;

#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (b == 0 && c == 0)
                bwd_kx(M(0, 0, 0), M(1, 0, 0), M(2, 0, 0), vx, vx2, twovx, x2mvh, x2pvh, T(1), T(1));
            else if (b == 2 && c == 2)
                bwd_kx(M(0, 2, 2), M(1, 2, 2), M(2, 2, 2), vx, vx2, twovx, x2mvh, x2pvh, T(9), T(1) / T(9));
            else if ((b == 2 && c == 0) || (b == 0 && c == 2))
                bwd_kx(M(0, b, c), M(1, b, c), M(2, b, c), vx, vx2, twovx, x2mvh, x2pvh, T(3), T(1) / T(3));
            else
                bwdx(M(0, b, c), M(1, b, c), M(2, b, c), vx, vx2, twovx);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (c == 1)
                bwdx(M(a, 0, 1), M(a, 1, 1), M(a, 2, 1), vy, vy2, twovy);
            else
                bwd_kx(M(a, 0, c), M(a, 1, c), M(a, 2, c), vy, vy2, twovy, y2mvh, y2pvh, kinv_y<T>(a, c), k_y<T>(a, c));
        }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            bwd_kx(M(a, b, 0), M(a, b, 1), M(a, b, 2), vz, vz2, twovz, z2mvh, z2pvh, kinv_z<T>(a, b), k_z<T>(a, b));
#undef M

#pragma unroll
    for (int d = 0; d < 27; ++d)
        f[d] = m[m3(d)];
    drho_out = drho;
    vx_out = vx;
    vy_out = vy;
    vz_out = vz;
}

// ---------------------------------------------------------------------------------------------
// The same collision, rearranged for fewer floating-point instructions (the FMA variant): 495
// operations and eight reciprocals per node. Mathematically identical to k17_collide, rounded
// differently:
//  * the populations are summed to raw moments (three additions per line, no velocity), which hold
//    density and momentum; only the moments up to third order are shifted to the velocity, with
//    the shifts of lower moments shared (j' = j - rho u, p = m_ab - u_b j_a). A transform line by
//    line, velocity in every line, took 100 operations more;
//  * a limited rate O + (1 - O) |m| / (|m| + q) leaves m (1 - O) q / (|m| + q) of its moment;
//  * with M = m + 1/3 for the second moments, c_s^2 terms and products of the post-collision
//    moments group to M m (e.g. 3 (xx y + 2 ..) + y = 3 ((xx + 1/3) y + ..));
//  * a backward line forms S = c + w v^2 + 2 b v and D = b + w v (w = a + K, the K offset of the
//    well-conditioned populations): its results are (S - D) / 2, a - S, (S + D) / 2.
// The error against 64 bits is that of the line-by-line form or less (FP32, 20000 random states per
// omega and velocity scale: 1.5e-7 .. 1.9e-7 of the populations against 2.0e-7 .. 2.5e-7).
//
// T is an arithmetic type whose operations each round on their own (Rn below, or the packed f2), so
// the compiler contracts nothing and every kernel computes the same bits from the same
// populations: a box, a pool domain, a list level, one node per thread or two.
// ---------------------------------------------------------------------------------------------

// one value with operations that are never contracted
template <class B>
struct Rn {
    B v;
    Rn() = default;
    __host__ __device__ __forceinline__ Rn(B a) : v(a) {}
};
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float rn_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double rn_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
template <class B> inline B rn_add(B a, B b) { return a + b; }
template <class B> inline B rn_mul(B a, B b) { return a * b; }
template <class B> inline B rn_fma(B a, B b, B c) { return std::fma(a, b, c); }
#endif
template <class B> __host__ __device__ __forceinline__ Rn<B> operator+(Rn<B> a, Rn<B> b) { return rn_add(a.v, b.v); }
template <class B> __host__ __device__ __forceinline__ Rn<B> operator-(Rn<B> a, Rn<B> b) { return rn_add(a.v, -b.v); }
template <class B> __host__ __device__ __forceinline__ Rn<B> operator*(Rn<B> a, Rn<B> b) { return rn_mul(a.v, b.v); }
template <class B> __host__ __device__ __forceinline__ Rn<B> operator/(Rn<B> a, Rn<B> b) { return a.v / b.v; }
template <class B> __host__ __device__ __forceinline__ Rn<B> operator-(Rn<B> a) { return Rn<B>(-a.v); }
template <class B> __host__ __device__ __forceinline__ Rn<B> fma(Rn<B> a, Rn<B> b, Rn<B> c) { return rn_fma(a.v, b.v, c.v); }

namespace k17detail {
// 1/x: IEEE division in double; the fast approximate division in float
__host__ __device__ __forceinline__ double fast_rcp(double x) { return 1.0 / x; }
__host__ __device__ __forceinline__ float fast_rcp(float x)
{
#ifdef __CUDA_ARCH__
    return __fdividef(1.0f, x);
#else
    return 1.0f / x;
#endif
}

// 1/rho for the velocity: correctly rounded in both precisions. u = j (1/rho) feeds the moment
// transforms, and the backward transform puts back j' = rho u + (the negated first central moment
// rho (j/rho - u)), so any error in u changes the node's momentum by twice that error times rho.
// A reciprocal that errs to one side (an approximate one) therefore makes the momentum drift step
// after step; a correctly rounded one errs both ways equally often. In float the rounded
// reciprocal flushes subnormals (rcp.rn.ftz): rho is near 1, so the bits are those of the IEEE
// reciprocal, and the form without flushing carries a slow path whose call raised the 16-bit
// pool kernel from 128 to 172 registers.
__host__ __device__ __forceinline__ double rho_rcp(double x) { return 1.0 / x; }
__host__ __device__ __forceinline__ float rho_rcp(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.rn.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}
template <class B>
__host__ __device__ __forceinline__ Rn<B> rho_rcp(Rn<B> x)
{
    return rho_rcp(x.v);
}

// 1 / (|m_i| + q_i) of the seven limited moments: in double one division and back-substitution
// through the running products (the denominators are >= the limiters, so the product stays far
// above the double range limit); in float seven fast divisions (a float product could underflow)
__host__ __device__ __forceinline__ void limiter_inverses(const Rn<double> (&m)[7], const double (&q)[7],
                                                          Rn<double> (&iv)[7])
{
    Rn<double> d[7], p[7];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        d[i] = Rn<double>(fabs(m[i].v)) + Rn<double>(q[i]);
        p[i] = i == 0 ? d[0] : p[i - 1] * d[i];
    }
    Rn<double> rr = fast_rcp(p[6].v);
#pragma unroll
    for (int i = 6; i > 0; --i) {
        iv[i] = rr * p[i - 1];
        rr = rr * d[i];
    }
    iv[0] = rr;
}
__host__ __device__ __forceinline__ void limiter_inverses(const Rn<float> (&m)[7], const float (&q)[7],
                                                          Rn<float> (&iv)[7])
{
#pragma unroll
    for (int i = 0; i < 7; ++i)
        iv[i] = fast_rcp(rn_add(fabsf(m[i].v), q[i]));
}

// raw moments 0, 1, 2 of one line
template <class T>
__host__ __device__ __forceinline__ void raw_line(T &a, T &b, T &c)
{
    const T p = c + a;
    const T q = c - a;
    a = p + b;
    b = q;
    c = p;
}
// central moments a, b, c of one line back to its populations; w = a + K
template <class T>
__host__ __device__ __forceinline__ void back_line(T &a, T &b, T &c, T v, T v2, T twov, T w, T half, T mhalf)
{
    const T S = fma(twov, b, fma(v2, w, c));
    const T D = fma(v, w, b);
    const T Sh = S * half;
    b = a - S;
    a = fma(mhalf, D, Sh);
    c = fma(half, D, Sh);
}
} // namespace k17detail

// T: the arithmetic type, B: its base type (constants and rates)
template <class T, class B>
__host__ __device__ __forceinline__ void k17_collide_fast(T *f, const K17Rates<B> &r, B fx, B fy, B fz, T &drho_out,
                                                          T &vx_out, T &vy_out, T &vz_out)
{
    using namespace k17detail;
    T m[27];
#pragma unroll
    for (int d = 0; d < 27; ++d)
        m[m3(d)] = f[d];
#define M(a, b, c) m[(a) * 9 + (b) * 3 + (c)]
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            raw_line(M(a, b, 0), M(a, b, 1), M(a, b, 2));
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            raw_line(M(a, 0, c), M(a, 1, c), M(a, 2, c));
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            raw_line(M(0, b, c), M(1, b, c), M(2, b, c));

    const T half = T(B(0.5)), mhalf = T(B(-0.5)), third = T(B(1) / B(3));
    const T drho = M(0, 0, 0), jx = M(1, 0, 0), jy = M(0, 1, 0), jz = M(0, 0, 1);
    const T rho = drho + T(B(1));
    const T ir = rho_rcp(rho);
    const T vx = fma(jx, ir, T(fx)), vy = fma(jy, ir, T(fy)), vz = fma(jz, ir, T(fz));
    const T mvx = -vx, mvy = -vy, mvz = -vz;
    // central moments up to third order (second ones without c_s^2: xx = sum (c_x - u_x)^2 f - 1/3)
    const T tx = fma(mvx, rho, jx), ty = fma(mvy, rho, jy), tz = fma(mvz, rho, jz);
    const T m200 = M(2, 0, 0), m020 = M(0, 2, 0), m002 = M(0, 0, 2);
    const T xx0 = fma(mvx, jx + tx, m200), yy0 = fma(mvy, jy + ty, m020), zz0 = fma(mvz, jz + tz, m002);
    const T pxy = fma(mvy, jx, M(1, 1, 0)), pxz = fma(mvz, jx, M(1, 0, 1)), pyz = fma(mvz, jy, M(0, 1, 1));
    const T qxy = fma(mvx, jy, M(1, 1, 0)), qxz = fma(mvx, jz, M(1, 0, 1)), qyz = fma(mvy, jz, M(0, 1, 1));
    const T xy0 = fma(mvx, ty, pxy), xz0 = fma(mvx, tz, pxz), yz0 = fma(mvy, tz, pyz);
    const T a200 = m200 + third, a020 = m020 + third, a002 = m002 + third;
    const T k210 = fma(mvx, pxy + xy0, fma(mvy, a200, M(2, 1, 0)));
    const T k120 = fma(mvy, qxy + xy0, fma(mvx, a020, M(1, 2, 0)));
    const T k201 = fma(mvx, pxz + xz0, fma(mvz, a200, M(2, 0, 1)));
    const T k102 = fma(mvz, qxz + xz0, fma(mvx, a002, M(1, 0, 2)));
    const T k021 = fma(mvy, pyz + yz0, fma(mvz, a020, M(0, 2, 1)));
    const T k012 = fma(mvz, qyz + yz0, fma(mvy, a002, M(0, 1, 2)));
    const T k111 = fma(mvx, yz0, fma(mvy, pxz, fma(mvz, M(1, 1, 0), M(1, 1, 1))));

    // velocity gradients times rho and the second order relaxation (K17...h:347-387)
    const T vx2 = vx * vx, vy2 = vy * vy, vz2 = vz * vz;
    const T dy0 = xx0 - yy0, dz0 = xx0 - zz0;
    const T gx = fma(T(r.mhw), dy0 + dz0, half * (drho - ((xx0 + yy0) + zz0)));
    const T gy = fma(T(r.w32), dy0, gx), gz = fma(T(r.w32), dz0, gx);
    const T ax = vx2 * gx, ay = vy2 * gy, az = vz2 * gz;
    const T trace = fma(T(B(-1.5)), (ax + ay) + az, drho);
    const T dy = fma(T(r.mc3h), ax - ay, T(r.omo) * dy0), dz = fma(T(r.mc3h), ax - az, T(r.omo) * dz0);
    const T xy = T(r.omo) * xy0, xz = T(r.omo) * xz0, yz = T(r.omo) * yz0;

    // third order with the quartic limiter (K17...h:397-433)
    const T lm[7] = { k111, k210 + k012, k201 + k021, k120 + k102, k210 - k012, k201 - k021, k120 - k102 };
    const B lq[7] = { r.qD, r.qP, r.qP, r.qP, r.qM, r.qM, r.qM };
    T li[7];
    limiter_inverses(lm, lq, li);
    const T c111 = (lm[0] * T(r.cD)) * li[0];
    const T px = (lm[1] * T(r.hP)) * li[1], mx = (lm[4] * T(r.hM)) * li[4];
    const T py = (lm[2] * T(r.hP)) * li[2], my = (lm[5] * T(r.hM)) * li[5];
    const T pz = (lm[3] * T(r.hP)) * li[3], mz = (lm[6] * T(r.hM)) * li[6];
    const T c210 = px + mx, c012 = px - mx, c201 = py + my, c021 = py - my, c120 = pz + mz, c102 = pz - mz;

    // central moments from the post-collision cumulants (K17...h:443-505)
    const T xx = ((dy + dz) + trace) * third, yy = xx - dy, zz = xx - dz;
    const T X = xx + third, Y = yy + third, Z = zz + third;
    const T xy2 = xy + xy, xz2 = xz + xz, yz2 = yz + yz;
    const T xy4 = xy2 + xy2, xz4 = xz2 + xz2, yz4 = yz2 + yz2;
    const T sxy = xy2 * xy, sxz = xz2 * xz, syz = yz2 * yz;
    const T u = xy2 * xz;
    const T c211 = fma(ir, fma(X, yz, u), T(r.kB) * yz0);
    const T c121 = fma(ir, fma(Y, xz, xy2 * yz), T(r.kB) * xz0);
    const T c112 = fma(ir, fma(Z, xy, xz2 * yz), T(r.kB) * xy0);
    const T y3 = yy * third, z3 = zz * third, d9 = drho * T(B(1) / B(9));
    const T z3d = z3 - d9;
    const T c220 = fma(ir, fma(xx, Y, (y3 - d9) + sxy), T(r.kA) * (gx + gy));
    const T c202 = fma(ir, fma(xx, Z, z3d + sxz), T(r.kA) * (gx + gz));
    const T c022 = fma(ir, fma(yy, Z, z3d + syz), T(r.kA) * (gy + gz));
    const T c122 = ir * fma(Z, c120, fma(Y, c102, fma(yz4, c111, fma(xz2, c021, xy2 * c012))));
    const T c212 = ir * fma(Z, c210, fma(X, c012, fma(xz4, c111, fma(yz2, c201, xy2 * c102))));
    const T c221 = ir * fma(X, c021, fma(Y, c201, fma(xy4, c111, fma(xz2, c120, yz2 * c210))));
    const T g3 = fma(xx, Y * Z, third * fma(yy, Z, z3));
    const T e2 = fma(T(B(2)), fma(u, yz4, fma(sxz, Y, fma(syz, X, fma(sxy, Z, g3)))),
                     T(B(1) / B(27)) * fma(drho, drho, -drho));
    const T c111t = c111 + c111;
    const T e0 = fma(Z, c220, fma(c111t, c111t, T(B(1) / B(9)) * trace));
    const T e1 = fma(yz4, c211, fma(xz4, c121, fma(xy4, c112, fma(X, c022, fma(Y, c202, e0)))));
    const T e3 = fma(T(B(2)), fma(c120, c102, fma(c210, c012, c201 * c021)), e1);
    const T c222 = ir * fma(-ir, e2, e3);

    // first moments change sign (K17...h:512-514)
    M(1, 0, 0) = -tx;
    M(0, 1, 0) = -ty;
    M(0, 0, 1) = -tz;
    M(2, 0, 0) = xx;
    M(0, 2, 0) = yy;
    M(0, 0, 2) = zz;
    M(1, 1, 0) = xy;
    M(1, 0, 1) = xz;
    M(0, 1, 1) = yz;
    M(1, 1, 1) = c111;
    M(2, 1, 0) = c210;
    M(0, 1, 2) = c012;
    M(2, 0, 1) = c201;
    M(0, 2, 1) = c021;
    M(1, 2, 0) = c120;
    M(1, 0, 2) = c102;
    M(2, 1, 1) = c211;
    M(1, 2, 1) = c121;
    M(1, 1, 2) = c112;
    M(2, 2, 0) = c220;
    M(2, 0, 2) = c202;
    M(0, 2, 2) = c022;
    M(1, 2, 2) = c122;
    M(2, 1, 2) = c212;
    M(2, 2, 1) = c221;
    M(2, 2, 2) = c222;
    const T twovx = vx + vx, twovy = vy + vy, twovz = vz + vz;
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T a0 = M(0, b, c);
            const T w = b == 1 || c == 1 ? a0 : a0 + T(b + c == 0 ? B(1) : b + c == 2 ? B(1) / B(3) : B(1) / B(9));
            back_line(M(0, b, c), M(1, b, c), M(2, b, c), vx, vx2, twovx, w, half, mhalf);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T a0 = M(a, 0, c);
            const T w = c == 1 ? a0 : a0 + T(k_y<B>(a, c));
            back_line(M(a, 0, c), M(a, 1, c), M(a, 2, c), vy, vy2, twovy, w, half, mhalf);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
            back_line(M(a, b, 0), M(a, b, 1), M(a, b, 2), vz, vz2, twovz, M(a, b, 0) + T(k_z<B>(a, b)), half, mhalf);
#undef M

#pragma unroll
    for (int d = 0; d < 27; ++d)
        f[d] = m[m3(d)];
    drho_out = drho;
    vx_out = vx;
    vy_out = vy;
    vz_out = vz;
}

} // namespace vfb

namespace vfb {
// the collision of the chosen arithmetic variant
template <class T, bool EXACT, bool VELOCITY = false>
__host__ __device__ __forceinline__ void collide(T *f, const K17Rates<T> &r, T fx, T fy, T fz, T &drho, T &vx, T &vy, T &vz)
{
    if constexpr (EXACT) {
        k17_collide<T, true, VELOCITY>(f, r, fx, fy, fz, drho, vx, vy, vz);
    } else {
        Rn<T> g[27], out[4];
#pragma unroll
        for (int d = 0; d < 27; ++d)
            g[d] = f[d];
        k17_collide_fast<Rn<T>, T>(g, r, fx, fy, fz, out[0], out[1], out[2], out[3]);
#pragma unroll
        for (int d = 0; d < 27; ++d)
            f[d] = g[d].v;
        drho = out[0].v;
        vx = out[1].v;
        vy = out[2].v;
        vz = out[3].v;
    }
}
} // namespace vfb
