// fnec_sincospi.cuh -- sin(pi x), cos(pi x) from a quadrant reduction and
// Taylor series, and 1/sqrt(x) by Newton's iteration (host and device), for
// the FMA-contracted kernels whose phases and distances need about 1e-16
// relative accuracy but not a particular libm's bits.
#pragma once
#include <cmath>
#include <cstring>

namespace fnec {

// The coefficients below, in the constant bank on the device: as literals
// each takes two moves into registers at every use (and the quadrant's signs
// are set on the high words, not by negations in the FP64 pipe).  The mixed
// fill of 4096 random antennas: 760 M -> 702 M warp instructions on its
// first 256, 15.97 -> 15.40 ms.
#ifdef __CUDACC__
static __constant__ double sp_const_dev[15] = {
    3.141592653589793,      -7.647163731819816e-13,  1.6059043836821613e-10, -2.505210838544172e-08,
    2.7557319223985893e-06, -0.0001984126984126984,  0.008333333333333333,   -0.16666666666666666,
    4.779477332387385e-14,  -1.1470745597729725e-11, 2.08767569878681e-09,   -2.755731922398589e-07,
    2.48015873015873e-05,   -0.001388888888888889,   0.041666666666666664};
#endif
#ifdef __CUDA_ARCH__
#define SP_K(i, v) sp_const_dev[i]
#else
#define SP_K(i, v) (v)
#endif

// sin(pi x) and cos(pi x) for 0 <= x < 2^50 (the phases of the mixed fill's
// samples and of the far field's wire runs).  Quadrant reduction in half-turns: adding 1.5 * 2^52 rounds 2x
// to the integer n (its low bits are n), and f = x - n / 2 is exact with
// |f| <= 1/4; then the Taylor series of sin and cos at theta = pi f
// (|theta| <= pi/4) to theta^15 and theta^16, whose truncation error is
// below 5e-17, in Horner form in theta^2, and the quadrant n mod 4 swaps
// and signs the pair.  About 22 FP64 operations and no table.
__host__ __device__ __forceinline__ void sincospi_taylor(double x, double &sn, double &cs) {
    const double big = 6755399441055744.0;  // 1.5 * 2^52
    const double t = fma(x, 2.0, big);
    const double nd = t - big;
#ifdef __CUDA_ARCH__
    const int q = __double2loint(t) & 3;
#else
    long long bits;
    memcpy(&bits, &t, sizeof(bits));
    const int q = (int)(bits & 3);
#endif
    const double th = fma(nd, -0.5, x) * SP_K(0, 3.141592653589793);
    const double t2 = th * th;
    // sin: theta (1 + t2 (-1/3! + t2 (1/5! - ... - t2 / 15!)))
    double ps = SP_K(1, -7.647163731819816e-13);      // -1/15!
    ps = fma(ps, t2, SP_K(2, 1.6059043836821613e-10));   // 1/13!
    ps = fma(ps, t2, SP_K(3, -2.505210838544172e-08));   // -1/11!
    ps = fma(ps, t2, SP_K(4, 2.7557319223985893e-06));   // 1/9!
    ps = fma(ps, t2, SP_K(5, -0.0001984126984126984));   // -1/7!
    ps = fma(ps, t2, SP_K(6, 0.008333333333333333));     // 1/5!
    ps = fma(ps, t2, SP_K(7, -0.16666666666666666));     // -1/3!
    const double s0 = fma(th * t2, ps, th);
    // cos: 1 + t2 (-1/2! + t2 (1/4! - ... + t2 / 16!))
    double pc = SP_K(8, 4.779477332387385e-14);       // 1/16!
    pc = fma(pc, t2, SP_K(9, -1.1470745597729725e-11));  // -1/14!
    pc = fma(pc, t2, SP_K(10, 2.08767569878681e-09));    // 1/12!
    pc = fma(pc, t2, SP_K(11, -2.755731922398589e-07));  // -1/10!
    pc = fma(pc, t2, SP_K(12, 2.48015873015873e-05));    // 1/8!
    pc = fma(pc, t2, SP_K(13, -0.001388888888888889));   // -1/6!
    pc = fma(pc, t2, SP_K(14, 0.041666666666666664));    // 1/4!
    pc = fma(pc, t2, -0.5);                              // -1/2!
    const double c0 = fma(t2, pc, 1.0);
    const double a = (q & 1) ? c0 : s0, b = (q & 1) ? s0 : c0;
#ifdef __CUDA_ARCH__
    // the quadrant's signs on the high words
    sn = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
    cs = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
#else
    sn = (q & 2) ? -a : a;
    cs = ((q + 1) & 2) ? -b : b;
#endif
}

// 1/sqrt(x) for normal, finite x > 0: a single-precision first guess
// (about 23 correct bits; the device's approximate reciprocal square root),
// then two Newton steps for f(y) = y^-2 - x in FP64,
// y <- y + (y / 2)(1 - x y^2), each doubling the correct bits: within about
// 3e-16 relative of the true value over the fill's range (R^2 from 1e-8 to
// 1e4 m^2).  Nine FP64 / conversion operations and no branch.
__host__ __device__ __forceinline__ double rsqrt_newton(double x) {
#ifdef __CUDA_ARCH__
    double y = (double)rsqrtf((float)x);
#else
    double y = (double)(1.0f / std::sqrt((float)x));
#endif
    double e = fma(-x * y, y, 1.0);
    y = fma(0.5 * y, e, y);
    e = fma(-x * y, y, 1.0);
    y = fma(0.5 * y, e, y);
    return y;
}

// Either sign: sin(pi x) is odd, cos(pi x) even.
__host__ __device__ __forceinline__ void sincospi_taylor_signed(double x, double &sn, double &cs) {
    sincospi_taylor(fabs(x), sn, cs);
    if (x < 0.0) sn = -sn;
}

}  // namespace fnec
