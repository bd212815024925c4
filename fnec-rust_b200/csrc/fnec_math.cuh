// fnec_math.cuh -- exact-parity arithmetic for the Hallen kernels.
//
// Complex arithmetic with the exact operation order of num-complex 0.4.6
// and no FMA contraction (explicit _rn intrinsics on the device), so sums
// and eliminations reproduce the reference bit for bit.  The libm functions
// the reference calls (sin, cos, hypot) are restated in fnec_libm.cuh.
//
// The header compiles as CUDA device code under nvcc and as plain C++ under
// g++ (host unit tests).
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#include "fnec_libm.cuh"

#ifdef __CUDACC__
#define FNEC_FN __device__ __forceinline__
#define D_ADD(a, b) __dadd_rn((a), (b))
#define D_SUB(a, b) __dsub_rn((a), (b))
#define D_MUL(a, b) __dmul_rn((a), (b))
#define D_DIV(a, b) __ddiv_rn((a), (b))
#define D_SQRT(a) __dsqrt_rn((a))
#define D_FMA(a, b, c) __fma_rn((a), (b), (c))
#else
#define FNEC_FN static inline
#define D_ADD(a, b) ((a) + (b))
#define D_SUB(a, b) ((a) - (b))
#define D_MUL(a, b) ((a) * (b))
#define D_DIV(a, b) ((a) / (b))
#define D_SQRT(a) sqrt((a))
#define D_FMA(a, b, c) fma((a), (b), (c))
#endif

namespace fnec {

// ---------------------------------------------------------------------------
// num-complex 0.4.6 arithmetic, each operation separately rounded
// ---------------------------------------------------------------------------
struct cx {
    double re, im;
};
FNEC_FN cx cx_make(double re, double im) { return {re, im}; }
FNEC_FN cx cx_add(cx a, cx b) { return {D_ADD(a.re, b.re), D_ADD(a.im, b.im)}; }
FNEC_FN cx cx_sub(cx a, cx b) { return {D_SUB(a.re, b.re), D_SUB(a.im, b.im)}; }
// (ac - bd, ad + bc)
FNEC_FN cx cx_mul(cx a, cx b) {
    return {D_SUB(D_MUL(a.re, b.re), D_MUL(a.im, b.im)), D_ADD(D_MUL(a.re, b.im), D_MUL(a.im, b.re))};
}
// conj(a) * b exactly as num-complex evaluates it: (ar*br - (-ai)*bi,
// ar*bi + (-ai)*br), which IEEE makes equal to (ar*br + ai*bi, ar*bi - ai*br).
FNEC_FN cx cx_conj_mul(cx a, cx b) {
    return {D_ADD(D_MUL(a.re, b.re), D_MUL(a.im, b.im)), D_SUB(D_MUL(a.re, b.im), D_MUL(a.im, b.re))};
}
// ((ac + bd) / |b|^2, (bc - ad) / |b|^2)
FNEC_FN cx cx_div(cx a, cx b) {
    double ns = D_ADD(D_MUL(b.re, b.re), D_MUL(b.im, b.im));
    double re = D_ADD(D_MUL(a.re, b.re), D_MUL(a.im, b.im));
    double im = D_SUB(D_MUL(a.im, b.re), D_MUL(a.re, b.im));
    return {D_DIV(re, ns), D_DIV(im, ns)};
}
// Complex64::norm = f64::hypot, as the platform libm evaluates it
FNEC_FN double cx_norm(cx a) { return fnec_libm::libm_hypot(a.re, a.im); }
FNEC_FN double cx_norm_sqr(cx a) { return D_ADD(D_MUL(a.re, a.re), D_MUL(a.im, a.im)); }

// ---------------------------------------------------------------------------
// Correctly rounded sqrt(x) and quotients by it, from one reciprocal square
// root: the fill's G(R) takes a square root and two divisions by it, and the
// three together cost less than one general division here.
//   y  = 1/sqrt(x): a single-precision first guess y0, then Householder's
//        cubic step y0 (1 + e/2 + 3 e^2/8) with e = 1 - x y0^2 (|e| < 2^-21,
//        so the step leaves 2^-65 beside the roundings);
//   r  = g + (x - g^2) y/2 with g = x y, the residual exact in an FMA;
//   z  = y + y (1 - r y), the reciprocal of r;
//   a/r = q + (a - q r) z with q = a z.
// The last corrections are Markstein's (Computation of elementary functions
// on the IBM RISC System/6000 processor, 1990): with z the rounded reciprocal
// of r and q within an ulp, a/r comes out rounded, and so does z itself unless
// r's mantissa is all ones.  The root's value before its final rounding is
// within about 2^-103 of exact, relative.  That bound alone does not settle
// every root (they come as near as about 2^-107 to the middle of two doubles):
// tests/test_gpu_exact_division.py constructs roots and quotients from 2^-97
// to 2^-104 of a middle and finds no wrong bit on the device.  Domain: x normal
// in [2^-100, 2^100) and quotients whose residual stays normal (a zero, or |a|
// above 2^-800); callers fall back to the general operations outside.
// ---------------------------------------------------------------------------
struct SqrtRecip {
    double r, z;  // sqrt(x), 1/sqrt(x) rounded from r
};
FNEC_FN SqrtRecip sqrt_recip(double x) {
#ifdef __CUDA_ARCH__
    float f;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(__double2float_rn(x)));
    const double y0 = (double)f;
#else
    const double y0 = (double)(1.0f / sqrtf((float)x));
#endif
    const double e = D_FMA(-D_MUL(x, y0), y0, 1.0);
    const double y = D_FMA(D_MUL(y0, e), D_FMA(e, 0.375, 0.5), y0);
    const double g = D_MUL(x, y);
    const double r = D_FMA(D_FMA(-g, g, x), D_MUL(0.5, y), g);
    double z = D_FMA(D_FMA(-r, y, 1.0), y, y);
    // an all-ones mantissa is the one whose reciprocal that step can leave
    // an ulp off (1/r lies just above the middle of two doubles)
    if ((uint32_t)fnec_libm::lm_bits(r) == 0xffffffffu) z = D_DIV(1.0, r);
    return {r, z};
}
// a / sr.r (the residual with its sign turned twice: a zero keeps its sign)
FNEC_FN double div_by(double a, SqrtRecip sr) {
    const double q = D_MUL(a, sr.z);
    return D_FMA(-D_FMA(q, sr.r, -a), sr.z, q);
}
FNEC_FN bool sqrt_recip_domain(double x) {
    const uint32_t k = (uint32_t)(fnec_libm::lm_bits(x) >> 32);
    return k - 0x39b00000u < 0x46300000u - 0x39b00000u;  // 2^-100 <= x < 2^100
}

}  // namespace fnec
