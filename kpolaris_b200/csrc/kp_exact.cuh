// kp_exact.cuh -- correctly rounded FP64 quotients and square roots without
// the range checks and the out-of-line path of the compiler's own, for
// operands known to lie well inside the range.  Several quotients by one
// divisor share its reciprocal, and nothing branches between independent
// ones, so they overlap: the compiler's division takes a lone warp 127
// cycles, one after the other, and the Kerr-Schild connection has twenty.
//
// Method: P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990) 111-119 (also Muller et
// al., Handbook of Floating-Point Arithmetic, ch. 4).  With fused
// multiply-adds, a reciprocal y of b within one ulp becomes the correctly
// rounded one by y + y (1 - b y), but for a divisor whose significand is all
// ones (exact_recip sees to it); with it, a quotient q of a / b within one ulp
// becomes the correctly rounded one by q - y (b q - a).  The residuals are
// formed as b q - a so that a zero numerator over a positive divisor keeps its
// sign.  A square root g of v within one ulp becomes the rounded one by
// g + (v - g g) h with h = 1 / (2 sqrt(v)), but for one significand
// (exact_sqrt sees to it).  The starting values are the hardware's approximate
// reciprocal and reciprocal square root, of 20 bits, taken to one ulp by the
// geometric series of 1 / b = y / (1 - e), e = 1 - b y, and the binomial series
// of v^-1/2 = y (1 - e)^-1/2, e = 1 - v y y, each to its term in e^2: what is
// left out is below e^3 = 2^-57.
#pragma once

#include <cmath>

#include "kp_common.cuh"

namespace kp {

#if defined(__CUDACC__) || defined(KP_EXACT_METHOD)  // the latter: a host test of the method

#ifdef __CUDACC__
__device__ __forceinline__ double recip_start(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}

__device__ __forceinline__ double rsqrt_start(double v) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    return y;
}
#endif

struct ExactRecip {
    double b, y;
};

// The correctly rounded reciprocal of b, 1e-150 < b < 1e150.
__device__ __forceinline__ ExactRecip exact_recip(double b) {
    double y = recip_start(b);
    double e = __fma_rn(-b, y, 1.0);
    // Rounded up: from the number above its reciprocal the last step finds that
    // of b = 2^n (2 - 2^-52) too, 2^-(n + 1) (1 + 2^-52).  From below, at
    // 2^-(n + 1), it lands halfway between the two and stays.  (Elsewhere the
    // step is off by e e / b, and a reciprocal within that of a halfway point,
    // which is 2^-106 / b from the nearest, is half an ulp from the number above.)
    y = __fma_ru(y, __fma_rn(e, e, e), y);
    e = __fma_rn(-b, y, 1.0);
    return ExactRecip{b, __fma_rn(y, e, y)};
}

// RN(a / b) for a zero or 1e-200 < |a| < 1e150 with 1e-250 < |a / b| < 1e150.
__device__ __forceinline__ double exact_quot(double a, const ExactRecip& r) {
    double q = __dmul_rn(a, r.y);
    q = __fma_rn(-__fma_rn(r.b, q, -a), r.y, q);
    return __fma_rn(-__fma_rn(r.b, q, -a), r.y, q);
}

// RN(sqrt(v)), 1e-290 < v < 1e290.
__device__ __forceinline__ double exact_sqrt(double v) {
    double y = rsqrt_start(v);
    const double e = __fma_rn(-__dmul_rn(v, y), y, 1.0);
    const double ye = __dmul_rn(y, e), c = __fma_rn(0.375, e, 0.5);
    const double h = __dmul_rn(0.5, __fma_rn(ye, c, y));
    // Rounded down: the root of v = 4^n (1 - 2^-53) lies a hair under the middle
    // between 2^n and the number below it.  The steps reach that number from
    // below; from 2^n they would stay there.
    double g = __dmul_rd(v, __fma_rd(ye, c, y));
    g = __fma_rn(__fma_rn(-g, g, v), h, g);
    return __fma_rn(__fma_rn(-g, g, v), h, g);
}

// A numerator's factor for which products of a few of its like stay clear of
// underflow.
__device__ __forceinline__ bool exact_factor(double v) { return abs_val(v) > 1e-50 || v == 0.0; }

// 2^-500 < |v| < 2^500 or zero: with a divisor between 2^-200 and 2^200 the
// quotient and its residuals are normal numbers.
__device__ __forceinline__ bool exact_numerator(double v) {
    return (unsigned(__double2hiint(v) >> 20) & 0x7ffu) - 523u < 1000u || v == 0.0;
}

// 2^-200 < b < 2^200.  A negative divisor would give a zero numerator's
// quotient the wrong sign.
__device__ __forceinline__ bool exact_divisor(double b) {
    return (unsigned(__double2hiint(b)) >> 20) - 823u < 400u;
}

// The rare operands out of range.
static __device__ __noinline__ double plain_quot(double a, double b) { return a / b; }

// v[i] = RN(v[i] / b) for any operands: together where all of them are in
// range, by the compiler's division otherwise.
template<int N>
__device__ __forceinline__ void exact_quots(double (&v)[N], double b) {
    bool ok = exact_divisor(b);
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && exact_numerator(v[i]);
    if (ok) {
        const ExactRecip r = exact_recip(b);
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = exact_quot(v[i], r);
    } else {
#pragma unroll 1
        for (int i = 0; i < N; ++i) v[i] = plain_quot(v[i], b);
    }
}

// RN(a / b) for a constant b of ordinary size: `inv` is RN(1 / b), folded by
// the compiler.
__device__ __forceinline__ double exact_over(double a, double b, double inv) {
    if (exact_numerator(a)) return exact_quot(a, ExactRecip{b, inv});
    return plain_quot(a, b);
}
#define KP_OVER(a, b) ::kp::exact_over((a), (b), 1.0 / (b))

#else  // host builds of the device code: the compiler's own

struct ExactRecip {
    double b;
};
inline ExactRecip exact_recip(double b) { return ExactRecip{b}; }
inline double exact_quot(double a, const ExactRecip& r) { return a / r.b; }
inline double exact_sqrt(double v) { return sqrt(v); }
template<int N>
inline void exact_quots(double (&v)[N], double b) {
    for (int i = 0; i < N; ++i) v[i] = v[i] / b;
}
#define KP_OVER(a, b) ((a) / (b))

#endif

}  // namespace kp
