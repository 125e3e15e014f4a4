// Host check of kpolaris_b200/csrc/kp_exact.cuh: its quotients and square
// roots against the IEEE operators, bit for bit.  The device's fused
// multiply-add, rounded product and bit casts are the C library's here; the
// hardware's approximate reciprocal and reciprocal square root, of which only
// the accuracy is known, are the correct values off by up to `err` relative
// (argument 2), at random.  argv: draws, err.  Prints the mismatches of each
// kind (xq::Counts).
#include <cfenv>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#define KP_EXACT_METHOD 1

static double start_err;
static unsigned long long start_state = 88172645463325252ull;

inline double off() {
    start_state = start_state * 6364136223846793005ull + 1442695040888963407ull;
    return 1.0 + start_err * (double(start_state >> 11) * 0x1p-52 - 1.0);
}
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline double rounded(int mode, double a, double b, double c) {
    volatile double x = a, y = b, z = c;
    std::fesetround(mode);
    volatile double r = std::fma(x, y, z);
    std::fesetround(FE_TONEAREST);
    return r;
}
inline double __fma_ru(double a, double b, double c) { return rounded(FE_UPWARD, a, b, c); }
inline double __fma_rd(double a, double b, double c) { return rounded(FE_DOWNWARD, a, b, c); }
inline double __dmul_rd(double a, double b) { return rounded(FE_DOWNWARD, a, b, 0.0); }
inline double __dmul_rn(double a, double b) { return a * b; }
inline long long __double_as_longlong(double v) {
    long long u;
    std::memcpy(&u, &v, 8);
    return u;
}
inline double __longlong_as_double(long long u) {
    double v;
    std::memcpy(&v, &u, 8);
    return v;
}
inline int __double2hiint(double v) { return int(__double_as_longlong(v) >> 32); }
inline int __double2loint(double v) { return int(__double_as_longlong(v) & 0xffffffffll); }
inline double __hiloint2double(int hi, int lo) {
    return __longlong_as_double((long long)(((unsigned long long)unsigned(hi) << 32) | unsigned(lo)));
}
namespace kp {
// 20 bits of the significand, as the hardware gives it
inline double approx(double v) {
    return std::isfinite(v) ? __longlong_as_double(__double_as_longlong(v * off()) & ~0xffffffffll) : v;
}
inline double recip_start(double b) { return approx(1.0 / b); }
inline double rsqrt_start(double v) { return approx(1.0 / std::sqrt(v)); }
}  // namespace kp

#include "kp_exact.cuh"
#include "exact_quotients.h"

int main(int argc, char** argv) {
    const long draws = std::atol(argv[1]);
    start_err = std::atof(argv[2]);
    uint64_t s = 0x9E3779B97F4A7C15ull;
    xq::Counts n = {};
    for (long i = 0; i < draws && argc > 2; ++i) xq::check(s, n);
    std::printf("%llu %llu %llu %llu %llu\n", n.quots, n.over, n.quot, n.recip, n.root);
    return 0;
}
