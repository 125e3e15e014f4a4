// Operands for the tests of kpolaris_b200/csrc/kp_exact.cuh, and the
// comparison of its quotients and roots with the IEEE operators.  Included by
// exact_quotients.cpp (host, with the device's operations restated) and
// exact_quotients.cu (device).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define XQ_FN __device__ __forceinline__
#else
#define XQ_FN inline
#endif

namespace xq {

XQ_FN uint64_t bits(double v) {
    uint64_t u;
    memcpy(&u, &v, 8);
    return u;
}

XQ_FN double value(uint64_t u) {
    double v;
    memcpy(&v, &u, 8);
    return v;
}

XQ_FN uint64_t next(uint64_t& s) {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}

// Significands: random, all ones, within 256 of all ones, a power of two, few
// leading bits, few trailing bits, and those of reciprocals and roots closest
// to halfway between two numbers: B with B M = 2^106 - 1, - 2 or - 4 for an M
// of 54 bits, V with M M = 2^54 V + 1, 9, -7, -15, 17 or 25.
XQ_FN uint64_t significand(uint64_t& s) {
    const uint64_t full = (uint64_t(1) << 52) - 1, m = next(s) & full;
    const uint64_t close[20] = {0x1e756f08df1792, 0x1e20adbc4078a2, 0x1ef7930608393e, 0x1de441d5331432, 0x1da210daeb138e,
                                0x1bea3278b789d2, 0x1ffb8a8b628dbc, 0x1fe24bffeb8794, 0x1c928b5b9dc714, 0x15555555555554,
                                0x10000000000001, 0x10000000000003, 0x10000000000005, 0x1fffffffffffff, 0x1ffffffffffffd,
                                0x1ffffffffffffb, 0x1d407bb3641da5, 0x15b95344972fe2, 0x12b035c1197f48,
                                0x1256565cadcbf4};
    if ((next(s) & 7) == 0) return close[next(s) % 20] & full;
    switch (next(s) >> 61) {
    case 0: return full;
    case 1: return full - (m & 255);
    case 2: return 0;
    case 3: return m & 255;
    case 4: return m & ~((uint64_t(1) << 40) - 1);
    default: return m;
    }
}

// A number of one in `span` binades around 1, of either sign if `negative`.
XQ_FN double number(uint64_t& s, int span, bool negative) {
    const uint64_t e = uint64_t(1023 - span / 2 + int(next(s) % uint64_t(span)));
    const uint64_t sign = negative ? next(s) & (uint64_t(1) << 63) : 0;
    return value(significand(s) | (e << 52) | sign);
}

// Any number: zeros, subnormal numbers, infinities and NaN among them, and
// the ends of exact_numerator's and exact_divisor's ranges.
XQ_FN double anything(uint64_t& s) {
    const uint64_t sign = next(s) & (uint64_t(1) << 63);
    const int edges[8] = {523, 1522, 823, 1222, 522, 1523, 822, 1223};
    switch (next(s) % 8) {
    case 0: return value(sign);
    case 1: return value(sign | (next(s) & 255));
    case 2: return value(sign | (uint64_t(0x7ff) << 52) | (next(s) & 1));
    case 3: return value(sign | (uint64_t(edges[next(s) % 8]) << 52) | significand(s));
    case 4: return value(sign | ((next(s) % 0x7ff) << 52) | significand(s));
    default: return value(sign | bits(number(s, 400, false)));
    }
}

XQ_FN bool same(double a, double b) { return bits(a) == bits(b) || (!(a == a) && !(b == b)); }

// What differed: quotients of any operands, by a constant, of operands that
// share an unchecked reciprocal, reciprocals, square roots.
struct Counts {
    unsigned long long quots, over, quot, recip, root;
};

// One draw of every kind.
XQ_FN void check(uint64_t& s, Counts& n) {
    {
        const double b = anything(s);
        double v[3] = {anything(s), anything(s), anything(s)}, q[3] = {v[0], v[1], v[2]};
        kp::exact_quots(q, b);
        for (int i = 0; i < 3; ++i) n.quots += !same(q[i], v[i] / b);
    }
    {
        const double a = anything(s);
        n.over += !same(KP_OVER(a, 3.75), a / 3.75) + !same(KP_OVER(a, 4.7), a / 4.7) + !same(KP_OVER(a, 0.1), a / 0.1) +
                  !same(KP_OVER(a, 2.99792458e10), a / 2.99792458e10) + !same(KP_OVER(a, 24.0), a / 24.0);
    }
    {
        const double b = number(s, 900, false), a = (next(s) & 15) ? number(s, 100, true) : value(next(s) & (uint64_t(1) << 63));
        const kp::ExactRecip r = kp::exact_recip(b);
        n.recip += !same(r.y, 1.0 / b);
        n.quot += !same(kp::exact_quot(a, r), a / b);
        n.root += !same(kp::exact_sqrt(b), sqrt(b));
    }
}

}  // namespace xq
