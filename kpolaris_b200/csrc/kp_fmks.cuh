// kp_fmks.cuh -- Kerr spacetime in funky modified Kerr-Schild (FMKS) native
// coordinates (t, x1, x2, phi), FP64: the theta(x1, x2) map and its
// derivatives, the native metric, the transport right-hand side through the
// spherical Kerr-Schild connection, and the pinhole camera.
//
// Reference: KerrFMKSMetric and its transport_rhs
// (src/geometry/kerr_fmks.hpp:11-481), the spherical Kerr-Schild connection
// work and fixed-p contraction (src/geometry/kerr_schild_spherical.hpp:192-323),
// the ipole camera tetrad (src/camera/camera.hpp:141-270, 302-456, 485-513).
// The theta map calls exp/sin/cos on every evaluation, so this path agrees
// with the reference's CPU run to libm accuracy, not bit for bit.
#pragma once

#include "kp_camera.cuh"
#include "kp_exact.cuh"
#include "kp_geometry_mixed.cuh"

namespace kp {

// The quotients of the FP64 right-hand side.  It has seventeen divisions by
// nine divisors; the compiler's, at 127 cycles each and one after the other,
// were two thirds of its 3,000 cycles.  They are formed by shared reciprocals
// (kp_exact.cuh, the same rounding) without a branch between them, and taken
// again by the compiler's division in the rare case that an operand was out
// of that method's range.
struct FmksDivisor {
    double b, y;
};

KP_HD FmksDivisor fmks_divisor(double b) {
#ifdef __CUDA_ARCH__
    return FmksDivisor{b, exact_recip(b).y};
#else
    return FmksDivisor{b, 0.0};
#endif
}

template<bool EXACT>
KP_HD double fmks_quot(double a, const FmksDivisor& d, bool& in_range) {
#ifdef __CUDA_ARCH__
    if constexpr (!EXACT) return plain_quot(a, d.b);
    in_range = in_range && exact_numerator(a) && exact_divisor(d.b);
    return exact_quot(a, ExactRecip{d.b, d.y});
#else
    return a / d.b;
#endif
}

KP_HD double fmks_power(double x, double p) {
    const int n = int(p + 0.5);
    if (abs_val(p - double(n)) < 1e-10 && n >= 0) {
        double y = 1.0;
        const double ax = abs_val(x);
        for (int i = 0; i < n; ++i) y *= ax;
        if (x < 0.0 && (n % 2) == 1) y = -y;
        return y;
    }
    return pow(abs_val(x), p);
}

// theta(x1, x2) and its first and second derivatives
// (build_fmks_connection_work, kerr_fmks.hpp:296-348).
struct FmksTheta {
    double r, th, dth1, dth2, d2th11, d2th12, d2th22;
};

// The quotients of the map: za / (alpha + 1), dthJ's second term, d2thJ's
// factor and its two terms.
struct FmksMap {
    double za_al, dj, cj, t1, t2;
};

KP_HD void fmks_powers(const FmksParams& m, double z, double& za, double& za1, double& za2) {
    if (abs_val(m.poly_alpha - 14.0) < 1e-12) {
        const double z2 = z * z;
        const double z4 = z2 * z2;
        const double z8 = z4 * z4;
        za2 = z8 * z4;
        za1 = za2 * z;
        za = za2 * z2;
    } else {
        za = fmks_power(z, m.poly_alpha);
        za1 = fmks_power(z, m.poly_alpha - 1.0);
        za2 = fmks_power(z, m.poly_alpha - 2.0);
    }
}

template<bool EXACT>
KP_HD FmksMap fmks_map(const FmksParams& m, double y, bool& in_range) {
    const double al1 = m.poly_alpha + 1.0;
    const FmksDivisor xt = fmks_divisor(m.poly_xt), al = fmks_divisor(al1);
    const double z = fmks_quot<EXACT>(y, xt, in_range);
    double za, za1, za2;
    fmks_powers(m, z, za, za1, za2);
    FmksMap q;
    q.za_al = fmks_quot<EXACT>(za, al, in_range);
    q.cj = fmks_quot<EXACT>(4.0 * m.poly_norm * m.poly_alpha, al, in_range);
    q.dj = fmks_quot<EXACT>(2.0 * m.poly_alpha * m.poly_norm * y * za1, fmks_divisor(al1 * m.poly_xt), in_range);
    q.t1 = fmks_quot<EXACT>(2.0 * za1, xt, in_range);
    q.t2 = fmks_quot<EXACT>(y * (m.poly_alpha - 1.0) * za2, fmks_divisor(m.poly_xt * m.poly_xt), in_range);
    return q;
}

template<bool MIXED = false>
KP_HD FmksTheta fmks_theta(const FmksParams& m, double x1, double x2) {
    const double y = 2.0 * x2 - 1.0;
    const double expfac = exp(m.mks_smooth * (m.startx1 - x1));
    double s2, c2;
    FmksMap q;
    if constexpr (MIXED) {
        // reciprocals of the map's constants, and its angle in half turns
        const double inv_xt = kp_recip(m.poly_xt);
        const double inv_al1 = kp_recip(m.poly_alpha + 1.0);
        double za, za1, za2;
        fmks_powers(m, y * inv_xt, za, za1, za2);
        q.za_al = za * inv_al1;
        q.dj = (2.0 * m.poly_alpha * m.poly_norm * y * za1) * (inv_al1 * inv_xt);
        q.cj = 4.0 * m.poly_norm * m.poly_alpha * inv_al1;
        q.t1 = 2.0 * za1 * inv_xt;
        q.t2 = y * (m.poly_alpha - 1.0) * za2 * (inv_xt * inv_xt);
#ifdef __CUDA_ARCH__
        sincospi(2.0 * x2, &s2, &c2);
#else
        sincos(2.0 * kPi * x2, &s2, &c2);
#endif
    } else {
        bool in_range = true;
        q = fmks_map<true>(m, y, in_range);
        if (!in_range) q = fmks_map<false>(m, y, in_range);
        sincos(2.0 * kPi * x2, &s2, &c2);
    }
    const double thG = kPi * x2 + ((1.0 - m.hslope) / 2.0) * s2;
    const double thJ = m.poly_norm * y * (1.0 + q.za_al) + 0.5 * kPi;
    const double dthG = kPi + (1.0 - m.hslope) * kPi * c2;
    const double dthJ = 2.0 * m.poly_norm * (1.0 + q.za_al) + q.dj;
    const double d2thG = -2.0 * (1.0 - m.hslope) * kPi * kPi * s2;
    const double d2thJ = q.cj * (q.t1 + q.t2);
    FmksTheta t;
    t.r = exp(x1);
    t.th = thG + expfac * (thJ - thG);
    t.dth1 = -m.mks_smooth * expfac * (thJ - thG);
    t.dth2 = dthG + expfac * (dthJ - dthG);
    t.d2th11 = -m.mks_smooth * t.dth1;
    t.d2th12 = -m.mks_smooth * expfac * (dthJ - dthG);
    t.d2th22 = d2thG + expfac * (d2thJ - d2thG);
    return t;
}

// theta alone (theta_from_x2, kerr_fmks.hpp:46-53).
KP_HD double fmks_theta_of(const FmksParams& m, double x1, double x2) {
    const double y = 2.0 * x2 - 1.0;
    const double thG = kPi * x2 + ((1.0 - m.hslope) / 2.0) * sin(2.0 * kPi * x2);
    const double thJ = m.poly_norm * y * (1.0 + fmks_power(y / m.poly_xt, m.poly_alpha) / (m.poly_alpha + 1.0)) +
                       0.5 * kPi;
    return thG + exp(m.mks_smooth * (m.startx1 - x1)) * (thJ - thG);
}

// x2 with theta(x1, x2) = theta, by 64 bisections (native_x2_from_theta, :102-112).
KP_HD double fmks_x2_of(const FmksParams& m, double x1, double theta) {
    double lo = 0.0, hi = 1.0;
    for (int it = 0; it < 64; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (fmks_theta_of(m, x1, mid) < theta) lo = mid; else hi = mid;
    }
    return 0.5 * (lo + hi);
}

KP_HD double fmks_radius(const D4& X) { return exp(X.v[1]); }

// Native metric g_{mu nu} at X (the Jacobian transform of the spherical
// Kerr-Schild metric, gcov_matrix :141-169, in closed form).
KP_HD void fmks_gcov(const FmksParams& m, const D4& X, double g[4][4]) {
    const FmksTheta t = fmks_theta(m, X.v[1], X.v[2]);
    double s, c;
    sincos(t.th, &s, &c);
    const double s2 = s * s, a = m.spin, a2 = a * a;
    const double rho2 = t.r * t.r + a2 * c * c;
    const double f = 2.0 * m.mass * t.r / rho2;
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) g[i][j] = 0.0;
    g[0][0] = -1.0 + f;
    g[0][1] = g[1][0] = f * t.r;
    g[0][3] = g[3][0] = -a * f * s2;
    g[1][1] = (1.0 + f) * t.r * t.r + rho2 * t.dth1 * t.dth1;
    g[1][2] = g[2][1] = rho2 * t.dth1 * t.dth2;
    g[1][3] = g[3][1] = -a * s2 * (1.0 + f) * t.r;
    g[2][2] = rho2 * t.dth2 * t.dth2;
    g[3][3] = s2 * (rho2 + a2 * s2 * (1.0 + f));
}

// Native inverse metric at X: the inverse Jacobian applied to the spherical
// Kerr-Schild inverse metric (native_metric, grmhd_grid.hpp:660-708).
KP_HD void fmks_gcon(const FmksParams& m, const D4& X, double gi[4][4]) {
    const FmksTheta t = fmks_theta(m, X.v[1], X.v[2]);
    double s, c;
    sincos(t.th, &s, &c);
    const double s2 = max_val(s * s, kTiny), a = m.spin, a2 = a * a;
    const double rho2 = t.r * t.r + a2 * c * c;
    const double delta = t.r * t.r - 2.0 * m.mass * t.r + a2;
    const double f = 2.0 * m.mass * t.r / rho2;
    double k[4][4] = {};
    k[0][0] = -(1.0 + f);
    k[0][1] = k[1][0] = f;
    k[1][1] = delta / rho2;
    k[1][3] = k[3][1] = a / rho2;
    k[2][2] = 1.0 / rho2;
    k[3][3] = 1.0 / (rho2 * s2);
    double J[4][4] = {};
    J[0][0] = 1.0;
    J[1][1] = 1.0 / t.r;
    J[2][1] = -t.dth1 / (t.r * t.dth2);
    J[2][2] = 1.0 / t.dth2;
    J[3][3] = 1.0;
    for (int mu = 0; mu < 4; ++mu)
        for (int nu = 0; nu < 4; ++nu) {
            double sum = 0.0;
            for (int p = 0; p < 4; ++p)
                for (int q = 0; q < 4; ++q) sum += J[mu][p] * J[nu][q] * k[p][q];
            gi[mu][nu] = sum;
        }
}

KP_HD double dot_gm(const double g[4][4], const D4& u, const D4& v) {
    double out = 0.0;
    for (int mu = 0; mu < 4; ++mu)
        for (int nu = 0; nu < 4; ++nu) out += g[mu][nu] * u.v[mu] * v.v[nu];
    return out;
}

// Spherical Kerr-Schild connection work at (r, theta): g^{mu nu} and the
// r- and theta-derivatives of g_{mu nu} (build_spherical_ks_connection_work,
// kerr_schild_spherical.hpp:198-266), by their distinct nonzero entries: d/dr
// g has (A A 0 B), (A A 0 B), (0 0 C 0), (B B 0 D) as its rows and d/dtheta g
// (E E 0 F0), (E E 0 F1), (0 0 G 0), (F0 F1 0 H).
struct SksConn {
    double g00, g01, g11, g13, g22, g33;
    double A, B, C, D, E, F0, F1, G, H;
};

template<bool EXACT>
KP_HD SksConn sks_conn(double mass, double a, double r, double s, double cc, bool& in_range) {
    SksConn c;
    const double a2 = a * a, s2 = s * s, safe_s2 = max_val(s2, kTiny);
    const double rho2 = r * r + a2 * cc * cc, rho4 = rho2 * rho2;
    const double delta = r * r - 2.0 * mass * r + a2;
    const double drho_dr = 2.0 * r, drho_dth = -2.0 * a2 * s * cc, ds2_dth = 2.0 * s * cc;
    const FmksDivisor d2 = fmks_divisor(rho2), d4 = fmks_divisor(rho4);
    const double f = fmks_quot<EXACT>(2.0 * mass * r, d2, in_range);
    const double df_dr = fmks_quot<EXACT>(2.0 * mass * (rho2 - r * drho_dr), d4, in_range);
    const double df_dth = fmks_quot<EXACT>(-2.0 * mass * r * drho_dth, d4, in_range);
    c.g00 = -(1.0 + f);
    c.g01 = f;
    c.g11 = fmks_quot<EXACT>(delta, d2, in_range);
    c.g13 = fmks_quot<EXACT>(a, d2, in_range);
    c.g22 = fmks_quot<EXACT>(1.0, d2, in_range);
    c.g33 = fmks_quot<EXACT>(1.0, fmks_divisor(rho2 * safe_s2), in_range);
    c.A = df_dr;
    c.B = -a * s2 * df_dr;
    c.C = drho_dr;
    c.E = df_dth;
    c.F0 = -a * (s2 * df_dth + ds2_dth * f);
    c.F1 = -a * (ds2_dth * (1.0 + f) + s2 * df_dth);
    c.G = drho_dth;
    const double bracket = rho2 + a2 * s2 * (1.0 + f);
    const double dbr = drho_dr + a2 * s2 * df_dr;
    const double dbt = drho_dth + a2 * (ds2_dth * (1.0 + f) + s2 * df_dth);
    c.D = s2 * dbr;
    c.H = ds2_dth * bracket + s2 * dbt;
    return c;
}

// dx = k, dk = -Gamma(k, k), de_i = -Gamma(k, e_i) in FMKS: vectors go to
// spherical Kerr-Schild components, the spherical connection is contracted
// with p = k fixed, and the second-derivative terms of theta(x1, x2) carry
// the result back (transport_rhs, kerr_fmks.hpp:455-479; fixed-p contraction,
// kerr_schild_spherical.hpp:288-323).
struct FmksConn {
    FmksTheta t;
    SksConn c;
};

KP_HD FmksConn fmks_conn(const FmksParams& m, const D4& x) {
    FmksConn o;
    o.t = fmks_theta(m, x.v[1], x.v[2]);
    double s, c;
    sincos(o.t.th, &s, &c);
    bool in_range = true;
    o.c = sks_conn<true>(m.mass, m.spin, o.t.r, s, c, in_range);
    if (!in_range) o.c = sks_conn<false>(m.mass, m.spin, o.t.r, s, c, in_range);
    return o;
}

// -Gamma(k, q) at a point: the reference's sums without their zero terms, in
// its order.
KP_HD D4 fmks_contract(const FmksConn& w, const D4& kn, const D4& qn) {
    const FmksTheta& t = w.t;
    const SksConn& c = w.c;
    auto to_sph = [&](const D4& v) {
        D4 o;
        o.v[0] = v.v[0];
        o.v[1] = t.r * v.v[1];
        o.v[2] = t.dth1 * v.v[1] + t.dth2 * v.v[2];
        o.v[3] = v.v[3];
        return o;
    };
    auto rows = [&](const D4& v, double (&r)[4], double (&h)[4]) {
        r[0] = c.A * v.v[0] + c.A * v.v[1] + c.B * v.v[3];
        r[1] = r[0];
        r[2] = c.C * v.v[2];
        r[3] = c.B * v.v[0] + c.B * v.v[1] + c.D * v.v[3];
        h[0] = c.E * v.v[0] + c.E * v.v[1] + c.F0 * v.v[3];
        h[1] = c.E * v.v[0] + c.E * v.v[1] + c.F1 * v.v[3];
        h[2] = c.G * v.v[2];
        h[3] = c.F0 * v.v[0] + c.F1 * v.v[1] + c.H * v.v[3];
    };
    const D4 ks = to_sph(kn), q = to_sph(qn);
    double rowk_r[4], rowk_t[4], rr[4], rt[4];
    rows(ks, rowk_r, rowk_t);
    rows(q, rr, rt);
    const double d1 = ks.v[0] * rr[0] + ks.v[1] * rr[1] + ks.v[2] * rr[2] + ks.v[3] * rr[3];
    const double d2 = ks.v[0] * rt[0] + ks.v[1] * rt[1] + ks.v[2] * rt[2] + ks.v[3] * rt[3];
    double tt[4];
    for (int nu = 0; nu < 4; ++nu) {
        double term = ks.v[1] * rr[nu] + q.v[1] * rowk_r[nu] + ks.v[2] * rt[nu] + q.v[2] * rowk_t[nu];
        if (nu == 1) term -= d1;
        else if (nu == 2) term -= d2;
        tt[nu] = term;
    }
    double hs[4];
    hs[0] = 0.5 * (c.g00 * tt[0] + c.g01 * tt[1]);
    hs[1] = 0.5 * (c.g01 * tt[0] + c.g11 * tt[1] + c.g13 * tt[3]);
    hs[2] = 0.5 * (c.g22 * tt[2]);
    hs[3] = 0.5 * (c.g13 * tt[1] + c.g33 * tt[3]);
    // back to native components (fmks_from_spherical_connection_contract, :414-431)
    hs[1] += t.r * kn.v[1] * qn.v[1];
    hs[2] += t.d2th11 * kn.v[1] * qn.v[1] + t.d2th12 * (kn.v[1] * qn.v[2] + kn.v[2] * qn.v[1]) +
             t.d2th22 * kn.v[2] * qn.v[2];
    bool in_range = true;
    const FmksDivisor dr = fmks_divisor(t.r), d2th = fmks_divisor(t.dth2);
    double o1 = fmks_quot<true>(hs[1], dr, in_range);
    double o2 = fmks_quot<true>(hs[2] - fmks_quot<true>(t.dth1 * hs[1], dr, in_range), d2th, in_range);
    if (!in_range) {
        o1 = fmks_quot<false>(hs[1], dr, in_range);
        o2 = fmks_quot<false>(hs[2] - fmks_quot<false>(t.dth1 * hs[1], dr, in_range), d2th, in_range);
    }
    D4 out;
    out.v[0] = -hs[0];
    out.v[1] = -o1;
    out.v[2] = -o2;
    out.v[3] = -hs[3];
    return out;
}

KP_HD Ray fmks_rhs(const FmksParams& m, const Ray& s) {
    const FmksConn w = fmks_conn(m, s.x);
    Ray d;
    d.x = s.k;
    d.k = fmks_contract(w, s.k, s.k);
    d.e1 = fmks_contract(w, s.k, s.e1);
    d.e2 = fmks_contract(w, s.k, s.e2);
    return d;
}

// The same right-hand side in factored form, for the mixed policy: the
// spherical Kerr-Schild derivatives have only seven distinct nonzero
// entries per direction (d/dr g: rows 0 and 1 coincide, A(q0 + q1) + B q3;
// d/dtheta g likewise with two different (0,3)/(1,3) entries), the inverse
// metric five, and the three divisions by rho^2, r and dtheta/dx2 become
// reciprocals.  Same algebra as fmks_rhs, regrouped: agrees to rounding.
struct FmksFactored {
    double r, inv_r, inv_dth2, dth1, dth2, d2th11, d2th12, d2th22;
    double G00, G01, G11, G13, G22, G33;      // inverse spherical metric: g22 and g33 last
    double A, B, C, Dr, E, F0, F1, Gt, Ht;    // d/dr g and d/dtheta g
};

KP_HD FmksFactored fmks_factored_conn(const FmksParams& m, const D4& x) {
    const FmksTheta t = fmks_theta<true>(m, x.v[1], x.v[2]);
    const double a = m.spin, M = m.mass, r = t.r;
    double sn, cs;
    sincos(t.th, &sn, &cs);
    const double a2 = a * a, s2 = sn * sn, safe_s2 = max_val(s2, kTiny);
    const double rho2 = r * r + a2 * cs * cs;
    const double inv_rho2 = kp_recip(rho2);
    const double inv_rho4 = inv_rho2 * inv_rho2;
    const double f = 2.0 * M * r * inv_rho2;
    const double delta = r * r - 2.0 * M * r + a2;
    FmksFactored o;
    o.r = r;
    o.inv_r = kp_recip(r);
    o.inv_dth2 = kp_recip(t.dth2);
    o.dth1 = t.dth1;
    o.dth2 = t.dth2;
    o.d2th11 = t.d2th11;
    o.d2th12 = t.d2th12;
    o.d2th22 = t.d2th22;
    o.G00 = -(1.0 + f);
    o.G01 = f;
    o.G11 = delta * inv_rho2;
    o.G13 = a * inv_rho2;
    o.G22 = inv_rho2;
    o.G33 = inv_rho2 * kp_recip(safe_s2);
    const double drho_dth = -2.0 * a2 * sn * cs, ds2_dth = 2.0 * sn * cs;
    const double df_dr = 2.0 * M * (rho2 - 2.0 * r * r) * inv_rho4;
    const double df_dth = -2.0 * M * r * drho_dth * inv_rho4;
    o.A = df_dr;
    o.B = -a * s2 * df_dr;
    o.C = 2.0 * r;
    o.Dr = s2 * (2.0 * r + a2 * s2 * df_dr);
    o.E = df_dth;
    o.F0 = -a * (s2 * df_dth + ds2_dth * f);
    o.F1 = -a * (ds2_dth * (1.0 + f) + s2 * df_dth);
    o.Gt = drho_dth;
    const double bracket = rho2 + a2 * s2 * (1.0 + f);
    o.Ht = ds2_dth * bracket + s2 * (drho_dth + a2 * (ds2_dth * (1.0 + f) + s2 * df_dth));
    return o;
}

// -Gamma(k, q) at a point.
KP_HD D4 fmks_factored_contract(const FmksFactored& w, const D4& kn, const D4& qn) {
    struct V {
        double v0, v1, v2, v3;
    };
    auto to_sph = [&](const D4& q) { return V{q.v[0], w.r * q.v[1], w.dth1 * q.v[1] + w.dth2 * q.v[2], q.v[3]}; };
    auto drow = [&](const V& q, V& rr, V& rt) {
        const double sig = q.v0 + q.v1;
        rr = V{w.A * sig + w.B * q.v3, w.A * sig + w.B * q.v3, w.C * q.v2, w.B * sig + w.Dr * q.v3};
        rt = V{w.E * sig + w.F0 * q.v3, w.E * sig + w.F1 * q.v3, w.Gt * q.v2, w.F0 * q.v0 + w.F1 * q.v1 + w.Ht * q.v3};
    };
    const V ks = to_sph(kn), q = to_sph(qn);
    V rk, tk, rr, rt;
    drow(ks, rk, tk);
    drow(q, rr, rt);
    const double d1 = ks.v0 * rr.v0 + ks.v1 * rr.v1 + ks.v2 * rr.v2 + ks.v3 * rr.v3;
    const double d2 = ks.v0 * rt.v0 + ks.v1 * rt.v1 + ks.v2 * rt.v2 + ks.v3 * rt.v3;
    const double t0 = ks.v1 * rr.v0 + q.v1 * rk.v0 + ks.v2 * rt.v0 + q.v2 * tk.v0;
    const double t1 = ks.v1 * rr.v1 + q.v1 * rk.v1 + ks.v2 * rt.v1 + q.v2 * tk.v1 - d1;
    const double t2 = ks.v1 * rr.v2 + q.v1 * rk.v2 + ks.v2 * rt.v2 + q.v2 * tk.v2 - d2;
    const double t3 = ks.v1 * rr.v3 + q.v1 * rk.v3 + ks.v2 * rt.v3 + q.v2 * tk.v3;
    const double h0 = 0.5 * (w.G00 * t0 + w.G01 * t1);
    double h1 = 0.5 * (w.G01 * t0 + w.G11 * t1 + w.G13 * t3);
    double h2 = 0.5 * (w.G22 * t2);
    const double h3 = 0.5 * (w.G13 * t1 + w.G33 * t3);
    h1 += w.r * kn.v[1] * qn.v[1];
    h2 += w.d2th11 * kn.v[1] * qn.v[1] + w.d2th12 * (kn.v[1] * qn.v[2] + kn.v[2] * qn.v[1]) +
          w.d2th22 * kn.v[2] * qn.v[2];
    const double h1r = h1 * w.inv_r;
    D4 out;
    out.v[0] = -h0;
    out.v[1] = -h1r;
    out.v[2] = -((h2 - w.dth1 * h1r) * w.inv_dth2);
    out.v[3] = -h3;
    return out;
}

KP_HD Ray fmks_rhs_factored(const FmksParams& m, const Ray& s) {
    const FmksFactored w = fmks_factored_conn(m, s.x);
    Ray d;
    d.x = s.k;
    d.k = fmks_factored_contract(w, s.k, s.k);
    d.e1 = fmks_factored_contract(w, s.k, s.e1);
    d.e2 = fmks_factored_contract(w, s.k, s.e2);
    return d;
}

// Camera at phi = 0 and its ipole tetrad in FMKS (camera.hpp:302-456): the
// normal observer, the raised centering covector (1, 1, 0, 0), and the native
// trial vectors (0, 0, 1, 0), (1, 1, 1, 1), made orthonormal by Gram-Schmidt.
// Evaluated once per image (host side).
KP_HD void fmks_camera_frame(const FmksParams& m, double radius, double inclination, D4& x, D4& e0, D4& e1,
                             D4& e2, D4& e3) {
    const double x1 = log(max_val(radius, kTiny));
    x = D4{{0.0, x1, fmks_x2_of(m, x1, inclination), 0.0}};
    double g[4][4], gi[4][4];
    fmks_gcov(m, x, g);
    fmks_gcon(m, x, gi);
    auto dot = [&](const D4& u, const D4& v) { return dot_gm(g, u, v); };
    auto scale = [](D4 v, double s) {
        for (int i = 0; i < 4; ++i) v.v[i] *= s;
        return v;
    };
    auto proj = [&](D4 a, const D4& b) {
        const double b2 = dot(b, b);
        if (abs_val(b2) > kTiny) {
            const double k = dot(a, b) / b2;
            for (int i = 0; i < 4; ++i) a.v[i] -= b.v[i] * k;
        }
        return a;
    };
    auto norm = [&](const D4& v) { return scale(v, 1.0 / sqrt(max_val(abs_val(dot(v, v)), kTiny))); };
    // normal observer: u^mu = -g^{mu 0}, normalised
    D4 u;
    for (int i = 0; i < 4; ++i) u.v[i] = -gi[i][0];
    const double n2 = dot(u, u);
    if (n2 < 0.0) u = scale(u, 1.0 / sqrt(-n2));
    e0 = u;
    const double cov[4] = {1.0, 1.0, 0.0, 0.0};
    for (int i = 0; i < 4; ++i) {
        double sum = 0.0;
        for (int j = 0; j < 4; ++j) sum += gi[i][j] * cov[j];
        e3.v[i] = sum;
    }
    e2 = D4{{0.0, 0.0, 1.0, 0.0}};
    e1 = D4{{1.0, 1.0, 1.0, 1.0}};
    e0 = norm(e0);
    e3 = proj(e3, e0);
    e3 = proj(e3, e0);
    e3 = norm(e3);
    e2 = proj(e2, e0);
    e2 = proj(e2, e3);
    e2 = proj(e2, e0);
    e2 = proj(e2, e3);
    e2 = norm(e2);
    e1 = proj(e1, e0);
    e1 = proj(e1, e2);
    e1 = proj(e1, e3);
    e1 = proj(e1, e0);
    e1 = proj(e1, e2);
    e1 = proj(e1, e3);
    e1 = norm(e1);
    // orientation: the Levi-Civita sign of (e0, e1, e2, e3)
    const double orient = tetrad_orientation(e0, e1, e2, e3);
    if (orient < 0.0) e1 = scale(e1, -1.0);
}

}  // namespace kp
