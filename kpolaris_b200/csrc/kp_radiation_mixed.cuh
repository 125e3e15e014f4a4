// kp_radiation_mixed.cuh -- the radiation side of the mixed policy: RIAF plasma
// state, thermal synchrotron coefficients and the Strang transfer step, with
// the formulas of kp_radiation.cuh (and the reference's
// src/model/riaf.hpp:54-549, src/radiation/thermal_synchrotron.hpp:60-627,
// src/radiation/semi_analytic.hpp:10-100) factored for throughput: every power
// of an argument from one logarithm, refined hardware reciprocals and square
// roots, dot products through the Kerr-Schild vector, frequency-independent
// factors once per sample, the Bessel K ratios without their common
// e^-x / sqrt(x).
//
// All of it is FP64.  A Faraday-thick ray turns its polarisation through
// thousands of radians, and powers of two of its depths decide how its steps
// are cut: coefficients in single precision put 1e-6 into Stokes I, up to 1e-3
// into Q and U, and let one image in a few lose a pixel to a decision that
// fell the other way.  On quads the difference in time is a tenth of near-B.
//
// Emission and the Stokes vector carry a per-image, per-frequency factor 2^E
// (the transfer equation is linear in (j, S)); the image is unscaled at the end.
#pragma once

#include "kp_geometry_mixed.cuh"

namespace kp {

namespace mixc {
constexpr double kPiD = 3.141592653589793;
constexpr double kEE = 4.803204712570263e-10;
constexpr double kME = 9.1093837015e-28;
constexpr double kCL = 2.99792458e10;
constexpr double kHPL = 6.62607015e-27;
constexpr double kMP = 1.67262192369e-24;
// Pandya emission: e^2 / c times the cyclotron frequency per gauss; sqrt(2) pi / 27
constexpr double kPandyaPref = kEE * kEE / kCL * (kEE / (2.0 * kPiD * kME * kCL));
constexpr double kTerm1 = 1.4142135623730951 * kPiD / 27.0;
// h / (m_e c^2) and c^2 / (2 h)
constexpr double kHOverMc2 = kHPL / (kME * kCL * kCL);
constexpr double kC2Over2h = kCL * kCL / (2.0 * kHPL);
// Dexter: 3 e / (4 pi m_e c); Pandya: 2/9 of the cyclotron frequency
constexpr double kDexNus = 3.0 * kEE / (4.0 * kPiD * kME * kCL);
constexpr double kPandyaNus = 2.0 / 9.0 * kEE / (2.0 * kPiD * kME * kCL);
// Dexter prefactors e^2 / (2 sqrt(3) c) and 2 e^2 / (3 sqrt(3) c)
constexpr double kDexPref = kEE * kEE / (2.0 * 1.7320508075688772 * kCL);
constexpr double kDexPrefV = 2.0 * kEE * kEE / (3.0 * 1.7320508075688772 * kCL);
// (x / Theta_e)^2 of the Faraday fits: sqrt(2) 1e3 omega0 / (2 pi nu) per gauss and 1 / nu
constexpr double kFaradayX2 = 1.4142135623730951 * 1e3 * kEE / (kME * kCL) / (2.0 * kPiD);
// rho_V nu = (4 pi e^2 / m_e) (e / (m_e c)) n_e B cos(theta) / (4 pi^2 c nu) x fit
constexpr double kRhoV = (4.0 * kPiD * kEE * kEE / kME) * (kEE / (kME * kCL)) / (4.0 * kPiD * kPiD * kCL);
// rho_Q nu = (4 pi e^2 / m_e) (e / (m_e c))^2 n_e B^2 sin^2(theta) / (2^4 pi^3 c nu^2) x fit
constexpr double kRhoQ = (4.0 * kPiD * kEE * kEE / kME) * (kEE / (kME * kCL)) * (kEE / (kME * kCL)) * kPiD /
                         (16.0 * kPiD * kPiD * kPiD * kPiD * kCL);
}  // namespace mixc

using CoeffsM = Coeffs<double>;

// K0/K2 and K1/K2 for x = 1/Theta_e with the polynomial fits of
// thermal_synchrotron.hpp:108-158; for x > 2 the factor e^-x / sqrt(x) cancels.
KP_HD void bessel_ratios(double x, double lg, double& r0, double& r1) {  // lg = log(x / 2)
    double p, q;
    if (x <= 2.0) {
        const double y = x * x * 0.25;
        const double t = y * (4.0 / (3.75 * 3.75));
        double i0 = 0.0045813;
        i0 = 0.0360768 + t * i0;
        i0 = 0.2659732 + t * i0;
        i0 = 1.2067492 + t * i0;
        i0 = 3.0899424 + t * i0;
        i0 = 3.5156229 + t * i0;
        i0 = 1.0 + t * i0;
        double i1 = 0.00032411;
        i1 = 0.00301532 + t * i1;
        i1 = 0.02658733 + t * i1;
        i1 = 0.15084934 + t * i1;
        i1 = 0.51498869 + t * i1;
        i1 = 0.87890594 + t * i1;
        i1 = x * (0.5 + t * i1);
        double a = 0.00000740;
        a = 0.00010750 + y * a;
        a = 0.00262698 + y * a;
        a = 0.03488590 + y * a;
        a = 0.23069756 + y * a;
        a = 0.42278420 + y * a;
        a = -0.57721566 + y * a;
        p = a - lg * i0;
        double b = -0.00004686;
        b = -0.00110404 + y * b;
        b = -0.01919402 + y * b;
        b = -0.18156897 + y * b;
        b = -0.67278579 + y * b;
        b = 0.15443144 + y * b;
        b = 1.0 + y * b;
        q = lg * i1 + b * kp_recip(x);
    } else {
        const double y = 2.0 * kp_recip(x);
        double a = 0.00053208;
        a = -0.00251540 + y * a;
        a = 0.00587872 + y * a;
        a = -0.01062446 + y * a;
        a = 0.02189568 + y * a;
        a = -0.07832358 + y * a;
        p = 1.25331414 + y * a;
        double b = -0.00068245;
        b = 0.00325614 + y * b;
        b = -0.00780353 + y * b;
        b = 0.01504268 + y * b;
        b = -0.03655620 + y * b;
        b = 0.23498619 + y * b;
        q = 1.25331414 + y * b;
    }
    const double k2 = p + 2.0 * q * kp_recip(x);
    const double inv = k2 > 0.0 ? kp_recip(k2) : 0.0;
    r0 = k2 > 0.0 ? p * inv : 1.0;
    r1 = k2 > 0.0 ? q * inv : 1.0;
}

// Plasma state at a sample point, with the frequency-independent factors of
// the thermal fits (riaf_sample_thermal_m).
struct RiafSampleM {
    double ne, thetae, b, nu_fluid, cos_theta, sin_theta;
    double unused;  // without this slot near-B of slow light spills 440 instead of 332 B (72 x 50: 32.5 / 31.6 ms)
    double cos2chi, sin2chi;
    double xs0;     // argument of the emission fit, over the frequency in hertz
    double xf0;     // argument of the Faraday fits times the root of the frequency
    double rv0;     // rho_V nu times the frequency, without the fit's logarithm
    double rq0;     // rho_Q nu times the frequency squared, without the fit's function of x
    double pref;    // emission prefactor
    double qterm;   // (7 T^0.96 + 35) / (10 T^0.96 + 75), Pandya jQ
    double vt1;     // (37 - 87 sin(theta - 0.45)) / (100 (T + 1)), Pandya jV
    double vt2a;    // T^0.6 / 25 + 0.7, Pandya jV
    int emitting, on_axis, has_chi;
};

// Cube root of x > 0: Newton's step in FP64 from a single-precision start, whose
// relative error it squares: 3e-13 for x in 1..1e7, 7e-12 over the whole range.
// The fits take exp(-x^(1/3)): an error of the root is multiplied by the root
// there.
KP_HD double cube_root(double x) {
    if (!(x > 1e-30 && x < 1e30)) return cbrt(x);
#ifdef __CUDA_ARCH__
    const double y = double(exp2f(__log2f(float(x)) * (1.0f / 3.0f)));
#else
    const double y = double(cbrtf(float(x)));
#endif
    const double y2 = y * y;
    return y - (y2 * y - x) * kp_recip(3.0 * y2);
}

// Frequency-independent factors of the thermal fits at one sample
// (thermal_synchrotron.hpp:312-395, 462-506), evaluated once per sample
// instead of once per frequency.  lt = log(Theta_e).
KP_HD void riaf_sample_thermal_m(const ImageConsts& c, RiafSampleM& p, double lt) {
    const double te = p.thetae, st = max_val(p.sin_theta, c.min_sin_theta);
    const double inv_nu = kp_recip(p.nu_fluid);
    double r0, r1;
    bessel_ratios(kp_recip(te), -lt - 0.69314718055994530942, r0, r1);
    p.rv0 = mixc::kRhoV * p.ne * p.b * r0 * p.cos_theta * inv_nu;
    p.rq0 = mixc::kRhoQ * p.ne * (p.b * p.b) * (r1 + 6.0 * te) * (st * st) * (inv_nu * inv_nu);
    {
        double g, inv;
        kp_sqrt_pair(max_val(mixc::kFaradayX2 * st * p.b * inv_nu, 1e-200), g, inv);
        p.xf0 = te * g;
    }
    const double nus = c.fit == 4 ? mixc::kDexNus * p.b * st * te * te + 1.0 : mixc::kPandyaNus * p.b * st * te * te;
    p.xs0 = p.nu_fluid * kp_recip(max_val(nus, 1e-200));
    p.qterm = p.vt1 = p.vt2a = 0.0;
    if (c.fit == 4) {
        p.pref = p.ne * kp_recip(te * te);
        return;
    }
    p.pref = mixc::kPandyaPref * p.ne * p.b;
    const double t2425 = exp(0.96 * lt);
    p.qterm = (7.0 * t2425 + 35.0) * kp_recip(10.0 * t2425 + 75.0);
    const double sin_shift = st * 0.4356824462767121 - p.cos_theta * 0.9001004421765051;
    p.vt1 = (37.0 - 87.0 * sin_shift) * kp_recip(100.0 * (te + 1.0));
    p.vt2a = exp(0.6 * lt) * 0.04 + 0.7;
}

KP_HD void riaf_sample_thermal_m(const ImageConsts& c, RiafSampleM& p) { riaf_sample_thermal_m(c, p, log(p.thetae)); }

// Boyer-Lindquist metric entries at (r, theta) with unit mass, FP64.
struct BlEntries {
    double tt, tp, pp, rr;      // covariant
    double itt, itp, ipp, irr;  // contravariant
};

KP_HD BlEntries bl_entries(double r, double s2, double c2, double a) {
    const double a2 = a * a, ra = r * r + a2;
    const double sigma = r * r + a2 * c2, delta = ra - 2.0 * r;
    const double i_s = kp_recip(sigma), i_d = kp_recip(max_val(delta, 1e-30));
    const double f = 2.0 * r * i_s, i_sd = i_s * i_d;
    BlEntries m;
    m.tt = f - 1.0;
    m.tp = -a * f * s2;
    m.pp = (ra + a2 * f * s2) * s2;
    m.rr = sigma * i_d;
    m.itt = -(ra * ra - a2 * delta * s2) * i_sd;
    m.itp = -2.0 * a * r * i_sd;
    m.ipp = (delta - a2 * s2) * i_sd * kp_recip(s2);
    m.irr = delta * i_s;
    return m;
}

// riaf_sample (kp_radiation.cuh) for the mixed policy.
// With the Kerr-Schild vector l = (1, l1, l2, l3) at the point, g = eta + f l l,
// so a dot product is eta(u, v) + f (l.u)(l.v) with l.u formed once per
// vector; (l1, l2) = sin(theta) (cos phi, sin phi) gives the BL angles, and
// the azimuthal vector is (0, -y, x, 0).
KP_HD RiafSampleM riaf_sample_m(const ImageConsts& c, const Ray& s) {
    RiafSampleM out;
    out.emitting = 0;
    out.on_axis = 0;
    out.has_chi = 0;
    const double a = c.spin, a2 = a * a;
    const double x = s.x.v[1], y = s.x.v[2], z = s.x.v[3];
    const double sqsum = x * x + y * y + z * z - a2;
    double discr, inv_discr, r, inv_r;
    kp_sqrt_pair(sqsum * sqsum + 4.0 * a2 * z * z, discr, inv_discr);
    kp_sqrt_pair(max_val(0.5 * (sqsum + discr), 1e-30), r, inv_r);
    const double r_bl = max_val(r, c.min_radius);
    if (r_bl <= c.horizon + c.horizon_buffer || r_bl < c.r_min || r_bl > c.r_max) return out;
    const double r2 = r * r, inv_rp = kp_recip(r2 + a2);
    const double l1 = (r * x + a * y) * inv_rp, l2 = (r * y - a * x) * inv_rp, l3 = z * inv_r;
    const double c2 = min_val(l3 * l3, 1.0), s2 = max_val((x * x + y * y) * inv_rp, 1e-30);
    const double amp = 2.0 * c.mass * r2 * r * kp_recip(r2 * r2 + a2 * z * z);
    // n_e, Theta_e and B (riaf.hpp:54-96)
    double ne, thetae, b, lt;
    {
        const double lr = log(r_bl);
        const double h = max_val(c.disk_h, 1e-6);
        const double rcyl2 = max_val(r_bl * r_bl * s2, c.min_radius * c.min_radius);
        const double zc = r_bl * l3;
        ne = c.nth0 * exp(c.pow_nth * lr - zc * zc * kp_recip(2.0 * rcyl2 * h * h));
        if (!(ne > 0.0)) return out;
        ne *= c.ne_unit;
        lt = c.log_te0 + c.pow_T * lr;
        thetae = exp(lt);
        if (!(thetae > c.min_thetae)) {
            thetae = c.min_thetae;
            lt = log(thetae);
        }
        const double kb = 8.0 * 3.141592653589793 * 0.1 * mixc::kMP * mixc::kCL * mixc::kCL / 6.0;
        double inv;
        kp_sqrt_pair(max_val(kb * ne * kp_recip(r_bl), 1e-24), b, inv);
    }
    out.emitting = 1;
    out.ne = ne;
    out.thetae = thetae;
    out.b = b;
    // fluid velocity (riaf.hpp:206-273): circular, with the plunge inside the ISCO
    double vt = 1.0, vr = 0.0, vphi = 0.0;
    {
        const double rr = r_bl;
        const BlEntries m = bl_entries(rr, s2, c2, a);
        const double kf = c.keplerian_factor, inf = c.infall_factor;
        if (rr < c.horizon) {
            vt = kp_recip(sqrt(max_val(-m.itt, 1e-30)));
        } else {
            double omega;
            const bool plunge = rr < c.isco;
            if (plunge) {
                const double ri = c.isco;
                const BlEntries mi = bl_entries(ri, s2, c2, a);
                const double oi = kp_recip(ri * sqrt(ri) + a);
                const double qi = mi.tt + 2.0 * oi * mi.tp + oi * oi * mi.pp;
                const double ut = kp_recip(sqrt(max_val(-qi, 1e-30)));
                const double e = (mi.tt + mi.tp * oi) * ut, l = (mi.tp + mi.pp * oi) * ut;
                const double kc = m.itt * e * e + 2.0 * m.itp * e * l + m.ipp * l * l;
                vr = -m.irr * sqrt(max_val(-(1.0 + kc) * kp_recip(max_val(m.irr, 1e-30)), 0.0));
                omega = (m.itp * e + m.ipp * l) * kp_recip(max_val(m.itt * e + m.itp * l, 1e-30));
            } else {
                double sr, isr;
                kp_sqrt_pair(rr, sr, isr);
                omega = kp_recip(rr * sr + a);
            }
            if (kf != 1.0) {
                const double g = m.itt;
                const double off = m.itp * kp_recip(abs_val(g) > 1e-30 ? g : (g < 0.0 ? -1e-30 : 1e-30));
                omega = omega + (1.0 - kf) * (off - omega);
            }
            if (inf != 0.0) {
                const double ff = -sqrt(max_val(-(1.0 + m.itt) * m.irr, 0.0));
                vr = plunge ? vr + inf * (ff - vr) : inf * ff;
            }
            const double q = m.tt + 2.0 * omega * m.tp + omega * omega * m.pp;
            double inv;
            kp_sqrt_pair(max_val(-(1.0 + vr * vr * m.rr) * kp_recip(q), 1e-60), vt, inv);
            vphi = omega * vt;
        }
        const double i_d = kp_recip(max_val(rr * rr - 2.0 * rr + a2, 1e-30));
        vt += 2.0 * rr * i_d * vr;
        vphi += a * i_d * vr;
    }
    struct Vec {
        double t, x, y, z, l;
    };
    auto vec = [&](double t, double vx, double vy, double vz) {
        return Vec{t, vx, vy, vz, t + l1 * vx + l2 * vy + l3 * vz};
    };
    auto dot = [&](const Vec& u, const Vec& v) {
        return u.x * v.x + u.y * v.y + u.z * v.z - u.t * v.t + amp * u.l * v.l;
    };
    Vec u = vec(vt, vr * l1 - vphi * y, vr * l2 + vphi * x, vr * l3);
    {
        const double n2 = dot(u, u);
        if (n2 < 0.0) {
            double n, inv;
            kp_sqrt_pair(max_val(-n2, 1e-30), n, inv);
            u = Vec{u.t * inv, u.x * inv, u.y * inv, u.z * inv, u.l * inv};
        }
    }
    const Vec k = vec(s.k.v[0], s.k.v[1], s.k.v[2], s.k.v[3]);
    const double uk = dot(u, k);
    const double nu_fluid = max_val(abs_val(uk), c.min_frequency_scale);
    // toroidal field unit vector, normal to u
    Vec bv;
    double bsq;
    auto project = [&](const Vec& t) {
        const double ub = dot(u, t);
        bv = Vec{t.t + u.t * ub, t.x + u.x * ub, t.y + u.y * ub, t.z + u.z * ub, t.l + u.l * ub};
        bsq = dot(bv, bv);
    };
    project(vec(0.0, -y, x, 0.0));
    if (!(bsq > 1e-30)) project(vec(0.0, 0.0, 0.0, 1.0));
    if (!(bsq > 1e-30)) project(vec(0.0, 1.0, 0.0, 0.0));
    if (bsq > 1e-30) {
        double n, inv;
        kp_sqrt_pair(bsq, n, inv);
        bv = Vec{bv.t * inv, bv.x * inv, bv.y * inv, bv.z * inv, bv.l * inv};
    }
    const double kb = dot(k, bv);
    const double ct = min_val(max_val(kb * kp_recip(max_val(nu_fluid, 1e-30)), -1.0), 1.0);
    out.nu_fluid = nu_fluid;
    out.cos_theta = ct;
    {
        double st, inv;
        kp_sqrt_pair(max_val(1.0 - ct * ct, 1e-60), st, inv);
        out.sin_theta = max_val(st, c.min_sin_theta);
    }
    riaf_sample_thermal_m(c, out, lt);
    if (ct >= 1.0 || ct <= -1.0) {
        out.on_axis = 1;
        return out;
    }
    // screen projections of b (riaf.hpp:320-336) with eK = -k / (u.k) - u
    const Vec e1 = vec(s.e1.v[0], s.e1.v[1], s.e1.v[2], s.e1.v[3]);
    const Vec e2 = vec(s.e2.v[0], s.e2.v[1], s.e2.v[2], s.e2.v[3]);
    double b1 = dot(e1, bv), b2 = dot(e2, bv);
    if (abs_val(uk) > 1e-30) {
        const double iu = -kp_recip(uk);
        const double ub = dot(u, bv), Kb = kb * iu - ub;
        const double ue1 = dot(u, e1), ue2 = dot(u, e2);
        b1 += ue1 * ub - (dot(k, e1) * iu - ue1) * Kb;
        b2 += ue2 * ub - (dot(k, e2) * iu - ue2) * Kb;
    }
    const double bproj2 = b1 * b1 + b2 * b2;
    if (bproj2 > 1e-30) {
        const double inv = kp_recip(bproj2);
        out.has_chi = 1;
        out.cos2chi = (b2 * b2 - b1 * b1) * inv;
        out.sin2chi = -2.0 * b1 * b2 * inv;
    }
    return out;
}

// Thermal coefficients at one frequency (in GHz), emission scaled by 2^E
// (`escale`).
KP_HD CoeffsM riaf_coefficients_m(const ImageConsts& c, const RiafSampleM& p, double freq_ghz, double escale) {
    CoeffsM o = {};
    if (!p.emitting) return o;
    const double freq = freq_ghz * 1e9;
    double sf, isf;
    kp_sqrt_pair(freq, sf, isf);
    const double inv_freq = isf * isf;
    // Faraday rotation and conversion (symphony_rho_QV), invariant rho nu
    const double x = max_val(p.xf0 * isf, 1e-12);
    const double rV = p.rv0 * (1.0 - 0.11 * log(1.0 + 0.035 * x)) * inv_freq;
    if (p.on_axis) {
        o.rV = c.faraday_scale * rV;
        return o;
    }
    double rQ;
    {
        const double lx = log(x);
        double j = 2.011 * exp(exp(1.035 * lx) * (-1.0 / 4.7));
        const double e12 = exp(1.2 * lx) * (-1.0 / 2.73);
        if (e12 > -60.0) j -= cos(0.5 * x) * exp(e12);
        const double e47 = 0.011 * exp(x * (-1.0 / 47.2));
        j -= e47;
        // 0.5 + 0.5 tanh(z) = 1 / (1 + e^-2z); below z = -20 it is under 1e-17
        const double z2 = 20.0 * (lx - 4.787491742782046);
        if (z2 > -40.0) j += (e47 - 369.69342869090815 * exp((-8.0 / 3.0) * lx)) * kp_recip(1.0 + exp(-z2));
        rQ = p.rq0 * j * (inv_freq * inv_freq);
    }
    // emissivities j / nu^2, scaled by 2^E
    const double nu = max_val(freq * p.nu_fluid, 1.0);
    const double inv_nu2 = escale * kp_recip(nu * nu);
    const double xs = max_val(p.xs0 * freq, 1e-200), root = cube_root(xs);
    double jI, jQ, jV;
    if (c.fit == 4) {
        const double inv_root = kp_recip(root), inv2 = inv_root * inv_root;
        const double shape = exp(-1.8899 * root);
        const double pref = mixc::kDexPref * p.pref * nu * shape * inv_nu2;
        jI = pref * (2.5651 * (1.0 + 1.92 * inv_root + 0.9977 * inv2));
        jQ = pref * (2.5651 * (1.0 + 0.93193 * inv_root + 0.499873 * inv2));
        const double iv = 1.81384 * (inv2 * inv_root) + 3.42319 * inv2 + 0.0292545 * sqrt(inv2 * inv_root) + 2.03773 * inv_root;
        double cft = p.cos_theta;
        if (abs_val(cft) < 1e-10) cft = cft >= 0.0 ? 1e-10 : -1e-10;
        const double st = max_val(p.sin_theta, c.min_sin_theta);
        jV = mixc::kDexPrefV * p.pref * nu * cft * kp_recip(st * p.thetae) * iv * shape * inv_nu2;
    } else {
        double sx, isx, sr, isr;
        kp_sqrt_pair(xs, sx, isx);
        kp_sqrt_pair(root, sr, isr);
        const double st = max_val(p.sin_theta, c.min_sin_theta);
        const double pref = p.pref * exp(-root) * inv_nu2, lin = pref * mixc::kTerm1 * st;
        const double bend = 1.8877486253633869933 * sr;
        const double hi = sx + bend, hq = sx + p.qterm * bend;
        jI = lin * (hi * hi);
        jQ = lin * (hq * hq);
        const double v = 1.0 + p.vt2a * exp(0.36 * log(xs)), rv = cube_root(v);
        jV = pref * p.vt1 * (v * (rv * rv));
    }
    // polarisation cap (thermal_synchrotron.hpp:575-588)
    const double jp2 = jQ * jQ + jV * jV, mpf = max_val(c.max_pol_frac, 1e-30);
    if (jI > 0.0 && jp2 > 0.0 && jI * jI * (mpf * mpf) < jp2) {
        const double sc = jI * c.max_pol_frac / sqrt(jp2);
        jQ *= sc;
        jV *= sc;
    }
    // Kirchhoff: a = j / B_nu, with B_nu = 2 h nu^3 / (c^2 (e^x - 1)) and the
    // reference's series for small x
    const double xb = mixc::kHOverMc2 * nu * kp_recip(p.thetae);
    const double em1 = xb < 2e-3 ? xb * (1.0 / 24.0) * (24.0 + xb * (12.0 + xb * (4.0 + xb))) : exp(xb) - 1.0;
    const double fac = mixc::kC2Over2h * em1 * kp_recip(escale) * c.absorption_scale;
    const double es = c.emission_scale, fs = c.faraday_scale;
    o.jI = es * jI;
    o.jV = es * jV;
    o.aI = fac * jI;
    o.aV = fac * jV;
    o.rV = fs * rV;
    if (p.has_chi) {
        o.jQ = es * jQ * p.cos2chi;
        o.jU = es * jQ * p.sin2chi;
        o.aQ = fac * jQ * p.cos2chi;
        o.aU = fac * jQ * p.sin2chi;
        o.rQ = fs * rQ * p.cos2chi;
        o.rU = fs * rQ * p.sin2chi;
    }
    return o;
}

// ---- transfer -----------------------------------------------------------
struct StokesM {
    double I, Q, U, V;  // scaled by 2^E
};

// e^-x - 1 and (1 - e^-x) / kappa for x = kappa dl.
KP_HD void fade_and_source(double kappa, double dl, double& em1, double& src) {
    const double x = kappa * dl;
    if (fabs(x) < 0.0625) {
        // (1 - e^-x) / x to the x^8 term
        double p = -1.0 / 362880.0 * x + 1.0 / 40320.0;
        p = 1.0 / 5040.0 - x * p;
        p = 1.0 / 720.0 - x * p;
        p = 1.0 / 120.0 - x * p;
        p = 1.0 / 24.0 - x * p;
        p = 1.0 / 6.0 - x * p;
        p = 0.5 - x * p;
        p = 1.0 - x * p;
        src = dl * p;
        em1 = -x * p;
        return;
    }
    em1 = x > 700.0 ? -1.0 : expm1(-x);
    src = -em1 / kappa;
}

// The Faraday rotation of one half step: axis n, sin and 1 - cos of its
// angle |rho| dl / 2, from the half angle reduced by its period pi.  Both half
// steps of a Strang step are this rotation.
struct RotationM {
    double nx, ny, nz, st, omc;
    int none;
};

KP_HD void kp_sincospi(double u, double* s, double* c) {
#ifdef __CUDA_ARCH__
    sincospi(u, s, c);
#else
    *s = sin(3.14159265358979323846 * u);
    *c = cos(3.14159265358979323846 * u);
#endif
}

KP_HD RotationM faraday_rotation(const CoeffsM& c, double dl) {
    RotationM r;
    const double rq = c.rQ, ru = c.rU, rv = c.rV;
    const double n2 = rq * rq + ru * ru + rv * rv;
    r.none = !(n2 > 0.0) || dl == 0.0;
    if (r.none) return r;
    double n, inv;
    if (n2 > 1e-280 && n2 < 1e280) {
        kp_sqrt_pair(n2, n, inv);
    } else {
        n = sqrt(n2);
        inv = 1.0 / n;
    }
    r.nx = rq * inv;
    r.ny = ru * inv;
    r.nz = rv * inv;
    double sh, ch;
    kp_sincospi(n * dl * (0.25 / 3.14159265358979323846), &sh, &ch);
    r.st = 2.0 * sh * ch;
    r.omc = 2.0 * sh * sh;
    return r;
}

// P + (n x P) sin + (n (n.P) - P) (1 - cos)
KP_HD void faraday_rotate(StokesM& s, const RotationM& r) {
    if (r.none) return;
    const double px = s.Q, py = s.U, pz = s.V;
    const double f = r.nx * px + r.ny * py + r.nz * pz;
    s.Q = px + ((r.ny * pz - r.nz * py) * r.st + (r.nx * f - px) * r.omc);
    s.U = py + ((r.nz * px - r.nx * pz) * r.st + (r.ny * f - py) * r.omc);
    s.V = pz + ((r.nx * py - r.ny * px) * r.st + (r.nz * f - pz) * r.omc);
}

KP_HD void absorb_emit(StokesM& s, const CoeffsM& c, double dl) {
    const double aq = c.aQ, au = c.aU, av = c.aV, ai = c.aI;
    const double jq = c.jQ, ju = c.jU, jv = c.jV, ji = c.jI;
    const double n2 = aq * aq + au * au + av * av;
    double em, src;
    fade_and_source(ai, dl, em, src);
    if (n2 < 1e-60) {
        s.I = s.I + (em * s.I + src * ji);
        s.Q = s.Q + (em * s.Q + src * jq);
        s.U = s.U + (em * s.U + src * ju);
        s.V = s.V + (em * s.V + src * jv);
        return;
    }
    double an, inv;
    kp_sqrt_pair(n2, an, inv);
    const double nx = aq * inv, ny = au * inv, nz = av * inv;
    const double par = nx * s.Q + ny * s.U + nz * s.V;
    const double jpar = nx * jq + ny * ju + nz * jv;
    double emp, srcp, emm, srcm;
    fade_and_source(ai + an, dl, emp, srcp);
    fade_and_source(ai - an, dl, emm, srcm);
    // changes of I + P_par, I - P_par and of the part of P across n
    const double dp = emp * (s.I + par) + srcp * (ji + jpar);
    const double dm = emm * (s.I - par) + srcm * (ji - jpar);
    const double dpar = 0.5 * (dp - dm);
    s.I += 0.5 * (dp + dm);
    s.Q += nx * dpar + (em * (s.Q - nx * par) + src * (jq - nx * jpar));
    s.U += ny * dpar + (em * (s.U - ny * par) + src * (ju - ny * jpar));
    s.V += nz * dpar + (em * (s.V - nz * par) + src * (jv - nz * jpar));
}

KP_HD void stokes_step_m(StokesM& s, const CoeffsM& c, double dl) {
    const RotationM r = faraday_rotation(c, dl);
    faraday_rotate(s, r);
    absorb_emit(s, c, dl);
    faraday_rotate(s, r);
}

}  // namespace kp
