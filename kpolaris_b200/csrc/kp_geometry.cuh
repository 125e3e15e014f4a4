// kp_geometry.cuh -- Kerr spacetime in Cartesian Kerr-Schild coordinates and
// the transport right-hand side, FP64.
//
// The metric is g = eta + f l (x) l (src/geometry/kerr_schild_cartesian.hpp:19-51).
// The connection is never formed: Gamma(p, q) is contracted directly from
// (f, df, l, dl) as the reference's specialised transport_rhs does
// (kerr_schild_cartesian.hpp:194-363).  The expressions keep the reference's
// IEEE operation order (compiled with --fmad=false in the FP64 kernels) so
// integer outputs (termination, step counts) are bit-identical to its CPU run.
#pragma once

#include "kp_common.cuh"
#include "kp_exact.cuh"

namespace kp {

KP_HD D4 d4(double a, double b, double c, double d) {
    D4 o;
    o.v[0] = a;
    o.v[1] = b;
    o.v[2] = c;
    o.v[3] = d;
    return o;
}

KP_HD D4 d4_scale(const D4& a, double s) {
    return d4(a.v[0] * s, a.v[1] * s, a.v[2] * s, a.v[3] * s);
}

KP_HD D4 d4_sub_scaled(const D4& a, const D4& b, double s) {
    return d4(a.v[0] - b.v[0] * s, a.v[1] - b.v[1] * s, a.v[2] - b.v[2] * s, a.v[3] - b.v[3] * s);
}


// Radius only: the `r` of KerrSchildInMetric::build_work (:27-40).
KP_HD double ks_radius(double spin, const D4& X) {
    const double x = X.v[1], y = X.v[2], z = X.v[3];
    const double a2 = spin * spin;
    const double radius2 = x * x + y * y + z * z;
    const double sqsum = radius2 - a2;
    const double v = sqsum * sqsum + 4.0 * a2 * z * z;
#ifdef __CUDA_ARCH__
    if (v > 1e-200 && v < 1e200) {
        const double r2x = 0.5 * (sqsum + exact_sqrt(v));
        if (r2x > 1e-200) return exact_sqrt(r2x);
    }
#endif
    const double discr = sqrt(v);
    const double r2 = 0.5 * (sqsum + discr);
    return sqrt(max_val(r2, kTiny));
}

// f and l of the Kerr-Schild form (build_work, :27-51).
struct KSMetricPoint {
    double amp;
    double l[4];
};

KP_HD KSMetricPoint ks_point(double mass, double spin, const D4& X) {
    const double x = X.v[1], y = X.v[2], z = X.v[3];
    const double a = spin;
    const double a2 = spin * spin;
    const double radius2 = x * x + y * y + z * z;
    const double sqsum = radius2 - a2;
    const double discr = sqrt(sqsum * sqsum + 4.0 * a2 * z * z);
    const double r2 = 0.5 * (sqsum + discr);
    const double r = sqrt(max_val(r2, kTiny));
    const double denom = r2 * r2 + a2 * z * z;
    KSMetricPoint p;
    const double r2pa2 = r2 + a2;
    p.l[0] = 1.0;
#ifdef __CUDA_ARCH__
    double amp[1] = {2.0 * mass * r2 * r}, l12[2] = {r * x + a * y, r * y - a * x}, l3[1] = {z};
    exact_quots(amp, denom);
    exact_quots(l12, r2pa2);
    exact_quots(l3, r);
    p.amp = amp[0];
    p.l[1] = l12[0];
    p.l[2] = l12[1];
    p.l[3] = l3[0];
#else
    p.amp = 2.0 * mass * r2 * r / denom;
    p.l[1] = (r * x + a * y) / r2pa2;
    p.l[2] = (r * y - a * x) / r2pa2;
    p.l[3] = z / r;
#endif
    return p;
}

// g(u, v) (KerrSchildInMetric::dot, :92-108).
KP_HD double ks_dot_at(const KSMetricPoint& w, const D4& u, const D4& v) {
    double eta_dot = 0.0 + (-u.v[0]) * v.v[0];
    eta_dot += u.v[1] * v.v[1];
    eta_dot += u.v[2] * v.v[2];
    eta_dot += u.v[3] * v.v[3];
    double lu = 0.0 + u.v[0];
    double lv = 0.0 + v.v[0];
    lu += w.l[1] * u.v[1];
    lv += w.l[1] * v.v[1];
    lu += w.l[2] * u.v[2];
    lv += w.l[2] * v.v[2];
    lu += w.l[3] * u.v[3];
    lv += w.l[3] * v.v[3];
    return eta_dot + w.amp * lu * lv;
}

KP_HD double ks_dot(double mass, double spin, const D4& X, const D4& u, const D4& v) {
    return ks_dot_at(ks_point(mass, spin, X), u, v);
}

// g_{mu nu} (gcov_matrix, :72-79).
KP_HD void ks_gcov_matrix(double mass, double spin, const D4& X, double g[4][4]) {
    const KSMetricPoint w = ks_point(mass, spin, X);
#pragma unroll
    for (int mu = 0; mu < 4; ++mu)
#pragma unroll
        for (int nu = 0; nu < 4; ++nu) {
            const double eta = mu != nu ? 0.0 : (mu == 0 ? -1.0 : 1.0);
            g[mu][nu] = eta + w.amp * w.l[mu] * w.l[nu];
        }
}

// g^{mu nu} (gcon, :65-70): eta - f lcon lcon with lcon_0 = -1.
KP_HD double ks_gcon_entry(const KSMetricPoint& w, int mu, int nu) {
    const double lmu = (mu == 0 ? -w.l[0] : w.l[mu]);
    const double lnu = (nu == 0 ? -w.l[0] : w.l[nu]);
    const double eta = mu != nu ? 0.0 : (mu == 0 ? -1.0 : 1.0);
    return eta - w.amp * lmu * lnu;
}

// Connection work: f, df, l, dl (build_ks_connection_work, :198-252).
// dl[mu][alpha] is stored for mu, alpha in 1..3 only (row/column 0 vanish).
struct KSConn {
    double amp;
    double damp[4];
    double l[4];
    double dl[4][4];
};

KP_HD KSConn ks_conn_plain(double mass, double spin, const D4& X) {
    const double x = X.v[1], y = X.v[2], z = X.v[3];
    const double a = spin;
    const double a2 = spin * spin;
    const double radius2 = x * x + y * y + z * z;
    const double sqsum = radius2 - a2;
    const double discr = sqrt(sqsum * sqsum + 4.0 * a2 * z * z);
    const double r2 = 0.5 * (sqsum + discr);
    const double r = sqrt(max_val(r2, kTiny));
    const double denom = r2 * r2 + a2 * z * z;
    const double amp = 2.0 * mass * r2 * r / denom;
    const double amp_r = -2.0 * mass * r2 * (r2 * r2 - 3.0 * a2 * z * z) / (denom * denom);
    const double r2pa2 = r2 + a2;
    KSConn c;
    c.amp = amp;
    c.l[0] = 1.0;
    c.l[1] = (r * x + a * y) / r2pa2;
    c.l[2] = (r * y - a * x) / r2pa2;
    c.l[3] = z / r;
    const double r2pa2_2 = r2pa2 * r2pa2;
    const double inv_2r = 0.5 / r;
    const double dr1 = (x + sqsum * x / discr) * inv_2r;
    const double dr2 = (y + sqsum * y / discr) * inv_2r;
    const double dr3 = (z + (sqsum * z + 2.0 * a2 * z) / discr) * inv_2r;
    c.damp[0] = 0.0;
    c.damp[1] = amp_r * dr1;
    c.damp[2] = amp_r * dr2;
    c.damp[3] = 6.0 * mass * r2 * dr3 / denom - amp / denom * (4.0 * r * r2 * dr3 + 2.0 * a2 * z);
    const double px = r * x + a * y;
    const double py = r * y - a * x;
    c.dl[1][1] = ((r + x * dr1) * r2pa2 - 2.0 * r * px * dr1) / r2pa2_2;
    c.dl[2][1] = ((-a + y * dr1) * r2pa2 - 2.0 * r * py * dr1) / r2pa2_2;
    c.dl[3][1] = -z / r2 * dr1;
    c.dl[1][2] = ((a + x * dr2) * r2pa2 - 2.0 * r * px * dr2) / r2pa2_2;
    c.dl[2][2] = ((r + y * dr2) * r2pa2 - 2.0 * r * py * dr2) / r2pa2_2;
    c.dl[3][2] = -z / r2 * dr2;
    c.dl[1][3] = (x * dr3 * r2pa2 - 2.0 * r * px * dr3) / r2pa2_2;
    c.dl[2][3] = (y * dr3 * r2pa2 - 2.0 * r * py * dr3) / r2pa2_2;
    c.dl[3][3] = (r - z * dr3) / r2;
    return c;
}

#ifdef __CUDACC__
// The same with the exact quotients and roots of kp_exact.cuh: every result
// has ks_conn_plain's bits.  A point for which an operand could leave their
// range (never one of a ray that is still traced in earnest) takes the plain
// form.  7 reciprocals and 19 quotients: 3225 -> 1341 cycles per
// right-hand side of a lone ray.
static __device__ __noinline__ void ks_conn_far_out(double mass, double spin, const D4& X, KSConn& c) {
    c = ks_conn_plain(mass, spin, X);
}

__device__ __forceinline__ KSConn ks_conn_exact(double mass, double spin, const D4& X) {
    const double x = X.v[1], y = X.v[2], z = X.v[3];
    const double a = spin;
    const double a2 = spin * spin;
    const double radius2 = x * x + y * y + z * z;
    const double sqsum = radius2 - a2;
    const double v = sqsum * sqsum + 4.0 * a2 * z * z;
    const double discr = exact_sqrt(v);
    const double r2 = 0.5 * (sqsum + discr);
    if (!(v > 1e-16 && r2 > 1e-16 && radius2 < 1e16 && exact_factor(x) && exact_factor(y) && exact_factor(z))) {
        KSConn plain;
        ks_conn_far_out(mass, spin, X, plain);
        return plain;
    }
    KSConn c;
    const double r = exact_sqrt(r2);
    const double denom = r2 * r2 + a2 * z * z;
    const double r2pa2 = r2 + a2;
    const double r2pa2_2 = r2pa2 * r2pa2;
    const ExactRecip i_discr = exact_recip(discr), i_r = exact_recip(r), i_r2 = exact_recip(r2);
    const ExactRecip i_denom = exact_recip(denom), i_denom2 = exact_recip(denom * denom);
    const ExactRecip i_rp = exact_recip(r2pa2), i_rp2 = exact_recip(r2pa2_2);
    const double amp = exact_quot(2.0 * mass * r2 * r, i_denom);
    const double amp_r = exact_quot(-2.0 * mass * r2 * (r2 * r2 - 3.0 * a2 * z * z), i_denom2);
    c.amp = amp;
    c.l[0] = 1.0;
    c.l[1] = exact_quot(r * x + a * y, i_rp);
    c.l[2] = exact_quot(r * y - a * x, i_rp);
    c.l[3] = exact_quot(z, i_r);
    const double inv_2r = exact_quot(0.5, i_r);
    const double dr1 = (x + exact_quot(sqsum * x, i_discr)) * inv_2r;
    const double dr2 = (y + exact_quot(sqsum * y, i_discr)) * inv_2r;
    const double dr3 = (z + exact_quot(sqsum * z + 2.0 * a2 * z, i_discr)) * inv_2r;
    c.damp[0] = 0.0;
    c.damp[1] = amp_r * dr1;
    c.damp[2] = amp_r * dr2;
    c.damp[3] = exact_quot(6.0 * mass * r2 * dr3, i_denom) -
                exact_quot(amp, i_denom) * (4.0 * r * r2 * dr3 + 2.0 * a2 * z);
    const double px = r * x + a * y;
    const double py = r * y - a * x;
    c.dl[1][1] = exact_quot((r + x * dr1) * r2pa2 - 2.0 * r * px * dr1, i_rp2);
    c.dl[2][1] = exact_quot((-a + y * dr1) * r2pa2 - 2.0 * r * py * dr1, i_rp2);
    const double mz = exact_quot(-z, i_r2);
    c.dl[3][1] = mz * dr1;
    c.dl[1][2] = exact_quot((a + x * dr2) * r2pa2 - 2.0 * r * px * dr2, i_rp2);
    c.dl[2][2] = exact_quot((r + y * dr2) * r2pa2 - 2.0 * r * py * dr2, i_rp2);
    c.dl[3][2] = mz * dr2;
    c.dl[1][3] = exact_quot(x * dr3 * r2pa2 - 2.0 * r * px * dr3, i_rp2);
    c.dl[2][3] = exact_quot(y * dr3 * r2pa2 - 2.0 * r * py * dr3, i_rp2);
    c.dl[3][3] = exact_quot(r - z * dr3, i_r2);
    return c;
}
#endif

KP_HD KSConn ks_conn(double mass, double spin, const D4& X) {
#ifdef __CUDA_ARCH__
    return ks_conn_exact(mass, spin, X);
#else
    return ks_conn_plain(mass, spin, X);
#endif
}

// Gamma^mu_{ab} p^a q^b without forming Gamma (ks_connection_contract, :302-327).
// l.p, l.q, dl_alpha.p, dl_alpha.q are evaluated once per call; every term
// keeps the reference's summation order.
KP_HD D4 ks_contract(const KSConn& c, const D4& p, const D4& q) {
    const double lp = ((0.0 + p.v[0]) + c.l[1] * p.v[1] + c.l[2] * p.v[2]) + c.l[3] * p.v[3];
    const double lq = ((0.0 + q.v[0]) + c.l[1] * q.v[1] + c.l[2] * q.v[2]) + c.l[3] * q.v[3];
    double dlp[4], dlq[4];
#pragma unroll
    for (int a = 1; a < 4; ++a) {
        dlp[a] = ((0.0 + c.dl[1][a] * p.v[1]) + c.dl[2][a] * p.v[2]) + c.dl[3][a] * p.v[3];
        dlq[a] = ((0.0 + c.dl[1][a] * q.v[1]) + c.dl[2][a] * q.v[2]) + c.dl[3][a] * q.v[3];
    }
    double t[4];
#pragma unroll
    for (int nu = 0; nu < 4; ++nu) {
        // dl[0][alpha] = 0: the row-0 contraction has no dl term.
        double term = 0.0;
#pragma unroll
        for (int a = 1; a < 4; ++a) {
            const double dlnu = nu == 0 ? 0.0 : c.dl[nu][a];
            const double row_q = c.damp[a] * c.l[nu] * lq + c.amp * (dlnu * lq + c.l[nu] * dlq[a]);
            const double row_p = c.damp[a] * c.l[nu] * lp + c.amp * (dlnu * lp + c.l[nu] * dlp[a]);
            term += p.v[a] * row_q + q.v[a] * row_p;
        }
        if (nu != 0) {
            term -= c.damp[nu] * lp * lq + c.amp * (dlp[nu] * lq + lp * dlq[nu]);
        } else {
            term -= 0.0;
        }
        t[nu] = term;
    }
    // lcon = (-1, l1, l2, l3)
    double lt = 0.0 + (-c.l[0]) * t[0];
    lt += c.l[1] * t[1];
    lt += c.l[2] * t[2];
    lt += c.l[3] * t[3];
    D4 out;
    out.v[0] = 0.5 * (-t[0] - c.amp * (-c.l[0]) * lt);
#pragma unroll
    for (int mu = 1; mu < 4; ++mu) out.v[mu] = 0.5 * (t[mu] - c.amp * c.l[mu] * lt);
    return out;
}

// dx = k, dk = -Gamma(k,k), de_i = -Gamma(k, e_i) (transport_rhs, :347-363).
KP_HD Ray ks_rhs(double mass, double spin, const Ray& s) {
    Ray d;
    d.x = s.k;
    const KSConn c = ks_conn(mass, spin, s.x);
    const D4 ck = ks_contract(c, s.k, s.k);
    const D4 ce1 = ks_contract(c, s.k, s.e1);
    const D4 ce2 = ks_contract(c, s.k, s.e2);
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        d.k.v[mu] = -ck.v[mu];
        d.e1.v[mu] = -ce1.v[mu];
        d.e2.v[mu] = -ce2.v[mu];
    }
    return d;
}

}  // namespace kp
