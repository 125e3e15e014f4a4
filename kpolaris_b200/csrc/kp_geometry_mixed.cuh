// kp_geometry_mixed.cuh -- the Kerr-Schild transport right-hand side of the
// mixed policy, in a factored form: a quad's lane contracts the connection
// with one vector (ks_factored_contract), a lane of a ray of its own with all
// three (ks_rhs_factored).
//
// Same algebra as ks_rhs in kp_geometry.cuh (the reference's specialised
// transport_rhs, src/geometry/kerr_schild_cartesian.hpp:194-363), regrouped:
//  * four reciprocals (1/r, 1/discr, 1/(r^2 + a^2), 1/denom) replace the
//    twenty divisions of the connection work;
//  * every transport contracts the connection with p = k, so the pieces of
//    Gamma(k, q) that depend on k alone (l.k, dl_{nu a} k^a, dl_{nu a} k^nu,
//    df.k) are formed once;
//  * the sum over a of Gamma's rows collapses to
//      t_nu = l_nu (lq Dk + lk Dq + f s(k, q)) + [nu > 0] (f (lq w_nu(k) + lk w_nu(q)) - df_nu lk lq),
//    with D = df.v and the symmetric and antisymmetric parts of dl,
//    s_{ab} = dl_{ab} + dl_{ba} and w_{ab} = dl_{ab} - dl_{ba};
// about 270 operations per evaluation instead of 1080: 110 for the point, 24
// for k and 45 for each transported vector.  The rounding differs
// from the reference's order, so this form serves the mixed policy only.
#pragma once

#include "kp_geometry.cuh"

namespace kp {

// sqrt(v) with its reciprocal, and 1/v.  FP64 on the device: the hardware's
// approximate reciprocal (square root) refined by one third-order step of
// Newton's iteration (e = 1 - v y^2, y' = y + y e (1/2 + 3 e / 8); e = 1 - v y,
// y' = y + y (e + e^2)), a few ulp, without the range checks and branches of
// the IEEE forms: sqsum and r of a ray are far from the ends of the range.
KP_HD void kp_sqrt_pair(double v, double& sq, double& inv) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double e = fma(-(v * y), y, 1.0);
    y = fma(y * e, fma(0.375, e, 0.5), y);
    const double g = v * y;
    sq = fma(fma(-g, g, v), 0.5 * y, g);
    inv = y;
#else
    sq = sqrt(v);
    inv = 1.0 / sq;
#endif
}
KP_HD double kp_recip(double v) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double e = fma(-v, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / v;
#endif
}

// ks_radius for the mixed policy: the refined square roots, with every
// operation spelled out so that the compiler's choice of fused operations
// cannot differ between two call sites (a ray resumed from its record takes
// the radius at one, an uninterrupted ray at another).
#ifdef __CUDACC__
__device__ __forceinline__ double kp_sqrt_refined(double v) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double e = __fma_rn(-__dmul_rn(v, y), y, 1.0);
    y = __fma_rn(__dmul_rn(y, e), __fma_rn(0.375, e, 0.5), y);
    const double g = __dmul_rn(v, y);
    return __fma_rn(__fma_rn(-g, g, v), __dmul_rn(0.5, y), g);
}

__device__ __forceinline__ double ks_radius_refined(double spin, const D4& X) {
    const double x = X.v[1], y = X.v[2], z = X.v[3];
    const double a2 = __dmul_rn(spin, spin);
    const double sqsum = __dsub_rn(__fma_rn(x, x, __fma_rn(y, y, __dmul_rn(z, z))), a2);
    const double az = __dmul_rn(2.0, __dmul_rn(spin, z));
    const double discr = kp_sqrt_refined(max_val(__fma_rn(sqsum, sqsum, __dmul_rn(az, az)), 1e-290));
    return kp_sqrt_refined(max_val(__dmul_rn(0.5, __dadd_rn(sqsum, discr)), 1e-290));
}
#else
KP_HD double ks_radius_refined(double spin, const D4& X) { return ks_radius(spin, X); }
#endif

// What a point's connection needs: f, df, l and dl_{nu a} = d l_nu / d x^a,
// the last as its symmetric part s_{ab} = dl_{ab} + dl_{ba} and its
// antisymmetric part w_{ab} = dl_{ab} - dl_{ba}.
struct KsFactored {
    double f, d[3], l[3];
    double s11, s22, s33, s12, s13, s23;
    double w12, w13, w23;
};

KP_HD KsFactored ks_factored_conn(double M, double a, double x, double y, double z) {
    const double a2 = a * a;
    const double sqsum = x * x + y * y + z * z - a2;
    double discr, inv_discr;
    kp_sqrt_pair(sqsum * sqsum + 4.0 * a2 * z * z, discr, inv_discr);
    const double r2 = 0.5 * (sqsum + discr);
    double r, inv_r;
    kp_sqrt_pair(r2 > 1e-30 ? r2 : 1e-30, r, inv_r);
    const double inv_denom = kp_recip(r2 * r2 + a2 * z * z);
    const double inv_rp = kp_recip(r2 + a2);
    KsFactored c;
    c.f = 2.0 * M * r2 * r * inv_denom;
    const double amp_r = -2.0 * M * r2 * (r2 * r2 - 3.0 * a2 * z * z) * (inv_denom * inv_denom);
    const double l1 = (r * x + a * y) * inv_rp;
    const double l2 = (r * y - a * x) * inv_rp;
    const double l3 = z * inv_r;
    const double inv_2r = 0.5 * inv_r;
    const double g12 = (1.0 + sqsum * inv_discr) * inv_2r;
    const double dr1 = x * g12, dr2 = y * g12;
    const double dr3 = z * (1.0 + (sqsum + 2.0 * a2) * inv_discr) * inv_2r;
    c.d[0] = amp_r * dr1;
    c.d[1] = amp_r * dr2;
    c.d[2] = (6.0 * M * r2 * dr3 - c.f * (4.0 * r * r2 * dr3 + 2.0 * a2 * z)) * inv_denom;
    const double tr = 2.0 * r;
    const double u1 = x - tr * l1, u2 = y - tr * l2, u3 = -l3 * inv_r;
    const double dl11 = (r + u1 * dr1) * inv_rp;
    const double dl21 = (-a + u2 * dr1) * inv_rp;
    const double dl31 = u3 * dr1;
    const double dl12 = (a + u1 * dr2) * inv_rp;
    const double dl22 = (r + u2 * dr2) * inv_rp;
    const double dl32 = u3 * dr2;
    const double dl13 = u1 * dr3 * inv_rp;
    const double dl23 = u2 * dr3 * inv_rp;
    const double dl33 = (r - z * dr3) * (inv_r * inv_r);
    c.l[0] = l1;
    c.l[1] = l2;
    c.l[2] = l3;
    c.s11 = dl11 + dl11;
    c.s22 = dl22 + dl22;
    c.s33 = dl33 + dl33;
    c.s12 = dl12 + dl21;
    c.s13 = dl13 + dl31;
    c.s23 = dl23 + dl32;
    c.w12 = dl12 - dl21;
    c.w13 = dl13 - dl31;
    c.w23 = dl23 - dl32;
    return c;
}

// The pieces of Gamma(k, .) that depend on k alone.
struct KsFactoredK {
    double lk, dk;        // l.k, df.k
    double wk[3], sk[3];  // w_{ia} k^a, s_{ia} k^a
};

KP_HD KsFactoredK ks_factored_k(const KsFactored& c, const double (&k)[4]) {
    KsFactoredK o;
    o.lk = k[0] + c.l[0] * k[1] + c.l[1] * k[2] + c.l[2] * k[3];
    o.dk = c.d[0] * k[1] + c.d[1] * k[2] + c.d[2] * k[3];
    o.wk[0] = c.w12 * k[2] + c.w13 * k[3];
    o.wk[1] = c.w23 * k[3] - c.w12 * k[1];
    o.wk[2] = -(c.w13 * k[1] + c.w23 * k[2]);
    o.sk[0] = c.s11 * k[1] + c.s12 * k[2] + c.s13 * k[3];
    o.sk[1] = c.s12 * k[1] + c.s22 * k[2] + c.s23 * k[3];
    o.sk[2] = c.s13 * k[1] + c.s23 * k[2] + c.s33 * k[3];
    return o;
}

// out = -Gamma(k, q).
KP_HD void ks_factored_contract(const KsFactored& c, const KsFactoredK& p, const double (&q)[4], double (&out)[4]) {
    const double lq = q[0] + c.l[0] * q[1] + c.l[1] * q[2] + c.l[2] * q[3];
    const double dq = c.d[0] * q[1] + c.d[1] * q[2] + c.d[2] * q[3];
    const double sq = p.sk[0] * q[1] + p.sk[1] * q[2] + p.sk[2] * q[3];
    const double wq0 = c.w12 * q[2] + c.w13 * q[3];
    const double wq1 = c.w23 * q[3] - c.w12 * q[1];
    const double wq2 = -(c.w13 * q[1] + c.w23 * q[2]);
    const double t0 = lq * p.dk + p.lk * dq + c.f * sq;
    const double lklq = p.lk * lq, fq = c.f * lq, fk = c.f * p.lk;
    const double t1 = c.l[0] * t0 + fq * p.wk[0] + fk * wq0 - c.d[0] * lklq;
    const double t2 = c.l[1] * t0 + fq * p.wk[1] + fk * wq1 - c.d[1] * lklq;
    const double t3 = c.l[2] * t0 + fq * p.wk[2] + fk * wq2 - c.d[2] * lklq;
    const double al = c.f * (c.l[0] * t1 + c.l[1] * t2 + c.l[2] * t3 - t0);
    out[0] = 0.5 * (t0 - al);
    out[1] = 0.5 * (c.l[0] * al - t1);
    out[2] = 0.5 * (c.l[1] * al - t2);
    out[3] = 0.5 * (c.l[2] * al - t3);
}

// The transport right-hand side of a ray.
KP_HD Ray ks_rhs_factored(double mass, double spin, const Ray& s) {
    const KsFactored c = ks_factored_conn(mass, spin, s.x.v[1], s.x.v[2], s.x.v[3]);
    const KsFactoredK p = ks_factored_k(c, s.k.v);
    Ray d;
    d.x = s.k;
    ks_factored_contract(c, p, s.k.v, d.k.v);
    ks_factored_contract(c, p, s.e1.v, d.e1.v);
    ks_factored_contract(c, p, s.e2.v, d.e2.v);
    return d;
}

}  // namespace kp
