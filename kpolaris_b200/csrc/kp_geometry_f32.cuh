// kp_geometry_f32.cuh -- the Kerr-Schild transport right-hand side of the
// mixed-precision policy, in a factored form templated on the arithmetic
// type; the kernels use it in FP64.  The core
// (ks_transport_factored) works on T values; ks_rhs_factored wraps it for
// FP64 Rays.
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
// FP32 (where the contraction's own cancellation already
// limits it to ~3e-5): one hardware reciprocal square root or reciprocal.
template<class T>
KP_HD void kp_sqrt_pair(T v, T& sq, T& inv) {
    sq = sqrt(v);
    inv = T(1) / sq;
}
template<>
KP_HD void kp_sqrt_pair<double>(double v, double& sq, double& inv) {
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
template<>
KP_HD void kp_sqrt_pair<float>(float v, float& sq, float& inv) {
#ifdef __CUDA_ARCH__
    inv = rsqrtf(v);
    sq = v * inv;
#else
    sq = sqrtf(v);
    inv = 1.0f / sq;
#endif
}
template<class T>
KP_HD T kp_recip(T v) {
    return T(1) / v;
}
template<>
KP_HD double kp_recip<double>(double v) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double e = fma(-v, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / v;
#endif
}
template<>
KP_HD float kp_recip<float>(float v) {
#ifdef __CUDA_ARCH__
    return __fdividef(1.0f, v);
#else
    return 1.0f / v;
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
template<class T>
struct KsFactored {
    T f, d[3], l[3];
    T s11, s22, s33, s12, s13, s23;
    T w12, w13, w23;
};

template<class T>
KP_HD KsFactored<T> ks_factored_conn(T M, T a, T x, T y, T z) {
    const T a2 = a * a;
    const T sqsum = x * x + y * y + z * z - a2;
    T discr, inv_discr;
    kp_sqrt_pair<T>(sqsum * sqsum + T(4) * a2 * z * z, discr, inv_discr);
    const T r2 = T(0.5) * (sqsum + discr);
    T r, inv_r;
    kp_sqrt_pair<T>(r2 > T(1e-30) ? r2 : T(1e-30), r, inv_r);
    const T inv_denom = kp_recip<T>(r2 * r2 + a2 * z * z);
    const T inv_rp = kp_recip<T>(r2 + a2);
    KsFactored<T> c;
    c.f = T(2) * M * r2 * r * inv_denom;
    const T amp_r = T(-2) * M * r2 * (r2 * r2 - T(3) * a2 * z * z) * (inv_denom * inv_denom);
    const T l1 = (r * x + a * y) * inv_rp;
    const T l2 = (r * y - a * x) * inv_rp;
    const T l3 = z * inv_r;
    const T inv_2r = T(0.5) * inv_r;
    const T g12 = (T(1) + sqsum * inv_discr) * inv_2r;
    const T dr1 = x * g12, dr2 = y * g12;
    const T dr3 = z * (T(1) + (sqsum + T(2) * a2) * inv_discr) * inv_2r;
    c.d[0] = amp_r * dr1;
    c.d[1] = amp_r * dr2;
    c.d[2] = (T(6) * M * r2 * dr3 - c.f * (T(4) * r * r2 * dr3 + T(2) * a2 * z)) * inv_denom;
    const T tr = T(2) * r;
    const T u1 = x - tr * l1, u2 = y - tr * l2, u3 = -l3 * inv_r;
    const T dl11 = (r + u1 * dr1) * inv_rp;
    const T dl21 = (-a + u2 * dr1) * inv_rp;
    const T dl31 = u3 * dr1;
    const T dl12 = (a + u1 * dr2) * inv_rp;
    const T dl22 = (r + u2 * dr2) * inv_rp;
    const T dl32 = u3 * dr2;
    const T dl13 = u1 * dr3 * inv_rp;
    const T dl23 = u2 * dr3 * inv_rp;
    const T dl33 = (r - z * dr3) * (inv_r * inv_r);
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
template<class T>
struct KsFactoredK {
    T lk, dk;        // l.k, df.k
    T wk[3], sk[3];  // w_{ia} k^a, s_{ia} k^a
};

template<class T>
KP_HD KsFactoredK<T> ks_factored_k(const KsFactored<T>& c, const T (&k)[4]) {
    KsFactoredK<T> o;
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
template<class T>
KP_HD void ks_factored_contract(const KsFactored<T>& c, const KsFactoredK<T>& p, const T (&q)[4], T (&out)[4]) {
    const T lq = q[0] + c.l[0] * q[1] + c.l[1] * q[2] + c.l[2] * q[3];
    const T dq = c.d[0] * q[1] + c.d[1] * q[2] + c.d[2] * q[3];
    const T sq = p.sk[0] * q[1] + p.sk[1] * q[2] + p.sk[2] * q[3];
    const T wq0 = c.w12 * q[2] + c.w13 * q[3];
    const T wq1 = c.w23 * q[3] - c.w12 * q[1];
    const T wq2 = -(c.w13 * q[1] + c.w23 * q[2]);
    const T t0 = lq * p.dk + p.lk * dq + c.f * sq;
    const T lklq = p.lk * lq, fq = c.f * lq, fk = c.f * p.lk;
    const T t1 = c.l[0] * t0 + fq * p.wk[0] + fk * wq0 - c.d[0] * lklq;
    const T t2 = c.l[1] * t0 + fq * p.wk[1] + fk * wq1 - c.d[1] * lklq;
    const T t3 = c.l[2] * t0 + fq * p.wk[2] + fk * wq2 - c.d[2] * lklq;
    const T al = c.f * (c.l[0] * t1 + c.l[1] * t2 + c.l[2] * t3 - t0);
    out[0] = T(0.5) * (t0 - al);
    out[1] = T(0.5) * (c.l[0] * al - t1);
    out[2] = T(0.5) * (c.l[1] * al - t2);
    out[3] = T(0.5) * (c.l[2] * al - t3);
}

// The transports of q[0] = k, q[1] = e1, q[2] = e2 at spatial position
// (x, y, z): out[w] = dq[w]/dlambda = -Gamma(k, q[w]).
template<class T>
KP_HD void ks_transport_factored(T M, T a, T x, T y, T z, const T (&q)[3][4], T (&out)[3][4]) {
    const KsFactored<T> c = ks_factored_conn<T>(M, a, x, y, z);
    const KsFactoredK<T> p = ks_factored_k<T>(c, q[0]);
#pragma unroll
    for (int which = 0; which < 3; ++which) ks_factored_contract<T>(c, p, q[which], out[which]);
}

template<class T>
KP_HD Ray ks_rhs_factored(double mass_d, double spin_d, const Ray& s) {
    T q[3][4], o[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        q[0][i] = T(s.k.v[i]);
        q[1][i] = T(s.e1.v[i]);
        q[2][i] = T(s.e2.v[i]);
    }
    ks_transport_factored<T>(T(mass_d), T(spin_d), T(s.x.v[1]), T(s.x.v[2]), T(s.x.v[3]), q, o);
    Ray d;
    d.x = s.k;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        d.k.v[i] = double(o[0][i]);
        d.e1.v[i] = double(o[1][i]);
        d.e2.v[i] = double(o[2][i]);
    }
    return d;
}

}  // namespace kp
