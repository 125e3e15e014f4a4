// kp_trace_fp64.cuh -- one ray, FP64: backward pass A from the camera to the
// radiating-sphere endpoint, then forward pass B with NF Stokes channels
// sharing the geodesic, then the observer-basis transform.
//
// Restates the fused per-pixel kernels trace_pass_b_segment_model_pixel_metric
// (src/geodesic/pass_b.hpp:769-1114) and its multi-frequency twin
// (pass_b.hpp:1131-1501) for the Kerr metric in Cartesian KS: the metric has
// no time domain, no excision hook and no effective-min-step hook, so those
// calls reduce to identities (src/geodesic/metric_domain.hpp:78-225).  The
// surface-crossing refinement restates locate_metric_surface_crossing
// (src/geodesic/pass_a_core.hpp:94-197).
#pragma once

#include "kp_camera.cuh"
#include "kp_integrate.cuh"
#include "kp_radiation.cuh"

namespace kp {

__device__ __forceinline__ int finite_ray(const Ray& s) {
#pragma unroll
    for (int mu = 0; mu < 4; ++mu) {
        const double v[4] = {s.x.v[mu], s.k.v[mu], s.e1.v[mu], s.e2.v[mu]};
#pragma unroll
        for (int f = 0; f < 4; ++f)
            if (!(v[f] == v[f]) || abs_val(v[f]) >= kLarge) return 0;
    }
    return 1;
}

// metric_surface_path_state (pass_a_core.hpp:76-87)
__device__ __forceinline__ Ray surface_path_state(double mass, double spin, const Ray& first,
                                                  double h, int composed) {
    if (composed) {
        const Ray half = rk4_step(mass, spin, first, h * 0.5);
        return rk4_step(mass, spin, half, h * 0.5);
    }
    return rk4_step(mass, spin, first, h);
}

// locate_metric_surface_crossing (pass_a_core.hpp:94-197) for the spherical
// surfaces r = surface_parameter; returns the last point on the original side.
static __device__ __noinline__ void locate_crossing(double mass, double spin, const Ray& first,
                                             const Ray& second, double full_h,
                                             double surface_parameter, int composed,
                                             Ray& out_state, double& out_h) {
    out_state = first;
    out_h = 0.0;
    double lo = 0.0, hi = 1.0;
    double flo = ks_radius(spin, first.x) - surface_parameter;
    if (flo == 0.0) return;
    if (!finite_ray(second)) return;
    const Ray hs = surface_path_state(mass, spin, first, full_h, composed);
    if (!finite_ray(hs)) return;
    double fhi = ks_radius(spin, hs.x) - surface_parameter;
    if (!(fhi == fhi) || abs_val(fhi) >= kLarge) return;
    if (fhi == 0.0) {
        out_state = hs;
        out_h = full_h;
        return;
    }
    if ((flo > 0.0) == (fhi > 0.0)) return;
    int use_secant = 1;
#pragma unroll 1
    for (int iter = 0; iter < 12; ++iter) {
        const double width = hi - lo;
        double trial = (lo + hi) * 0.5;
        const double denom = flo - fhi;
        if (use_secant && abs_val(denom) > kTiny) {
            const double secant = lo + width * flo / denom;
            const double guard = width * 0.1;
            if (secant > lo + guard && secant < hi - guard) trial = secant;
        }
        const Ray ts = surface_path_state(mass, spin, first, full_h * trial, composed);
        if (!finite_ray(ts)) {
            hi = trial;
            use_secant = 0;
            continue;
        }
        const double ft = ks_radius(spin, ts.x) - surface_parameter;
        if (!(ft == ft) || abs_val(ft) >= kLarge) {
            hi = trial;
            use_secant = 0;
            continue;
        }
        if (ft == 0.0) {
            out_state = ts;
            out_h = full_h * trial;
            return;
        }
        if ((flo > 0.0) == (ft > 0.0)) {
            lo = trial;
            flo = ft;
            out_state = ts;
            out_h = full_h * trial;
        } else {
            hi = trial;
            fhi = ft;
        }
    }
}

__device__ __forceinline__ double max_frame_error(double mass, double spin, const Ray& s) {
    const KSMetricPoint w = ks_point(mass, spin, s.x);
    double o = abs_val(ks_dot_at(w, s.k, s.k));
    o = max_val(o, abs_val(ks_dot_at(w, s.e1, s.k)));
    o = max_val(o, abs_val(ks_dot_at(w, s.e2, s.k)));
    o = max_val(o, abs_val(ks_dot_at(w, s.e1, s.e1) - 1.0));
    o = max_val(o, abs_val(ks_dot_at(w, s.e2, s.e2) - 1.0));
    o = max_val(o, abs_val(ks_dot_at(w, s.e1, s.e2)));
    return o;
}

__device__ __forceinline__ double spatial_distance(const D4& a, const D4& b) {
    return sqrt(sq(a.v[1] - b.v[1]) + sq(a.v[2] - b.v[2]) + sq(a.v[3] - b.v[3]));
}

__device__ __forceinline__ double vmaxabsdiff(const D4& a, const D4& b) {
    double o = abs_val(a.v[0] - b.v[0]);
    for (int i = 1; i < 4; ++i) o = max_val(o, abs_val(a.v[i] - b.v[i]));
    return o;
}

// radiation_substep_count (pass_b.hpp:147-179) with requested_substeps = 1.
// nsub is a power of two, so q / nsub > lim is exactly q > lim * nsub (both
// sides are exact scalings): the doubling loops compare against lim * nsub
// instead of dividing, with the reference's outcomes.
template<class C>
__device__ __forceinline__ int radiation_substep_count(const C& co, double h, double dls,
                                                       double max_rad_step, double max_rad_depth,
                                                       double max_abs_depth, double max_far_depth) {
    int nsub = 1;
    const double abs_h = abs_val(h);
    if (max_rad_step > 0.0)
        while (abs_h > max_rad_step * double(nsub) && nsub < 4096) nsub *= 2;
    const double dl = abs_h * abs_val(dls);
    const double alim = max_abs_depth >= 0.0 ? max_abs_depth : max_rad_depth;
    if (alim > 0.0) {
        const double aQ = co.aQ, aU = co.aU, aV = co.aV;
        const double depth = (abs_val(double(co.aI)) + sqrt(aQ * aQ + aU * aU + aV * aV)) * dl;
        while (depth > alim * double(nsub) && nsub < 4096) nsub *= 2;
    }
    const double flim = max_far_depth >= 0.0 ? max_far_depth : max_rad_depth;
    if (flim > 0.0) {
        const double rQ = co.rQ, rU = co.rU, rV = co.rV;
        const double depth = sqrt(rQ * rQ + rU * rU + rV * rV) * dl;
        while (depth > flim * double(nsub) && nsub < 4096) nsub *= 2;
    }
    return nsub;
}

#ifdef __CUDACC__
// The same count in closed form: the depths of a unit dl, then for each limit
// the smallest power of two n (at most 4096) with depth <= lim n.  For two
// positive normal numbers n is the ratio of their binades, doubled if the
// depth's significand is the larger; anything else takes the loop.
struct RadDepths {
    double a, r, dls;  // absorption and Faraday depth per dl; |dls|
};

__device__ __forceinline__ RadDepths radiation_depths(const Coeffs<double>& co, double dls) {
    return RadDepths{abs_val(co.aI) + sqrt(co.aQ * co.aQ + co.aU * co.aU + co.aV * co.aV),
                     sqrt(co.rQ * co.rQ + co.rU * co.rU + co.rV * co.rV), abs_val(dls)};
}

__device__ __forceinline__ int pow2_steps(double depth, double lim) {
    if (!(depth > lim)) return 1;
    const unsigned long long d = (unsigned long long)__double_as_longlong(depth);
    const unsigned long long l = (unsigned long long)__double_as_longlong(lim);
    const int ed = int(d >> 52), el = int(l >> 52);
    if (el == 0) {
        int n = 1;
        while (depth > lim * double(n) && n < 4096) n *= 2;
        return n;
    }
    const unsigned long long frac = (1ull << 52) - 1;
    const int e = ed - el + ((d & frac) > (l & frac) ? 1 : 0);
    return 1 << (e > 12 ? 12 : e);
}

__device__ __forceinline__ int substeps_for(const RadDepths& p, double h, double max_rad_step, const ImageConsts& c) {
    const double abs_h = abs_val(h);
    int n = max_rad_step > 0.0 ? pow2_steps(abs_h, max_rad_step) : 1;
    const double dl = abs_h * p.dls;
    const double alim = c.max_absorption_depth >= 0.0 ? c.max_absorption_depth : c.max_radiation_depth;
    if (alim > 0.0) n = max(n, pow2_steps(p.a * dl, alim));
    const double flim = c.max_faraday_depth >= 0.0 ? c.max_faraday_depth : c.max_radiation_depth;
    if (flim > 0.0) n = max(n, pow2_steps(p.r * dl, flim));
    return n;
}

// h / n for a power of two n <= 4096, as the exact product with 1 / n.
__device__ __forceinline__ double over_pow2(double h, int n) {
    return h * __longlong_as_double((long long)(1023 - (31 - __clz(n))) << 52);
}
#endif

struct PixelOut {
    double r11, r12, r21, r22;
    double closure_x, closure_k, final_null, frame_error;
    int pass_a_steps, steps, reason;
};

// Pass A (pass_b.hpp:786-938).  Returns 1 when the endpoint is valid for
// pass B (entered the radiating sphere and ended on its inner or outer surface).
__device__ __forceinline__ int trace_pass_a(const ImageConsts& c, Ray& state, int& pa_steps,
                                            int& pa_reason) {
    const double mass = c.mass, spin = c.spin;
    pa_reason = kMaxSteps;
    pa_steps = 0;
    StepControl ctl;
    ctl.tolerance = c.tolerance;
    ctl.min_step = c.min_step_abs;
    ctl.max_step = c.max_step;
    double h_current = -abs_val(c.step);
    int entered = 0;
    int inside = 0;
#pragma unroll 1
    for (int n = 0; n < c.max_steps; ++n) {
        const double r_bl = ks_radius(spin, state.x);
        if (!entered) {
            if (r_bl <= c.outer_radius) {
                entered = 1;
                inside = 0;
            }
        } else {
            if (r_bl - c.inner_radius <= 0.0) {
                pa_reason = kReachedInner;
                break;
            }
            if (inside > 0 && r_bl >= c.outer_radius) {
                pa_reason = kEscaped;
                break;
            }
        }
        const double old_r = r_bl;
        const double old_inner = r_bl - c.inner_radius;
        double used_h = h_current;
        Ray next;
        if (c.adaptive) {
            StepControl tc = ctl;
            if (abs_val(used_h) < tc.min_step) tc.min_step = abs_val(used_h);
            AdaptiveStep st;
            adaptive_step(c.integrator, mass, spin, state, used_h, tc, st);
            if (!st.accepted) {
                h_current = st.next_h;
                if (abs_val(h_current) <= c.min_step_abs * 1.0001) {
                    pa_reason = kAdaptiveUnderflow;
                    break;
                }
                continue;
            }
            next = st.state;
            used_h = st.used_h;
            h_current = st.next_h;
        } else {
            next = rk4_step(mass, spin, state, used_h);
        }
        const double next_r = ks_radius(spin, next.x);
        const double next_inner = next_r - c.inner_radius;
        if (!entered && next_r <= c.outer_radius) {
            entered = 1;
            inside = 0;
        } else if (!entered && next_r >= old_r) {
            state = next;
            pa_steps += 1;
            pa_reason = kEscaped;
            break;
        }
        int crossing = kNone;
        if (entered && old_inner > 0.0 && next_inner <= 0.0) {
            crossing = kReachedInner;
        } else if (entered && inside > 0 && old_r < c.outer_radius && next_r >= c.outer_radius) {
            crossing = kEscaped;
        }
        if (crossing != kNone) {
            const double sp = crossing == kReachedInner ? c.inner_radius : c.outer_radius;
            Ray ev;
            double ev_h;
            locate_crossing(mass, spin, state, next, used_h, sp, c.adaptive, ev, ev_h);
            state = ev;
            pa_steps += 1;
            pa_reason = crossing;
            break;
        }
        state = next;
        pa_steps += 1;
        if (entered) inside += 1;
    }
    return entered && (pa_reason == kReachedInner || pa_reason == kEscaped);
}

// Screen overlap, observer transform and closure diagnostics
// (pass_b.hpp:87-98, :1096-1113; stokes_rotation.hpp:39-57).
template<class R, int NF>
__device__ __forceinline__ void finish_ray(const ImageConsts& c, const Ray& cam, const Ray& state,
                                           int passed_b, Stokes4<R> (&stokes)[NF], PixelOut& o,
                                           double (&obs)[NF][4]) {
    const KSMetricPoint w = ks_point(c.mass, c.spin, state.x);
    if (passed_b) {
        o.r11 = ks_dot_at(w, cam.e1, state.e1);
        o.r12 = ks_dot_at(w, cam.e1, state.e2);
        o.r21 = ks_dot_at(w, cam.e2, state.e1);
        o.r22 = ks_dot_at(w, cam.e2, state.e2);
    } else {
        o.r11 = 1.0;
        o.r12 = 0.0;
        o.r21 = 0.0;
        o.r22 = 1.0;
    }
    const double r11 = o.r11, r12 = o.r12, r21 = o.r21, r22 = o.r22;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        if (passed_b) {
            const double I = stokes[f].I, Q = stokes[f].Q, U = stokes[f].U, V = stokes[f].V;
            obs[f][0] = I;
            obs[f][1] = 0.5 * Q * (r11 * r11 - r12 * r12 - r21 * r21 + r22 * r22) + U * (r11 * r12 - r21 * r22);
            obs[f][2] = Q * (r11 * r21 - r12 * r22) + U * (r11 * r22 + r12 * r21);
            obs[f][3] = (r11 * r22 - r12 * r21) * V;
        } else {
            obs[f][0] = obs[f][1] = obs[f][2] = obs[f][3] = 0.0;
        }
    }
    o.closure_x = spatial_distance(state.x, cam.x);
    o.closure_k = vmaxabsdiff(state.k, cam.k);
    o.final_null = ks_dot_at(w, state.k, state.k);
    o.frame_error = max_frame_error(c.mass, c.spin, state);
}

__device__ __forceinline__ void store_diagnostics(const ImageOutPtrs& out, int pixel, const PixelOut& o) {
    out.closure_x[pixel] = o.closure_x;
    out.closure_k[pixel] = o.closure_k;
    out.final_null[pixel] = o.final_null;
    out.frame_error[pixel] = o.frame_error;
    out.det_r[pixel] = o.r11 * o.r22 - o.r12 * o.r21;
    out.r11[pixel] = o.r11;
    out.r12[pixel] = o.r12;
    out.r21[pixel] = o.r21;
    out.r22[pixel] = o.r22;
    out.basis_identity_error[pixel] = max_val(max_val(abs_val(o.r11 - 1.0), abs_val(o.r22 - 1.0)),
                                              max_val(abs_val(o.r12), abs_val(o.r21)));
    out.basis_rotation_angle[pixel] = atan2(o.r21 - o.r12, o.r11 + o.r22);
    out.pass_a_steps[pixel] = o.pass_a_steps;
    out.steps[pixel] = o.steps;
    out.reason[pixel] = o.reason;
}

template<int NF>
__device__ __forceinline__ void store_stokes(const ImageOutPtrs& out, int pixel, int npix,
                                             const double (&obs)[NF][4]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        const size_t idx = size_t(f) * size_t(npix) + size_t(pixel);
        out.image_i[idx] = obs[f][0];
        out.image_q[idx] = obs[f][1];
        out.image_u[idx] = obs[f][2];
        out.image_v[idx] = obs[f][3];
    }
}

}  // namespace kp
