// kp_engine.cuh -- the ray engine's policies, control modes and one-lane RK
// jobs.  A quad (kp_quad.cuh) or a lane (kp_persistent.cuh) holds one ray and
// advances it through a resumable state machine whose loop iteration is one RK
// job (a step-doubling attempt, an RK4 step, a composed pair of RK4
// half steps or a Cash-Karp attempt) started from the lane's current state.
// Jobs run as a stage loop around ONE right-hand-side site, so lanes of a warp
// evaluate the RHS together whatever their phase (pass A, surface refinement,
// pass B, camera crossing).  Finished rays are replaced from a global ray queue
// shared by every image of the launch (warp-aggregated atomics), which removes
// both the tail of uneven rays and the launch-per-image cost.
//
// The control machine restates, as explicit states, the loops of
// trace_pass_b_segment_model_pixel_metric / _multifrequency_pixel_metric
// (src/geodesic/pass_b.hpp:769-1114, :1131-1501), adaptive_rk4_step
// (src/geodesic/rk4.hpp:108-161) and locate_metric_surface_crossing
// (src/geodesic/pass_a_core.hpp:94-197).  With the FP64 policy every
// arithmetic operation is the reference's, in its order: results are
// bit-identical to the per-pixel FP64 kernel.
#pragma once

#include "kp_camera.cuh"
#include "kp_integrate.cuh"
#include "kp_radiation.cuh"
#include "kp_trace_fp64.cuh"
#include "kp_geometry_mixed.cuh"
#include "kp_radiation_mixed.cuh"
#include "kp_scene.cuh"

namespace kp {

// Kinds of RK job.
enum RkKind : int { kRkSD = 0, kRkRK4 = 1, kRkRK4x2 = 2, kRkCK = 3 };

// Control modes: what the pending RK job's result is for.
enum Mode : int {
    kIdle = 0,
    kAStep = 1,        // pass-A step attempt (adaptive sequence or fixed RK4)
    kACrossHi = 2,     // crossing search: full-step endpoint with the trial evaluator
    kACrossTrial = 3,  // crossing search: trial at fraction `trial`
    kBStep = 4,        // pass-B step attempt
    kBCamCross = 5,    // pass-B partial step to the camera surface
    kDone = 6,
};

// ---------------------------------------------------------------- RHS policy
// FP64 policy: the reference's arithmetic.
struct PolicyFP64 {
    static constexpr bool kMixed = false;
};
// Mixed policy: FP64 state, connection (in factored, fused form), step control
// and radiation (factored, fused forms that round differently); many far-field
// steps taken at once (kp_quad.cuh).
struct PolicyMixed {
    static constexpr bool kMixed = true;
};

// Radiation side of a policy and scene: FP64 (the reference's arithmetic) or
// the factored form with the per-frequency 2^E emission scale
// (kp_radiation_mixed.cuh).
template<class P, class S = SceneRiaf>
struct RadTraits;

template<>
struct RadTraits<PolicyFP64, SceneRiaf> {
    using Stokes = Stokes4<double>;
    using Co = Coeffs<double>;
    using Sample = RiafSample;
    __device__ static void zero(Stokes& s) { s = Stokes4<double>{0.0, 0.0, 0.0, 0.0}; }
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return riaf_sample(c, r); }
    __device__ static Sample none() {
        Sample s;
        s.emitting = 0;
        return s;
    }
    __device__ static Co coeffs(const ImageConsts& c, const Sample& p, int f) {
        return riaf_coefficients(c, p, c.freq[f]);
    }
    __device__ static RadDepths depths(const Co& co, double dls) { return radiation_depths(co, dls); }
    __device__ static Co coeffs_ctl(const ImageConsts& c, const Sample& p, int g) {
        return riaf_coefficients(c, p, c.ctl_freq[g]);
    }
    // step() with coefficients of zero
    __device__ static void add_zero(Stokes& s) {
        s = Stokes{s.I + 0.0, s.Q + 0.0, s.U + 0.0, s.V + 0.0};
    }
    __device__ static void step(Stokes& s, const Co& co, double h, const ImageConsts& c, int f) {
        stokes_apply(s, stokes_op(co, abs_val(h) * c.dlambda_scale[f]), co.jI, co.jQ, co.jU, co.jV);
    }
    __device__ static Stokes4<double> result(const Stokes& s, const ImageConsts&, int) { return s; }
};

__device__ __forceinline__ double norm_refined(double x, double y, double z) {
    const double n2 = x * x + y * y + z * z;
    if (!(n2 > 1e-280 && n2 < 1e280)) return sqrt(n2);
    double n, inv;
    kp_sqrt_pair(n2, n, inv);
    return n;
}

template<>
struct RadTraits<PolicyMixed, SceneRiaf> {
    using Stokes = StokesM;
    using Co = CoeffsM;
    using Sample = RiafSampleM;
    __device__ static void zero(Stokes& s) { s = StokesM{0.0, 0.0, 0.0, 0.0}; }
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return riaf_sample_m(c, r); }
    __device__ static Sample none() {
        Sample s;
        s.emitting = 0;
        return s;
    }
    __device__ static Co coeffs(const ImageConsts& c, const Sample& p, int f) {
        return riaf_coefficients_m(c, p, c.freq[f] * 1e-9, c.emission_scale_pow2[f]);
    }
    __device__ static Co coeffs_ctl(const ImageConsts& c, const Sample& p, int g) {
        return riaf_coefficients_m(c, p, c.ctl_freq[g] * 1e-9, c.ctl_emission_scale_pow2[g]);
    }
    __device__ static RadDepths depths(const Co& co, double dls) {
        return RadDepths{abs_val(co.aI) + norm_refined(co.aQ, co.aU, co.aV), norm_refined(co.rQ, co.rU, co.rV),
                         abs_val(dls)};
    }
    __device__ static void step(Stokes& s, const Co& co, double h, const ImageConsts& c, int f) {
        stokes_step_m(s, co, abs_val(h) * c.dlambda_scale[f]);
    }
    __device__ static Stokes4<double> result(const Stokes& s, const ImageConsts& c, int f) {
        const double inv = c.inv_emission_scale_pow2[f];
        return Stokes4<double>{s.I * inv, s.Q * inv, s.U * inv, s.V * inv};
    }
};

// GRMHD grid plasma, FP64 throughout.
template<>
struct RadTraits<PolicyFP64, SceneGrmhd> {
    using Stokes = Stokes4<double>;
    using Co = Coeffs<double>;
    using Sample = GrmhdSample;
    __device__ static void zero(Stokes& s) { s = Stokes4<double>{0.0, 0.0, 0.0, 0.0}; }
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return grmhd_sample(c, r); }
    __device__ static Sample none() {
        Sample s;
        s.emitting = 0;
        return s;
    }
    __device__ static Co coeffs(const ImageConsts& c, const Sample& p, int f) {
        return grmhd_coefficients(c, p, c.freq[f]);
    }
    __device__ static RadDepths depths(const Co& co, double dls) { return radiation_depths(co, dls); }
    __device__ static Co coeffs_ctl(const ImageConsts& c, const Sample& p, int g) {
        return grmhd_coefficients(c, p, c.ctl_freq[g]);
    }
    __device__ static void step(Stokes& s, const Co& co, double h, const ImageConsts& c, int f) {
        stokes_apply(s, stokes_op(co, abs_val(h) * c.dlambda_scale[f]), co.jI, co.jQ, co.jU, co.jV);
    }
    __device__ static Stokes4<double> result(const Stokes& s, const ImageConsts&, int) { return s; }
};

// GRMHD grid plasma under the mixed policy: the grid gather, the fluid and
// field four-vectors and the screen angle stay FP64 (grmhd_sample, the
// reference's fluid_state); the thermal fit per frequency and the transfer
// are the mixed RIAF scene's.
__device__ __forceinline__ RiafSampleM grmhd_sample_to_m(const ImageConsts& c, const GrmhdSample& p) {
    RiafSampleM o;
    o.emitting = p.emitting && p.ne > 0.0;
    o.on_axis = 0;
    o.has_chi = p.has_chi;
    if (!o.emitting) return o;
    o.ne = p.ne;
    o.thetae = p.thetae;
    o.b = p.b;
    o.nu_fluid = p.nu_scale;
    o.cos_theta = p.ct;
    o.sin_theta = p.st;
    o.cos2chi = p.cos2chi;
    o.sin2chi = p.sin2chi;
    riaf_sample_thermal_m(c, o);
    return o;
}

__device__ __forceinline__ RiafSampleM grmhd_sample_m(const ImageConsts& c, const Ray& r) {
    return grmhd_sample_to_m(c, grmhd_sample(c, r));
}

template<>
struct RadTraits<PolicyMixed, SceneGrmhd> : RadTraits<PolicyMixed, SceneRiaf> {
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return grmhd_sample_m(c, r); }
};

// Slow light: the grid plasma interpolated in time between the resident
// snapshots around each sample's fluid time (grmhd_sample_series).
template<>
struct RadTraits<PolicyFP64, SceneGrmhdSlow> : RadTraits<PolicyFP64, SceneGrmhd> {
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return grmhd_sample_series(c, r); }
};

__device__ __forceinline__ RiafSampleM grmhd_series_sample_m(const ImageConsts& c, const Ray& r) {
    return grmhd_sample_to_m(c, grmhd_sample_series(c, r));
}

template<>
struct RadTraits<PolicyMixed, SceneGrmhdSlow> : RadTraits<PolicyMixed, SceneRiaf> {
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return grmhd_series_sample_m(c, r); }
};

// The RIAF in Boyer-Lindquist coordinates: the same plasma model, sampled
// in the ray's own BL components (riaf_sample_t<true>); under the mixed
// policy its sample feeds the factored fits.
template<>
struct RadTraits<PolicyFP64, SceneRiafBL> : RadTraits<PolicyFP64, SceneRiaf> {
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) { return riaf_sample_t<true>(c, r); }
};

__device__ __forceinline__ RiafSampleM riaf_sample_to_m(const ImageConsts& c, const RiafSample& p) {
    RiafSampleM o;
    o.emitting = p.emitting;
    o.on_axis = p.on_axis;
    o.has_chi = p.has_chi;
    if (!p.emitting) return o;
    o.ne = p.ne;
    o.thetae = p.thetae;
    o.b = p.b;
    o.nu_fluid = p.nu_fluid;
    o.cos_theta = p.cos_theta;
    o.sin_theta = p.sin_theta;
    o.cos2chi = p.cos2chi;
    o.sin2chi = p.sin2chi;
    riaf_sample_thermal_m(c, o);
    return o;
}

template<>
struct RadTraits<PolicyMixed, SceneRiafBL> : RadTraits<PolicyMixed, SceneRiaf> {
    __device__ static Sample sample(const ImageConsts& c, const Ray& r) {
        return riaf_sample_to_m(c, riaf_sample_t<true>(c, r));
    }
};

// A far-phase chart scene radiates nothing; its Stokes types are its
// record scene's.
template<class P, class B>
struct RadTraits<P, SceneFarCks<B>> : RadTraits<P, B> {};

// The scene's transport RHS under a policy.  The FP64 policy keeps the
// reference's operation order; the mixed policy uses the factored form
// (kp_geometry_mixed.cuh).
template<class P, class S>
__device__ __forceinline__ Ray policy_rhs(const ImageConsts& c, const Ray& X) {
    return S::template rhs<P::kMixed>(c, X);
}

// ---------------------------------------------------------------- RK jobs
// Runs one RK job from S with signed step h.  Outputs: next (endpoint), mid
// (sample point: the first half step for SD, the endpoint otherwise) and err
// (SD / CK only).  The stage arithmetic is the reference's (see file header).
// Cash-Karp attempt with the reference's stage coefficients (rk4.hpp:171-228).
template<class P, class SC>
__device__ __noinline__ void ck_job(const ImageConsts& c, const Ray& S, double h, Ray& next,
                                    Ray& mid, double& err) {
    {
        const Ray k1 = policy_rhs<P, SC>(c, S);
        Ray t;
        ray_axpy(t, S, h * 1.0 / 5.0, k1);
        const Ray k2 = policy_rhs<P, SC>(c, t);
        {
            const Ray* const kk[2] = {&k1, &k2};
            const double cc[2] = {3.0 / 40.0, 9.0 / 40.0};
            ray_lincomb<2>(t, S, h, kk, cc);
        }
        const Ray k3 = policy_rhs<P, SC>(c, t);
        {
            const Ray* const kk[3] = {&k1, &k2, &k3};
            const double cc[3] = {3.0 / 10.0, -9.0 / 10.0, 6.0 / 5.0};
            ray_lincomb<3>(t, S, h, kk, cc);
        }
        const Ray k4 = policy_rhs<P, SC>(c, t);
        {
            const Ray* const kk[4] = {&k1, &k2, &k3, &k4};
            const double cc[4] = {-11.0 / 54.0, 5.0 / 2.0, -70.0 / 27.0, 35.0 / 27.0};
            ray_lincomb<4>(t, S, h, kk, cc);
        }
        const Ray k5 = policy_rhs<P, SC>(c, t);
        {
            const Ray* const kk[5] = {&k1, &k2, &k3, &k4, &k5};
            const double cc[5] = {1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0,
                                  253.0 / 4096.0};
            ray_lincomb<5>(t, S, h, kk, cc);
        }
        const Ray k6 = policy_rhs<P, SC>(c, t);
        {
            const Ray* const kk[4] = {&k1, &k3, &k4, &k6};
            const double cc[4] = {37.0 / 378.0, 250.0 / 621.0, 125.0 / 594.0, 512.0 / 1771.0};
            ray_lincomb<4>(next, S, h, kk, cc);
        }
        Ray fourth;
        {
            const Ray* const kk[5] = {&k1, &k3, &k4, &k5, &k6};
            const double cc[5] = {2825.0 / 27648.0, 18575.0 / 48384.0, 13525.0 / 55296.0, 277.0 / 14336.0,
                                  1.0 / 4.0};
            ray_lincomb<5>(fourth, S, h, kk, cc);
        }
        err = control_error(next, fourth, max_val(c.tolerance, kTolFloor));
        mid = next;
    }
}

// Step-doubling attempt, RK4 step or composed RK4 pair as a stage loop around
// one RHS site.  Out of line: the caller's control state is saved once per
// job and the stage loop has the register file to itself.  `sure`: a
// step-doubling attempt that is certain to be accepted with the growth of err
// = 0 (certain_step) leaves its full chain out.  PAIRS: composed pairs occur
// (the surface-crossing search's trials).
template<class P, class SC, bool PAIRS>
__device__ __noinline__ void rk_job(int kind, const ImageConsts& c, const Ray& S, double h, bool sure,
                                    Ray& next, Ray& mid, double& err) {
    if (kind == kRkCK) {
        ck_job<P, SC>(c, S, h, next, mid, err);
        return;
    }
    // Stage schedule (see file header): SD = half chain (4), second half
    // chain (4), full chain (3); RK4 = 4; RK4x2 = 4 + 4.
    const bool pair = PAIRS && kind == kRkRK4x2;
    const int nstage = kind == kRkSD && !sure ? 11 : (kind == kRkRK4 ? 4 : 8);
    const double hs = kind == kRkSD || pair ? h * 0.5 : h;  // step of the first chain
    const double hh_s = 0.5 * hs;
    const double h6_s = hs / 6.0;
    const double hh_f = 0.5 * h;
    const double h6_f = h / 6.0;
    Ray X = S;   // RHS input
    Ray A;       // stage accumulator
    Ray R1;      // SD: k1 of S, then the two-half endpoint
    Ray R2;      // SD / RK4x2: the first chain's endpoint (half step)
#pragma unroll 1
    for (int st = 0; st < nstage; ++st) {
        const Ray k = policy_rhs<P, SC>(c, X);
        // position of this stage inside its 4-stage RK4 chain
        const int cs = st < 4 ? st : (st < 8 ? st - 4 : st - 7);
        const bool full_chain = kind == kRkSD && st >= 8;
        const bool second_chain = st >= 4 && st < 8;
        const double hh = full_chain ? hh_f : hh_s;
        const double hl = full_chain ? h : hs;       // last-stage step of the chain
        const double h6 = full_chain ? h6_f : h6_s;
        const Ray& base = second_chain ? R2 : S;
        if (cs == 0) {
            A = k;
            if (st == 0 && kind == kRkSD) R1 = k;
            ray_axpy(X, base, hh, k);
        } else if (cs == 1) {
            ray_acc(A, k, 2.0);
            ray_axpy(X, base, hh, k);
        } else if (cs == 2) {
            ray_acc(A, k, 2.0);
            ray_axpy(X, base, hl, k);
        } else {
            ray_add(A, k);
            if (st == 3) {
                if (kind == kRkRK4) {
                    ray_axpy(next, S, h6, A);
                } else {
                    ray_axpy(R2, S, h6, A);  // half step endpoint
                    X = R2;
                }
            } else if (st == 7) {
                if (pair || sure) {
                    ray_axpy(next, R2, h6, A);
                    mid = R2;
                } else {
                    // two_half = R2 + (hs/6) A; start the full chain from k1 of S
                    Ray two_half;
                    ray_axpy(two_half, R2, h6, A);
                    A = R1;
                    ray_axpy(X, S, hh_f, R1);
                    R1 = two_half;
                    // the full chain's first stage (k1) is already done: advance
                    // its position counter by running stages 8..10 as cs 1..3.
                }
            } else {  // st == 10: full step endpoint
                Ray full;
                ray_axpy(full, S, h6_f, A);
                err = control_error(full, R1, max_val(c.tolerance, kTolFloor));
                next = R1;
                mid = R2;
            }
        }
    }
    if (kind == kRkRK4 || pair) mid = next;
    if (nstage < 11) err = 0.0;
}

}  // namespace kp
