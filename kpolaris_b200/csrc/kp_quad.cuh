// kp_quad.cuh -- the ray engine on quads: four consecutive lanes of a warp
// advance one ray.  Lane `role` of a quad holds one of the ray's four
// vectors (0: position x, 1: wavevector k, 2: e1, 3: e2, the record's order)
// and every per-ray scalar of the control state (same value in the four).
//
// Why four lanes: a ray is one serial chain -- the longest rays of an image
// take 2,000 to 18,000 radiating steps of 11 right-hand sides each -- and an
// image ends with its longest ray.  One lane per ray made every instruction
// of the three transports and of the four frequencies part of that chain and
// needed 255 registers plus spills, which left 8 warps per SM and 24 us per
// radiating step.  On a quad each lane contracts the connection with its own
// vector, adds up its own RK4 stages and transfers its own frequency.  The
// connection of the point and what depends on k alone are evaluated by all
// four lanes: exchanging them costs more shuffles than it saves.
//
// The lanes of a warp run the RK job, the gathers and the reductions
// together (shuffles name the full warp); the control between them may
// diverge from quad to quad.  Every operation on a component is that of the
// one-lane form (kp_integrate.cuh), in its order, so the FP64 policy's images
// do not change.
#pragma once

#include "kp_far_steps.cuh"
#include "kp_persistent.cuh"

namespace kp {

constexpr unsigned kFullWarp = 0xffffffffu;

// The value lane `role` of the caller's quad holds.
__device__ __forceinline__ double quad_get(double v, int role) { return __shfl_sync(kFullWarp, v, role, 4); }

__device__ __forceinline__ D4 quad_get4(const D4& v, int role) {
    return d4(quad_get(v.v[0], role), quad_get(v.v[1], role), quad_get(v.v[2], role), quad_get(v.v[3], role));
}

// Components 1..3 of lane `role`'s vector (0 in component 0).
__device__ __forceinline__ D4 quad_get3(const D4& v, int role) {
    return d4(0.0, quad_get(v.v[1], role), quad_get(v.v[2], role), quad_get(v.v[3], role));
}

__device__ __forceinline__ Ray quad_ray(const D4& v) {
    Ray s;
    s.x = quad_get4(v, 0);
    s.k = quad_get4(v, 1);
    s.e1 = quad_get4(v, 2);
    s.e2 = quad_get4(v, 3);
    return s;
}

__device__ __forceinline__ bool quad_all(bool p) {
    const unsigned b = __ballot_sync(kFullWarp, p);
    return ((b >> (threadIdx.x & 28u)) & 15u) == 15u;
}

__device__ __forceinline__ int quad_max(int v) {
    v = max(v, __shfl_xor_sync(kFullWarp, v, 1));
    return max(v, __shfl_xor_sync(kFullWarp, v, 2));
}

__device__ __forceinline__ double quad_max(double v) {
    v = max_val(v, __shfl_xor_sync(kFullWarp, v, 1));
    return max_val(v, __shfl_xor_sync(kFullWarp, v, 2));
}

// finite_ray for a quad: 1 if all four vectors are finite.
__device__ __forceinline__ int quad_finite(const D4& v) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < 4; ++i) ok = ok && v.v[i] == v.v[i] && abs_val(v.v[i]) < kLarge;
    return quad_all(ok);
}

// The derivative of this lane's vector X (policy_rhs).
template<class P, class SC>
__device__ __forceinline__ D4 quad_rhs(const typename SC::Geo& c, const D4& X, int role) {
    const D4 x = quad_get3(X, 0);
    const D4 k = quad_get4(X, 1);
    const D4 d = SC::template transport<P::kMixed>(c, x, k, X);
    return role == 0 ? k : d;
}

template<class P, class SC>
__device__ __noinline__ D4 quad_rhs_call(const typename SC::Geo& c, const D4& X, int role) {
    return quad_rhs<P, SC>(c, X, role);
}

__device__ __forceinline__ void d4_axpy(D4& out, const D4& y, double a, const D4& x) {
#pragma unroll
    for (int i = 0; i < 4; ++i) out.v[i] = y.v[i] + x.v[i] * a;
}

__device__ __forceinline__ void d4_acc(D4& acc, const D4& x, double a) {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc.v[i] = acc.v[i] + x.v[i] * a;
}

__device__ __forceinline__ void d4_add(D4& acc, const D4& x) {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc.v[i] = acc.v[i] + x.v[i];
}

template<int N>
__device__ __forceinline__ void d4_lincomb(D4& out, const D4& s, double h, const D4* const (&k)[N],
                                           const double (&c)[N]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double a = k[0]->v[i] * c[0];
#pragma unroll
        for (int j = 1; j < N; ++j) a = a + k[j]->v[i] * c[j];
        out.v[i] = s.v[i] + a * h;
    }
}

// control_error (kp_integrate.cuh) over the quad.  The norm visits x, k, e1,
// e2 per component, and max_val lets a later value replace a NaN: with a NaN
// among the sixteen ratios they are folded in that order.
template<bool MIXED>
__device__ __forceinline__ double quad_control_error(const D4& a, const D4& b, double tol) {
    const double lim = tol * (1.0 / 64.0);
    bool small = true;
    double m = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double d = abs_val(a.v[i] - b.v[i]);
        small = small && d <= lim;
        m = max_val(m, d);
    }
    small = quad_all(small);
    m = quad_max(m);
    if (__all_sync(kFullWarp, small)) return m;
    double e[4];
    bool nan = false;
    double n = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double s = max_val(1.0, max_val(abs_val(a.v[i]), abs_val(b.v[i])));
        const double d = abs_val(a.v[i] - b.v[i]);
        e[i] = MIXED && s < 1e150 ? d * kp_recip(s) : d / s;
        nan = nan || !(e[i] == e[i]);
        n = max_val(n, e[i]);
    }
    n = quad_max(n);
    if (__any_sync(kFullWarp, nan)) {
        n = 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int r = 0; r < 4; ++r) n = max_val(n, quad_get(e[i], r));
    }
    return small ? m : n;
}

// Cash-Karp attempt (ck_job).
template<class P, class SC>
__device__ __noinline__ void quad_ck_job(const typename SC::Geo& c, double tolerance, const D4& S, double h, int role, D4& next,
                                         double& err) {
    const D4 k1 = quad_rhs_call<P, SC>(c, S, role);
    D4 t;
    d4_axpy(t, S, h * 1.0 / 5.0, k1);
    const D4 k2 = quad_rhs_call<P, SC>(c, t, role);
    {
        const D4* const kk[2] = {&k1, &k2};
        const double cc[2] = {3.0 / 40.0, 9.0 / 40.0};
        d4_lincomb<2>(t, S, h, kk, cc);
    }
    const D4 k3 = quad_rhs_call<P, SC>(c, t, role);
    {
        const D4* const kk[3] = {&k1, &k2, &k3};
        const double cc[3] = {3.0 / 10.0, -9.0 / 10.0, 6.0 / 5.0};
        d4_lincomb<3>(t, S, h, kk, cc);
    }
    const D4 k4 = quad_rhs_call<P, SC>(c, t, role);
    {
        const D4* const kk[4] = {&k1, &k2, &k3, &k4};
        const double cc[4] = {-11.0 / 54.0, 5.0 / 2.0, -70.0 / 27.0, 35.0 / 27.0};
        d4_lincomb<4>(t, S, h, kk, cc);
    }
    const D4 k5 = quad_rhs_call<P, SC>(c, t, role);
    {
        const D4* const kk[5] = {&k1, &k2, &k3, &k4, &k5};
        const double cc[5] = {1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0, 253.0 / 4096.0};
        d4_lincomb<5>(t, S, h, kk, cc);
    }
    const D4 k6 = quad_rhs_call<P, SC>(c, t, role);
    {
        const D4* const kk[4] = {&k1, &k3, &k4, &k6};
        const double cc[4] = {37.0 / 378.0, 250.0 / 621.0, 125.0 / 594.0, 512.0 / 1771.0};
        d4_lincomb<4>(next, S, h, kk, cc);
    }
    D4 fourth;
    {
        const D4* const kk[5] = {&k1, &k3, &k4, &k5, &k6};
        const double cc[5] = {2825.0 / 27648.0, 18575.0 / 48384.0, 13525.0 / 55296.0, 277.0 / 14336.0, 1.0 / 4.0};
        d4_lincomb<5>(fourth, S, h, kk, cc);
    }
    err = quad_control_error<P::kMixed>(next, fourth, max_val(tolerance, kTolFloor));
}

// ---- the far field of the mixed policy
// Beyond the radiating sphere a ray is transported and nothing else, and its
// steps are those the step control is known to take (macro_run).  There the
// engine takes a run of steps at once: the ray moves by their sum, the step
// counters by their number, and the step control stays where they leave it,
// so the steps inside the sphere fall where they fell.  The distance is
// bridged by Gragg's modified midpoint rule with 2, 4, 6 and 8 substeps
// extrapolated to zero step (W. Gragg, SIAM J. Numer. Anal. 2 (1965) 384;
// Hairer, Norsett, Wanner, Solving ODEs I, II.9: order 8), 21 right-hand
// sides in FP64 for up to hundreds of steps of 11.  A 256^2 image has 908 far
// steps per ray: 147 ms of an 8 x 256^2 step one by one, 45 ms bridged.
constexpr int kRkMacro = 4;

template<class P, class SC>
__device__ __forceinline__ D4 quad_macro_step(const ImageConsts& c, const D4& S, double H, int role) {
    const typename SC::Geo geo = SC::geo(c);
    const D4 f0 = quad_rhs<P, SC>(geo, S, role);
    D4 C[3], t;
#pragma unroll 1
    for (int j = 0; j < 4; ++j) {
        const int n = 2 * j + 2;
        const double hs = H * (j == 0 ? 0.5 : (j == 1 ? 0.25 : (j == 2 ? 1.0 / 6.0 : 0.125)));
        D4 z0 = S, z1, f;
        d4_axpy(z1, S, hs, f0);
#pragma unroll 1
        for (int i = 1;; ++i) {
            f = quad_rhs<P, SC>(geo, z1, role);
            if (i == n) break;
            const D4 z2 = z0;
            z0 = z1;
            d4_axpy(z1, z2, 2.0 * hs, f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            t.v[i] = macro_row(j, 0.5 * (z1.v[i] + (z0.v[i] + hs * f.v[i])), C[0].v[i], C[1].v[i], C[2].v[i]);
    }
    return t;
}

// The RK jobs of a warp's quads (rk_job's outputs for this lane's vector).
// Every lane of the warp calls it; quads without a job (kind < 0) compute
// along on what they hold and their outputs mean nothing.  A step-doubling
// attempt runs three chains of four stages (half step, second half step, full
// step with its first derivative reused), a composed pair two, a single step
// one.  `sure`: the attempt is certain to be accepted with the growth of err =
// 0 (certain_step); if the warp's other attempts are too, the full chain is
// left out.
template<class P, class SC, bool MACRO>
__device__ __forceinline__ void quad_job(int kind, const ImageConsts& c, const D4& S, double h, int role, bool sure,
                                         D4& next, D4& mid, double& err) {
    err = 0.0;
    const typename SC::Geo geo = SC::geo(c);
    const bool ck = kind == kRkCK;
    if (__any_sync(kFullWarp, ck)) {
        D4 n;
        double e;
        quad_ck_job<P, SC>(geo, c.tolerance, S, h, role, n, e);
        if (ck) {
            next = n;
            mid = n;
            err = e;
        }
        if (!__any_sync(kFullWarp, kind >= 0 && !ck)) return;
    }
    const bool macro = MACRO && kind == kRkMacro;
    if constexpr (MACRO) {
        if (__any_sync(kFullWarp, macro)) {
            const D4 n = quad_macro_step<P, SC>(c, S, h, role);
            if (macro) next = n;
            if (!__any_sync(kFullWarp, kind >= 0 && !macro && !ck)) return;
        }
    }
    const bool sd = kind == kRkSD, single = kind == kRkRK4;
    const int nchain = __any_sync(kFullWarp, sd && !sure) ? 3 : (__any_sync(kFullWarp, sd || kind == kRkRK4x2) ? 2 : 1);
    D4 B = S;             // chain base
    D4 K1, R2, end, A, X = S, k;
    double hc = single ? h : h * 0.5;
#pragma unroll 1
    for (int chain = 0; chain < nchain; ++chain) {
        // acc = ((k1 + 2 k2) + 2 k3) + k4, around one right-hand side: three
        // copies of it outgrow the innermost instruction cache
        const double hh = 0.5 * hc;
#pragma unroll 1
        for (int st = chain < 2 ? 0 : 1;; ++st) {
            k = quad_rhs<P, SC>(geo, X, role);
            if (st == 3) break;
            if (st == 0) {
                A = k;
                if (chain == 0) K1 = k;
            } else {
                d4_acc(A, k, 2.0);
            }
            d4_axpy(X, B, st == 2 ? hc : hh, k);
        }
        d4_add(A, k);
        d4_axpy(end, B, hc / 6.0, A);
        if (chain == 0) {
            R2 = end;
            B = end;
            X = end;
        } else if (chain == 1) {
            if (nchain == 2) break;
            // the full chain from S, its first derivative known
            A = K1;
            K1 = end;  // the two-half endpoint
            B = S;
            hc = h;
            d4_axpy(X, S, 0.5 * h, A);
        }
    }
    if (nchain == 3) {
        const double e = quad_control_error<P::kMixed>(end, K1, max_val(c.tolerance, kTolFloor));
        if (sd) err = e;
        end = K1;
    }
    if (ck || macro) return;
    next = single ? R2 : end;
    mid = sd ? R2 : next;
}

// The run of steps to bridge from a step just issued (count 0: take the
// step): a step-doubling or a fixed step, in Cartesian Kerr-Schild.
template<class SC, class LS>
__device__ __forceinline__ MacroRun far_run(const ImageConsts& c, const LS& st, double r, double xk, double v,
                                            double dir, bool pass_a, int left) {
    const MacroRun none = {0, 0.0, 0.0};
    if (!SC::chart_active(c) || st.rk_kind != (c.adaptive ? kRkSD : kRkRK4)) return none;
    const double h = abs_val(st.h_try);
    const MacroRun run = macro_run(c, r, xk, v, h, c.adaptive ? c.max_step : h, dir, pass_a, left);
    // one or two steps cost less as themselves
    return run.count >= 3 ? run : none;
}

// A claimed ray enters the far phase's chart (a record parked for this phase
// already holds it).
template<class SC, class LS>
__device__ __forceinline__ void enter_chart(LS& st, const ImageConsts& c, Ray& S) {
    if constexpr (SC::kFarChart) {
        if (!st.chart && SC::chart_active(c)) {
            st.x3_ref = S.x.v[3];
            S = SC::to_phase(c, S);
            st.chart = 1;
        }
    }
}

// A phase kernel of the wavefront engine on quads: persistent_body's control
// machine, one ray per quad.  With kPhaseAll: the rays [fresh_begin,
// fresh_end) of job 0, `per_warp` of them to each warp of the grid.  SHARED: the
// launch has rays of lane images too, which a lane kernel takes.
template<class P, int PHASE, class SC = SceneRiaf, bool SHARED = false>
__device__ __forceinline__ void quad_body(const WaveDesc& W, int per_warp = 8) {
    constexpr bool kAll = PHASE == kPhaseAll;
    constexpr bool kPassA = PHASE != kPhaseNearB;   // pass-A steps run here
    constexpr bool kPassB = PHASE != kPhaseNearA;   // pass-B steps run here
    constexpr bool kCross = kAll || PHASE == kPhaseNearA;  // surface-crossing search
    // the mixed policy's far field takes many steps at once (quad_macro_step)
    constexpr bool kMacro = P::kMixed && PHASE == kPhaseFar && SC::kCksRhs;
    constexpr bool kRad = kAll || PHASE == kPhaseNearB;    // radiative transfer
    const int lane = threadIdx.x & 31, role = lane & 3, quad = lane >> 2;
    using RT = RadTraits<P, SC>;
    LaneState st;
    st.mode = kIdle;
    st.job = 0;
    st.rk_kind = -1;
    // a quad that never gets a ray computes along on an ordinary point: the
    // origin would take the warp through the rare paths
    D4 V = d4(1.0, 2.0, 0.4, 0.3), best = V;
    double r_top = 0.0;  // radius of the ray's position at the loop top
    typename RT::Stokes stokes;
    unsigned my_id = 0;
    int exhausted = 0;
    long long quad_jobs = 0;
    const JobDesc* J = W.jobs;
    const long long nfresh = W.fresh_end - W.fresh_begin;
    long long total_in = 0;
    bool claims = false;
    if constexpr (kAll) {
        const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        const long long pixel = warp * per_warp + quad;
        if (quad < per_warp && pixel < nfresh) {
            Ray S;
            start_ray<SC>(st, S, J, 0, int(pixel));
            V = role == 0 ? S.x : (role == 1 ? S.k : (role == 2 ? S.e1 : S.e2));
            r_top = SC::template top_radius<P::kMixed>(J->c, S.x);
        }
    } else {
        total_in = wave_rays(W);
        // With fewer rays than quads the rays spread over the warps: a warp's
        // issue slots then serve fewer rays.
        const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
        claims = total_in >= 8 * warps || quad < int((total_in + warps - 1) / warps);
    }

#pragma unroll 1
    while (true) {
        bool forward = false;
        if constexpr (!kAll) {
            // ------------------------------------------------------------ claim
            // The far phase refills a warp as a whole: its rays then stay in
            // step, all in a bridged run or all in an ordinary step (79 -> 30 ms
            // per 8 x 256^2 step against refilling quad by quad).
            const bool busy = kMacro && __any_sync(kFullWarp, st.mode != kIdle);
            bool foreign = false, pushing = false;
#pragma unroll 1
            do {
                foreign = false;
                const bool want = claims && !exhausted && st.mode == kIdle && !busy && !forward;
                const unsigned need = __ballot_sync(kFullWarp, want && role == 0);
                if (need) {
                    unsigned long long base = 0;
                    if (lane == 0) base = atomicAdd(W.in_head, (unsigned long long)__popc(need));
                    base = __shfl_sync(kFullWarp, base, 0);
                    if (want) {
                        const long long k = (long long)(base + __popc(need & ((1u << (quad * 4)) - 1u)));
                        if (k >= total_in) {
                            exhausted = 1;
                        } else if (k < nfresh) {
                            // a fresh camera ray: locate its job and start pass A
                            const long long id = W.fresh_begin + k;
                            int lo = 0, hi = W.njobs - 1;
                            while (lo < hi) {
                                const int mid = (lo + hi + 1) >> 1;
                                if (W.jobs[mid].ray_begin <= id) lo = mid; else hi = mid - 1;
                            }
                            my_id = unsigned(id);
                            J = &W.jobs[lo];
                            Ray S;
                            start_ray<SC>(st, S, J, lo, int(id - J->ray_begin));
                            enter_chart<SC>(st, J->c, S);
                            V = role == 0 ? S.x : (role == 1 ? S.k : (role == 2 ? S.e1 : S.e2));
                            r_top = SC::template top_radius<P::kMixed>(J->c, S.x);
                        } else if (SHARED && !of_form(W, W.in_ids[k - nfresh], 0)) {
                            foreign = true;
                        } else if (W.budget > 0 && quad_jobs >= W.budget) {
                            // past the budget: hand the id on untouched (below)
                            my_id = W.in_ids[k - nfresh];
                            forward = true;
                        } else {
                            // a parked ray: resume from its record
                            my_id = W.in_ids[k - nfresh];
                            const RayRecord& rec = W.pool[my_id];
                            memcpy(&st, rec.st, kLaneStateBytes<PHASE>);
                            J = &W.jobs[st.job];
                            if constexpr (SC::kFarChart) {
                                Ray S = rec.S;
                                const bool paused = st.chart;
                                enter_chart<SC>(st, J->c, S);
                                V = role == 0 ? S.x : (role == 1 ? S.k : (role == 2 ? S.e1 : S.e2));
                                r_top = paused ? st.start_r : SC::template top_radius<P::kMixed>(J->c, S.x);
                            } else {
                                V = reinterpret_cast<const D4*>(&rec.S)[role];
                                r_top = SC::template top_radius<P::kMixed>(J->c, rec.S.x);
                            }
                            if constexpr (kRad) memcpy(&stokes, rec.stokes + 4 * role, sizeof(stokes));
                        }
                    }
                }
                pushing = pushing || need;
            } while (SHARED && __any_sync(kFullWarp, foreign));
            if (pushing) queue_push(W.out_ids[PHASE], W.out_count[PHASE], forward && role == 0, my_id);
        }
        const bool active = st.mode != kIdle;
        // The block's warps leave the loop together: the barriers are reached by
        // all of them in every iteration.  A quad that forwarded an id has more
        // input to claim.
        if (!__syncthreads_or(active || forward)) break;

        // ---------------------------------------------- control before the job
        int dest = -1;  // phase the ray is handed to (PHASE itself: its next launch)
        MacroRun run_of = {0, 0.0, 0.0};  // steps this job bridges; none: an ordinary step
        double xk = 0.0, speed = 0.0;
        if constexpr (kMacro) {
            const D4 x = quad_get3(V, 0), k = quad_get3(V, 1);
            xk = x.v[1] * k.v[1] + x.v[2] * k.v[2] + x.v[3] * k.v[3];
            speed = sqrt(k.v[1] * k.v[1] + k.v[2] * k.v[2] + k.v[3] * k.v[3]);
        }
        if constexpr (kPassA) {
            if (active && st.mode == kAStep && st.rk_kind < 0) {
                const ImageConsts& c = J->c;
                const int want_phase = kAll ? PHASE : phase_of(c, 0, r_top);
                if (want_phase != PHASE) {
                    dest = want_phase;
                } else if (!kAll && W.budget > 0 && quad_jobs >= W.budget) {
                    dest = PHASE;
                } else if (st.n >= c.max_steps) {
                    // pass-A loop top (pass_b.hpp:793-838)
                    st.mode = kEndA;
                } else {
                    if (!st.entered) {
                        if (r_top <= c.outer_radius) {
                            st.entered = 1;
                            st.inside = 0;
                        }
                    } else if (r_top - c.inner_radius <= 0.0) {
                        st.reason = kReachedInner;
                        st.mode = kEndA;
                    } else if (st.inside > 0 && r_top >= c.outer_radius) {
                        st.reason = kEscaped;
                        st.mode = kEndA;
                    }
                    if (st.mode == kAStep) {
                        st.old_r = r_top;
                        double mn = c.min_step_abs;
                        if (abs_val(st.h_current) < mn) mn = abs_val(st.h_current);
                        issue_step(st, c, st.h_current, mn, c.max_step);
                        if constexpr (kMacro) {
                            if (!st.entered)
                                run_of = far_run<SC>(c, st, r_top, xk, speed, -1.0, true, c.max_steps - st.n);
                        }
                    }
                }
            }
            if (active && dest < 0 && st.mode == kEndA) {
                // end of pass A (pass_b.hpp:940-955)
                const ImageConsts& c = J->c;
                if (st.entered && (st.reason == kReachedInner || st.reason == kEscaped)) {
                    st.in_b = 1;
                    st.mode = kBStep;
                    st.rk_kind = -1;
                    st.steps = 0;
                    st.reached = 0;
                    st.h_current = c.step;
                    st.cap = c.max_radiation_step > 0.0 ? c.max_radiation_step : c.max_step;
                    // pass B starts from zero Stokes, kept in the record until
                    // the ray reaches the radiating phase
                    RT::zero(stokes);
                    if constexpr (!kAll) memcpy(W.pool[my_id].stokes + 4 * role, &stokes, sizeof(stokes));
                } else {
                    st.mode = kDone;
                }
            }
        }
        if (active && dest < 0 && st.mode == kBStep && st.rk_kind < 0) {
            const ImageConsts& c = J->c;
            if (st.reached || st.steps >= c.max_steps) {
                st.mode = kDone;
            } else {
                const int want_phase = kAll ? PHASE : phase_of(c, 1, r_top);
                if (want_phase != PHASE) {
                    dest = want_phase;
                } else if (!kAll && W.budget > 0 && quad_jobs >= W.budget) {
                    dest = PHASE;
                } else {
                    // pass-B loop top (pass_b.hpp:966-981)
                    double h = st.h_current;
                    st.start_r = r_top;
                    if (st.start_r <= c.outer_radius && st.cap > 0.0) h = min_val(h, st.cap);
                    st.hB = h;
                    issue_step(st, c, h, c.min_step_abs, c.max_step);
                    if constexpr (kMacro) {
                        run_of = far_run<SC>(c, st, r_top, xk, speed, 1.0, false, c.max_steps - st.steps);
                    }
                }
            }
        }
        const bool park = !kAll && dest >= 0;
        if constexpr (!kAll) {
            if constexpr (SC::kFarChart) {
                // leaving the phase: back to the records' chart; parked for
                // this phase (a tick budget): kept as is, so the ray resumes
                // bit for bit as if it had not been parked
                const bool leave = park && st.chart && dest != PHASE;
                if (__any_sync(kFullWarp, leave)) {
                    const Ray S = quad_ray(V);
                    if (leave) {
                        const Ray R = SC::to_record(J->c, S, st.x3_ref);
                        V = role == 0 ? R.x : (role == 1 ? R.k : (role == 2 ? R.e1 : R.e2));
                        st.chart = 0;
                    }
                }
            }
            if (park) {
                RayRecord& rec = W.pool[my_id];
                // a pause keeps the chart's radius too (start_r is unused
                // here): evaluated again at another call site, its fused
                // operations may differ
                if constexpr (SC::kFarChart) st.start_r = r_top;
                reinterpret_cast<D4*>(&rec.S)[role] = V;
                if (role == 0) memcpy(rec.st, &st, kLaneStateBytes<PHASE>);
                if constexpr (kRad) memcpy(rec.stokes + 4 * role, &stokes, sizeof(stokes));
            }
            // A quad past its budget keeps claiming and parks each claimed ray at
            // once, so every input ends the launch finished or in a queue.
            if (__any_sync(kFullWarp, park)) {
#pragma unroll
                for (int d = 0; d < kPhases; ++d)
                    queue_push(W.out_ids[d], W.out_count[d], dest == d && role == 0, my_id);
            }
            if (park) st.mode = kIdle;
        }

        // ------------------------------------------------------------ RK job
        const bool crossing_job = kCross && (st.mode == kACrossHi || st.mode == kACrossTrial);
        const bool run = !park && (st.mode == kAStep || crossing_job || st.mode == kBStep || st.mode == kBCamCross);
        D4 next = V, mid = V;
        double err = 0.0, next_r = 0.0;
        if (__any_sync(kFullWarp, run)) {
            // quads without a job compute along under the constants of one that has one
            int kind = -1;
            double hj = 0.0;
            const int src = __ffs(__ballot_sync(kFullWarp, run)) - 1;
            const unsigned long long jr = __shfl_sync(kFullWarp, reinterpret_cast<unsigned long long>(J), src);
            const ImageConsts& c = run ? J->c : reinterpret_cast<const JobDesc*>(jr)->c;
            if (run) {
                kind = crossing_job ? (J->c.adaptive ? kRkRK4x2 : kRkRK4) : st.rk_kind;
                hj = crossing_job ? (st.mode == kACrossHi ? st.full_h : st.full_h * st.trial) : st.h_try;
                if (kMacro && run_of.count > 0) {
                    kind = kRkMacro;
                    hj = st.h_try < 0.0 ? -run_of.length : run_of.length;
                }
            }
            bool sure = false;
            if constexpr (SC::kCksRhs) {
                double m = 0.0;
#pragma unroll
                for (int i = 0; i < 4; ++i) m = max_val(m, abs_val(V.v[i]));
                const double z = (V.v[0] + V.v[1]) + (V.v[2] + V.v[3]);
                if (!(z - z == 0.0)) m = kLarge;  // a NaN or an infinity among them
                const double km = quad_get(m, 1), w = quad_max(role == 0 ? 0.0 : m);
                if (run && kind == kRkSD && SC::chart_active(c)) {
                    const double tol = max_val(c.tolerance, kTolFloor);
                    sure = certain_step(c.mass, r_top, km, w, hj, (abs_val(hj) == st.ctl_max ? 0.25 : 1.0 / 64.0) * tol);
                }
            }
            quad_job<P, SC, kMacro>(kind, c, V, hj, role, sure, next, mid, err);
            next_r = SC::template top_radius<P::kMixed>(c, quad_get3(next, 0));
        }
        if (!kAll && run && ++quad_jobs > (1LL << 30)) {
            st.reason = kInvalidState;
            st.mode = kDone;
            st.in_b = 0;
            atomicExch(W.status, 2);
        }
        // In step, the block's warps run one region of code at a time, which
        // keeps it in the instruction caches (8 x 256^2: near-B 231 -> 190 ms,
        // near-A 63 -> 57 ms, far 29.6 -> 26 ms).
        __syncthreads();
        int next_finite = 1;
        if constexpr (kPassA) next_finite = quad_finite(next);

        // ----------------------------------------------- control after the job
        bool proceed = false;  // a pass-B step whose radiation is due
        int crosses = 1;
        double h = 0.0;
        if (kMacro && run && run_of.count > 0) {
            V = next;
            r_top = next_r;
            st.rk_kind = -1;
            if (J->c.adaptive) st.h_current = st.h_try < 0.0 ? -run_of.next_h : run_of.next_h;
            if (st.mode == kAStep) {
                st.pa_steps += run_of.count;
                st.n += run_of.count;
            } else {
                st.cap = J->c.max_step;
                st.steps += run_of.count;
            }
            if (!(next_r > J->c.far_radius)) atomicExch(W.status, 3);
        } else if (kPassA && run && st.mode == kAStep) {
            const ImageConsts& c = J->c;
            bool accepted = true;
            const double used_h = st.h_try;
            if (st.rk_kind != kRkRK4) {
                const double tol = max_val(c.tolerance, kTolFloor);
                if (err <= tol) {
                    st.h_current = accepted_next_h<P::kMixed>(st.h_try, err, tol, st.ctl_min, st.ctl_max, st.req_h);
                } else {
                    accepted = false;
                    if (rejected_attempt<P::kMixed>(st, err, tol)) {
                        st.rk_kind = -1;
                        if (abs_val(st.h_current) <= c.min_step_abs * 1.0001) {
                            st.reason = kAdaptiveUnderflow;
                            st.mode = kEndA;
                        } else {
                            st.n += 1;  // `continue` of the pass-A for loop
                        }
                    }
                }
            }
            if (accepted) {
                // pass_b.hpp:864-937
                st.rk_kind = -1;
                const double old_r = st.old_r;
                if (!st.entered && next_r <= c.outer_radius) {
                    st.entered = 1;
                    st.inside = 0;
                } else if (!st.entered && next_r >= old_r) {
                    V = next;
                    r_top = next_r;
                    st.pa_steps += 1;
                    st.reason = kEscaped;
                    st.mode = kEndA;
                }
                if (st.mode == kAStep) {
                    int crossing = kNone;
                    if (st.entered && old_r - c.inner_radius > 0.0 && next_r - c.inner_radius <= 0.0) {
                        crossing = kReachedInner;
                    } else if (st.entered && st.inside > 0 && old_r < c.outer_radius && next_r >= c.outer_radius) {
                        crossing = kEscaped;
                    }
                    if (crossing != kNone) {
                        if constexpr (kCross) {
                            st.cross_reason = crossing;
                            st.surf = crossing == kReachedInner ? c.inner_radius : c.outer_radius;
                            st.full_h = used_h;
                            best = V;
                            st.lo = 0.0;
                            st.hi = 1.0;
                            st.flo = r_top - st.surf;
                            if (st.flo == 0.0 || !next_finite) {
                                st.pa_steps += 1;  // the event keeps the first state
                                st.reason = crossing;
                                st.mode = kEndA;
                            } else {
                                st.mode = kACrossHi;
                            }
                        } else {
                            atomicExch(W.status, 3);  // surfaces lie inside the near phase
                            st.reason = kInvalidState;
                            st.mode = kDone;
                        }
                    } else {
                        V = next;
                        r_top = next_r;
                        st.pa_steps += 1;
                        if (st.entered) st.inside += 1;
                        st.n += 1;
                    }
                }
            }
        } else if (kCross && run && (st.mode == kACrossHi || st.mode == kACrossTrial)) {
            bool finish = false;
            if (st.mode == kACrossHi) {
                if (!next_finite) {
                    finish = true;
                } else {
                    const double fhi = next_r - st.surf;
                    if (!(fhi == fhi) || abs_val(fhi) >= kLarge) {
                        finish = true;
                    } else if (fhi == 0.0) {
                        best = next;
                        finish = true;
                    } else if ((st.flo > 0.0) == (fhi > 0.0)) {
                        finish = true;
                    } else {
                        st.fhi = fhi;
                        st.iter = 0;
                        st.use_secant = 1;
                    }
                }
            } else {
                const double ft = next_finite ? next_r - st.surf : 0.0;
                if (!next_finite || !(ft == ft) || abs_val(ft) >= kLarge) {
                    st.hi = st.trial;
                    st.use_secant = 0;
                } else if (ft == 0.0) {
                    best = next;
                    finish = true;
                } else if ((st.flo > 0.0) == (ft > 0.0)) {
                    st.lo = st.trial;
                    st.flo = ft;
                    best = next;
                } else {
                    st.hi = st.trial;
                    st.fhi = ft;
                }
                st.iter += 1;
            }
            if (!finish && st.iter >= 12) finish = true;
            if (finish) {
                V = best;
                st.pa_steps += 1;
                st.reason = st.cross_reason;
                st.mode = kEndA;
            } else {
                st.trial = crossing_trial(st);
                st.mode = kACrossTrial;
            }
        } else if (kPassB && run && (st.mode == kBStep || st.mode == kBCamCross)) {
            const ImageConsts& c = J->c;
            const bool cam = st.mode == kBCamCross;
            proceed = true;
            h = st.hB;
            if (st.rk_kind != kRkRK4) {
                const double tol = max_val(c.tolerance, kTolFloor);
                if (err <= tol) {
                    h = abs_val(st.h_try);
                    if (!cam) st.h_current = abs_val(accepted_next_h<P::kMixed>(st.h_try, err, tol, st.ctl_min, st.ctl_max, st.req_h));
                } else {
                    proceed = false;
                    if (rejected_attempt<P::kMixed>(st, err, tol)) {
                        st.h_current = abs_val(st.h_current);
                        st.rk_kind = -1;
                        st.mode = kBStep;
                        if (!cam && st.h_current <= c.min_step_abs * 1.0001) {
                            // the slow-light window kernel reports max_steps here
                            // (slow_light_driver.hpp:1172-1177)
                            st.reason = SC::kSlowLight ? kMaxSteps : kAdaptiveUnderflow;
                            st.mode = kDone;
                        }
                    }
                }
            }
            if (proceed && !cam) {
                // camera surface (pass_b.hpp:999-1028)
                const double s0 = st.start_r - c.cam_radius;
                const double s1 = next_r - c.cam_radius;
                crosses = (s0 == 0.0 || s1 == 0.0) ? 1 : ((s0 < 0.0 && s1 > 0.0) || (s0 > 0.0 && s1 < 0.0));
                if (crosses) {
                    const double denom = s0 - s1;
                    const double frac = abs_val(denom) <= kTiny ? 1.0 : min_val(1.0, max_val(0.0, s0 / denom));
                    const double h_cross = h * frac;
                    if (abs_val(h_cross) <= 1e-14) {
                        h = 0.0;
                        next = V;
                        mid = V;
                        next_r = r_top;
                    } else if (frac < 0.999999999999) {
                        h = h_cross;
                        const double mn = min_val(c.min_step_abs, abs_val(h));
                        issue_step(st, c, h, mn, max_val(mn, abs_val(h)));
                        st.mode = kBCamCross;
                        st.hB = h;
                        proceed = false;
                    }
                }
            }
        }

        // ------------------------------------------------------- radiation
        if constexpr (kPassB) {
            if (__any_sync(kFullWarp, proceed)) {
                // radiation at the sample point (pass_b.hpp:1414-1496); each
                // lane takes one frequency, lanes past the image's last repeat it
                const ImageConsts& c = J->c;
                bool stopped = false;
                // a step without plasma: its coefficients are zero, its
                // transfer adds zero (the plain kernel's far field)
                bool empty = false;
                int required = 1, pred = 1;
                double local_max_rs = 0.0;
                typename RT::Co co;
                const Ray sample = quad_ray(mid);  // shuffled as what of it is read
                const int nf = c.nfreq < kMaxFreq ? c.nfreq : kMaxFreq;
                const int f = role < nf ? role : nf - 1;
                if (proceed) {
                    const double sample_r = SC::template top_radius<P::kMixed>(c, sample.x);
                    local_max_rs = (c.max_radiation_step > 0.0 &&
                                    (st.start_r <= c.outer_radius || sample_r <= c.outer_radius ||
                                     next_r <= c.outer_radius))
                                       ? c.max_radiation_step : 0.0;
                    bool radiating = sample_r - c.inner_radius > 0.0 && sample_r < c.outer_radius;
                    if constexpr (kRad) {
                        typename RT::Sample ps = RT::none();
                        if constexpr (SC::kSlowLight) {
                            // slow_light_driver.hpp:1295-1304: a radiating sample
                            // needs its fluid time among the resident snapshots;
                            // otherwise the ray ends where it stands
                            radiating = sample_r >= c.inner_radius && sample_r < c.outer_radius;
                            if (radiating && !SC::time_resident(c, sample)) {
                                st.reason = kSlowLightTimeExhausted;
                                st.mode = kDone;
                                stopped = true;
                            }
                        }
                        if (radiating && !stopped) ps = RT::sample(c, sample);
                        empty = kAll && !radiating;
                        if (empty) {
                            const RadDepths none = {0.0, 0.0, 0.0};
                            required = substeps_for(none, h, local_max_rs, c);
                            pred = substeps_for(none, st.h_current, local_max_rs, c);
                        } else if (!stopped) {
                            co = RT::coeffs(c, ps, f);
                            if (!c.faraday_rotation) co.rV = 0.0;
                            // Substep counts at h (required) and at h_current
                            // (predictive) in one pass: neither test changes h or
                            // h_current.  Over the image's frequencies, or over a
                            // separate step-control list (pass_b.hpp:1787-1833).
                            const bool fused = c.nctl == 0;
#pragma unroll 1
                            for (int g = role; g < (fused ? 4 : c.nctl); g += 4) {
                                typename RT::Co cg = co;
                                double dls = c.dlambda_scale[f];
                                if (!fused) {
                                    cg = RT::coeffs_ctl(c, ps, g);
                                    if (!c.faraday_rotation) cg.rV = 0.0;
                                    dls = c.ctl_dlambda_scale[g];
                                }
                                const RadDepths depth = RT::depths(cg, dls);
                                const int cand = substeps_for(depth, h, local_max_rs, c);
                                required = cand > required ? cand : required;
                                const int pc = substeps_for(depth, st.h_current, local_max_rs, c);
                                pred = pc > pred ? pc : pred;
                            }
                        }
                    } else if (local_max_rs > 0.0 || radiating) {
                        // far phase: every sample lies outside the radiating sphere
                        atomicExch(W.status, 3);
                    }
                }
                if constexpr (kRad) {
                    required = quad_max(required);
                    pred = quad_max(pred);
                }
                if (proceed && !stopped) {
                    if (kRad && required > 1 && h > c.min_step_abs * 1.0001) {
                        st.h_current = max_val(c.min_step_abs, over_pow2(h, required));
                        st.cap = st.h_current;
                    } else {
                        st.cap = c.max_step;
                        if (kRad && pred > 1 &&
                            (local_max_rs > 0.0 || c.max_radiation_depth > 0.0 || c.max_absorption_depth > 0.0 ||
                             c.max_faraday_depth > 0.0))
                            st.cap = max_val(c.min_step_abs, over_pow2(st.h_current, pred));
                        if constexpr (kRad) {
                            if (empty) {
                                if constexpr (kAll) RT::add_zero(stokes);
                            } else if (h > 0.0) {
                                RT::step(stokes, co, h, c, f);
                            }
                        }
                        V = next;
                        r_top = next_r;
                        st.steps += 1;
                        if (crosses) st.reached = 1;
                    }
                    st.mode = kBStep;
                    st.rk_kind = -1;
                }
            }
        }

        // the crossing search ends at a state whose radius was not kept
        if constexpr (kCross) {
            const bool ended = run && st.mode == kEndA;
            if (__any_sync(kFullWarp, ended)) {
                const double r = SC::template top_radius<P::kMixed>(J->c, quad_get3(V, 0));
                if (ended) r_top = r;
            }
        }

        // ------------------------------------------------------------ finish
        const bool done = !park && st.mode == kDone;
        if (__any_sync(kFullWarp, done)) {
            const Ray S = quad_ray(V);
            if (done) {
                const ImageConsts& c = J->c;
                PixelOut o;
                o.pass_a_steps = st.pa_steps;
                o.steps = st.in_b ? st.steps : 0;
                int reason = st.reason;
                if (st.in_b) {
                    if (st.reached) {
                        reason = kReachedCamera;
                    } else if (reason != kAdaptiveUnderflow && reason != kSlowLightTimeExhausted) {
                        reason = kMaxSteps;
                    }
                }
                o.reason = reason;
                const Ray cam = SC::camera(c, J->frame, st.pixel);
                // only the radiating phase carries the Stokes vector: it is in the record
                if constexpr (!kRad) {
                    if (st.in_b) memcpy(&stokes, W.pool[my_id].stokes + 4 * role, sizeof(stokes));
                }
                const int nf = c.nfreq < kMaxFreq ? c.nfreq : kMaxFreq;
                const int f = role < nf ? role : nf - 1;
                Stokes4<double> sd[1];
                sd[0] = st.in_b ? RT::result(stokes, c, f) : Stokes4<double>{0.0, 0.0, 0.0, 0.0};
                double obs[1][4];
                if constexpr (SC::kFarChart) {
                    const Ray S_rec = st.chart ? SC::to_record(c, S, st.x3_ref) : S;
                    finish_ray_scene<typename RecordScene<SC>::type, 1>(c, cam, S_rec, st.in_b, sd, o, obs);
                } else {
                    finish_ray_scene<SC, 1>(c, cam, S, st.in_b, sd, o, obs);
                }
                if (role < nf) {
                    const size_t idx = size_t(f) * size_t(J->npix) + size_t(st.pixel);
                    J->out.image_i[idx] = obs[0][0];
                    J->out.image_q[idx] = obs[0][1];
                    J->out.image_u[idx] = obs[0][2];
                    J->out.image_v[idx] = obs[0][3];
                }
                if (role == 0) {
                    store_diagnostics(J->out, st.pixel, o);
                    if constexpr (SC::kSlowLight) {
                        if (!st.in_b) J->out.basis_identity_error[st.pixel] = 0.0;
                    }
                    if (!kAll && W.job_done) atomicAdd(&W.job_done[st.job], 1u);
                }
                st.mode = kIdle;
            }
        }
    }
}

}  // namespace kp
