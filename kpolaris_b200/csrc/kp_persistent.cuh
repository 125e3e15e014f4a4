// kp_persistent.cuh -- the wavefront image kernels.  Lanes claim rays from a
// phase queue (fresh camera rays, then ray ids handed over by other phases),
// advance them one RK job per loop iteration through the pass-A / crossing /
// pass-B control machine, and either finish the pixel or park the ray's
// record in HBM for another phase (or for its own next launch when an iteration
// budget is set).  See kp_engine.cuh for the RK jobs.
//
// Three phases, one kernel each, so that the lanes of a warp run the same
// code and each kernel's instruction working set stays small (this file: what
// they share, and the far phase with one ray per lane; kp_quad.cuh: four lanes
// per ray):
//   far     rays beyond ImageConsts::fp32_radius, pass A and pass B: pure
//           transport (no surface lies within a step, no plasma is sampled);
//   near-A  pass A inside: the surface-crossing search, no radiation;
//   near-B  pass B inside: radiative transfer.
//
// Parking happens only at the top of the pass-A or pass-B loop, where the
// whole state is the record: a ray resumed from its record takes exactly the
// arithmetic it would have taken without parking, so results do not depend on
// how rays are distributed over launches, lanes or warps.
#pragma once

#include <cstddef>

#include "kp_engine.cuh"
#include "kp_far_steps.cuh"

namespace kp {

enum : int { kEndA = 7 };

// Control state of one ray (17 doubles + 17 ints, 208 bytes), in three
// parts: what every phase uses; what only the pass-A phases (far and
// near-A) use; the surface-crossing search (near-A).  A phase kernel moves
// only the parts it uses between its registers and the record, so the
// others hold no registers there; the record keeps them as the last phase
// that used them left them.
struct LaneState {
    // adaptive attempt sequence (rk4.hpp:108-161)
    double h_try, req_h, ctl_min, ctl_max;
    double h_current;
    // pass B (pass_b.hpp:940-1114)
    double cap, hB, start_r;
    int job, pixel, mode, in_b;
    int attempt, rk_kind;
    int pa_steps, reason;
    int steps, reached;
    // pass A (pass_b.hpp:786-938)
    double old_r;
    // far-phase chart scenes: the FMKS azimuth the ray entered the far
    // phase with, and whether S (here and in a record parked for the far
    // phase itself) holds the far phase's chart
    double x3_ref;
    int n, entered, inside;
    int chart;
    // surface-crossing search (pass_a_core.hpp:94-197)
    double lo, hi, flo, fhi, full_h, surf, trial;
    int cross_reason, iter, use_secant;
};
static_assert(sizeof(LaneState) <= sizeof(((RayRecord*)nullptr)->st), "LaneState must fit its record slot");
static_assert(offsetof(LaneState, old_r) % 8 == 0 && offsetof(LaneState, lo) % 8 == 0, "parts are whole doubles");

// Bytes of LaneState a phase kernel moves: near-B runs no pass-A step and
// never holds a far chart, far runs no crossing search, and a search never
// spans two launches.
template<int PHASE>
constexpr size_t kLaneStateBytes = PHASE == kPhaseNearB ? offsetof(LaneState, old_r) : offsetof(LaneState, lo);

template<class LS>
__device__ __forceinline__ void begin_adaptive(LS& L, double requested, double min_step, double max_step) {
    L.req_h = requested;
    L.ctl_min = min_step;
    L.ctl_max = max_step;
    double h = min_val(max_val(abs_val(requested), min_step), max_step);
    if (requested < 0.0) h = -h;
    L.h_try = h;
    L.attempt = 0;
}

// x^0.2 for x > 0: pow under the FP64 policy (the reference's); under the
// mixed policy Newton's iteration for y^5 = x from a single-precision
// exponential, two steps from 1e-6 to a few ulp (pow and its division cost a
// lone ray 900 cycles a step).  Out of range it is pow.
template<bool MIXED>
__device__ __forceinline__ double fifth_root(double x) {
    if constexpr (MIXED) {
        if (x > 1e-30 && x < 1e30) {
            double y = double(exp2f(0.2f * __log2f(float(x))));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double y2 = y * y, y4 = y2 * y2;
                y = y - (y4 * y - x) * kp_recip<double>(5.0 * y4);
            }
            return y;
        }
    }
    return pow(x, 0.2);
}

// Step growth after an accepted attempt (rk4.hpp:130-142).  With
// tol >= 64 err the factor 0.9 (tol/err)^0.2 is at least 2.07 and clamps to
// 2, so pow is evaluated only below that ratio (same result).
template<bool MIXED = false>
__device__ __forceinline__ double accepted_next_h(double h, double err, double tol, double min_step,
                                                  double max_step, double requested) {
    double factor = 2.0;
    if (err > 0.0 && !(tol >= 64.0 * err)) {
        factor = 0.9 * fifth_root<MIXED>(MIXED ? tol * kp_recip<double>(err) : tol / err);
        factor = min_val(2.0, max_val(0.2, factor));
    }
    double next_h = min_val(max_step, max_val(min_step, abs_val(h) * factor));
    if (requested < 0.0) next_h = -next_h;
    return next_h;
}

// A rejected attempt: shrink and retry, or give up (rk4.hpp:143-160).
// Returns 1 when the sequence is exhausted; L.h_current then holds the
// signed next_h of the failed sequence.
template<bool MIXED = false, class LS>
__device__ __forceinline__ int rejected_attempt(LS& L, double err, double tol) {
    L.attempt += 1;
    int exhausted = L.attempt >= 10;
    if (abs_val(L.h_try) <= L.ctl_min * 1.0001) {
        exhausted = 1;
    } else {
        double factor = 0.9 * pow(tol / max_val(err, kTiny), L.rk_kind == kRkCK ? 0.2 : 0.25);
        factor = min_val(0.8, max_val(0.1, factor));
        L.h_try *= factor;
    }
    if (exhausted) {
        const double next_abs = max_val(L.ctl_min, abs_val(L.h_try) * 0.5);
        L.h_current = L.req_h < 0.0 ? -next_abs : next_abs;
    }
    return exhausted;
}

template<class LS>
__device__ __forceinline__ void issue_step(LS& L, const ImageConsts& c, double h, double min_step, double max_step) {
    if (c.adaptive) {
        begin_adaptive(L, h, min_step, max_step);
        L.rk_kind = c.integrator == 1 ? kRkCK : kRkSD;
    } else {
        L.h_try = h;
        L.rk_kind = kRkRK4;
    }
}

template<int NF>
__device__ __forceinline__ void store_stokes_n(const ImageOutPtrs& out, int pixel, int npix, int nf,
                                               const double (&obs)[NF][4]) {
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        if (f < nf) {
            const size_t idx = size_t(f) * size_t(npix) + size_t(pixel);
            out.image_i[idx] = obs[f][0];
            out.image_q[idx] = obs[f][1];
            out.image_u[idx] = obs[f][2];
            out.image_v[idx] = obs[f][3];
        }
    }
}

// Warp-aggregated append of the ids of the lanes in `mask` to a queue.
__device__ __forceinline__ void queue_push(unsigned* ids, unsigned* count, bool push, unsigned id) {
    const unsigned FULL = 0xffffffffu;
    const unsigned m = __ballot_sync(FULL, push);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    unsigned base = 0;
    if (lane == leader) base = atomicAdd(count, unsigned(__popc(m)));
    base = __shfl_sync(FULL, base, leader);
    if (push) ids[base + __popc(m & ((1u << lane) - 1u))] = id;
}

// Initial control state of a camera ray at the top of pass A
// (pass_b.hpp:786-792).
template<class SC>
__device__ __forceinline__ void start_ray(LaneState& st, Ray& S, const JobDesc* J, int job, int pixel) {
    memset(&st, 0, sizeof(st));
    st.job = job;
    st.pixel = pixel;
    S = SC::camera(J->c, J->frame, pixel);
    st.reason = kMaxSteps;
    st.h_current = -abs_val(J->c.step);
    st.mode = kAStep;
    st.rk_kind = -1;
}

// Seeds the rays of newly admitted jobs: one thread per ray writes the ray's
// initial record (pass-A loop top) and appends its id to the far queue.
// entries: (job slot, first ray id, pixel count) with prefix sums of the
// counts in `prefix` (nentries + 1 values).
template<class SC>
__device__ __forceinline__ void seed_body(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix,
                                          int nentries, RayRecord* pool, unsigned* far_ids,
                                          unsigned* far_count) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < prefix[nentries];
    unsigned id = 0;
    if (live) {
        int lo = 0, hi = nentries - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (prefix[mid] <= i) lo = mid; else hi = mid - 1;
        }
        const SeedEntry e = entries[lo];
        const int pixel = int(i - prefix[lo]);
        id = unsigned(e.ray_base + pixel);
        LaneState st;
        Ray S;
        start_ray<SC>(st, S, &jobs[e.slot], e.slot, pixel);
        RayRecord& rec = pool[id];
        rec.S = S;
        memcpy(rec.st, &st, sizeof(LaneState));
    }
    queue_push(far_ids, far_count, live, id);
}

// Phase that advances a ray from the top of its pass-A or pass-B loop.
__device__ __forceinline__ int phase_of(const ImageConsts& c, int in_b, double r_bl) {
    if (r_bl > c.fp32_radius) return kPhaseFar;
    return in_b ? kPhaseNearB : kPhaseNearA;
}

// The scene a ray is finished in: a far-phase chart scene hands the ray
// back to the scene its records use.
template<class SC>
struct RecordScene {
    using type = SC;
};
template<class B>
struct RecordScene<SceneFarCks<B>> {
    using type = B;
};

// The far phase with one ray per lane, for the scenes and policies that take
// its steps one by one (FP64, and Boyer-Lindquist under either policy).  Pure
// transport: every lane runs the same instructions, and with tens of
// thousands of rays a lane per ray needs half the operations of a quad
// (kp_quad.cuh), which evaluates a point's connection four times.
template<class P, int NF, class SC = SceneRiaf>
__device__ __forceinline__ void far_body(const WaveDesc& W) {
    constexpr int PHASE = kPhaseFar;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    using RT = RadTraits<P, SC>;
    LaneState st;
    st.mode = kIdle;
    st.job = -1;
    st.rk_kind = -1;
    Ray S;
    typename RT::Stokes stokes[NF];
    unsigned my_id = 0;
    int exhausted = 0;
    long long lane_jobs = 0;
    const JobDesc* J = nullptr;
    const long long nfresh = W.fresh_end - W.fresh_begin;
    const long long total_in = nfresh + (long long)(W.in_ids ? *W.in_count : 0u);

#pragma unroll 1
    while (true) {
        // ------------------------------------------------------------ claim
        const bool want = !exhausted && st.mode == kIdle;
        bool forward = false;
        const unsigned need = __ballot_sync(FULL, want);
        if (need) {
            unsigned long long base = 0;
            const int leader = __ffs(need) - 1;
            if (lane == leader) base = atomicAdd(W.in_head, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (want) {
                const long long k = (long long)(base + __popc(need & ((1u << lane) - 1u)));
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
                    start_ray<SC>(st, S, J, lo, int(id - J->ray_begin));
                } else if (W.budget > 0 && lane_jobs >= W.budget) {
                    // past the budget: hand the id on untouched (below)
                    my_id = W.in_ids[k - nfresh];
                    forward = true;
                } else {
                    // a parked ray: resume from its record
                    my_id = W.in_ids[k - nfresh];
                    const RayRecord& rec = W.pool[my_id];
                    S = rec.S;
                    memcpy(&st, rec.st, kLaneStateBytes<PHASE>);
                    J = &W.jobs[st.job];
                }
            }
        }
        queue_push(W.out_ids[PHASE], W.out_count[PHASE], forward, my_id);
        const bool active = st.mode != kIdle;
        // The block leaves the loop together, so the barrier below is
        // reached by every thread of the block in every iteration.  A lane
        // that forwarded an id has more input to claim: it keeps the block
        // in the loop like an active lane.
        if (!__syncthreads_or(active || forward)) break;

        // ---------------------------------------------- control before the job
        int dest = -1;  // phase the ray is handed to (PHASE itself: its next launch)
        {
            if (active && st.mode == kAStep && st.rk_kind < 0) {
                const ImageConsts& c = J->c;
                const double r_bl = SC::radius(c, S.x);
                const int want_phase = phase_of(c, 0, r_bl);
                if (want_phase != PHASE) {
                    dest = want_phase;
                } else if (W.budget > 0 && lane_jobs >= W.budget) {
                    dest = PHASE;
                } else if (st.n >= c.max_steps) {
                    // pass-A loop top (pass_b.hpp:793-838)
                    st.mode = kEndA;
                } else {
                    if (!st.entered) {
                        if (r_bl <= c.outer_radius) {
                            st.entered = 1;
                            st.inside = 0;
                        }
                    } else if (r_bl - c.inner_radius <= 0.0) {
                        st.reason = kReachedInner;
                        st.mode = kEndA;
                    } else if (st.inside > 0 && r_bl >= c.outer_radius) {
                        st.reason = kEscaped;
                        st.mode = kEndA;
                    }
                    if (st.mode == kAStep) {
                        st.old_r = r_bl;
                        double mn = c.min_step_abs;
                        if (abs_val(st.h_current) < mn) mn = abs_val(st.h_current);
                        issue_step(st, c, st.h_current, mn, c.max_step);
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
#pragma unroll
                    for (int f = 0; f < NF; ++f) RT::zero(stokes[f]);
                    memcpy(W.pool[my_id].stokes, &stokes[0], sizeof(stokes));
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
                const double r_bl = SC::radius(c, S.x);
                const int want_phase = phase_of(c, 1, r_bl);
                if (want_phase != PHASE) {
                    dest = want_phase;
                } else if (W.budget > 0 && lane_jobs >= W.budget) {
                    dest = PHASE;
                } else {
                    // pass-B loop top (pass_b.hpp:966-981)
                    double h = st.h_current;
                    st.start_r = r_bl;
                    if (st.start_r <= c.outer_radius && st.cap > 0.0) h = min_val(h, st.cap);
                    st.hB = h;
                    issue_step(st, c, h, c.min_step_abs, c.max_step);
                }
            }
        }
        const bool park = dest >= 0;
        if (park) {
            RayRecord& rec = W.pool[my_id];
            rec.S = S;
            memcpy(rec.st, &st, kLaneStateBytes<PHASE>);
        }
        // A lane past its budget keeps claiming and parks each claimed ray at
        // once, so every input ends the launch finished or in a queue.
#pragma unroll
        for (int d = 0; d < kPhases; ++d) queue_push(W.out_ids[d], W.out_count[d], dest == d, my_id);
        if (park) st.mode = kIdle;

        // ------------------------------------------------------------ RK job
        const bool run = !park && (st.mode == kAStep || st.mode == kBStep || st.mode == kBCamCross);
        Ray next, mid;
        double err = 0.0;
        if (run) {
            bool sure = false;
            if constexpr (SC::kCksRhs) {
                if (st.rk_kind == kRkSD) {
                    double km = 0.0, w = 0.0, z = 0.0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        km = max_val(km, abs_val(S.k.v[i]));
                        w = max_val(w, max_val(abs_val(S.e1.v[i]), abs_val(S.e2.v[i])));
                        z += S.k.v[i] + (S.e1.v[i] + S.e2.v[i]);
                    }
                    if (!(z - z == 0.0)) w = kLarge;  // a NaN or an infinity among them
                    const double tol = max_val(J->c.tolerance, kTolFloor);
                    sure = certain_step(J->c.mass, st.mode == kAStep ? st.old_r : st.start_r, km, max_val(km, w), st.h_try,
                                        (abs_val(st.h_try) == st.ctl_max ? 0.25 : 1.0 / 64.0) * tol);
                }
            }
            rk_job<P, SC>(st.rk_kind, J->c, S, st.h_try, sure, next, mid, err);
            if (++lane_jobs > (1LL << 30)) {
                st.reason = kInvalidState;
                st.mode = kDone;
                st.in_b = 0;
                atomicExch(W.status, 2);
            }
        }

        // The warps of a block finish their RK jobs together and run the
        // control and radiation code together: one code region at a time
        // per SM keeps it in the instruction cache.
        __syncthreads();

        // ----------------------------------------------- control after the job
        if (run && st.mode == kAStep) {
            const ImageConsts& c = J->c;
            bool accepted = true;
            if (st.rk_kind != kRkRK4) {
                const double tol = max_val(c.tolerance, kTolFloor);
                if (err <= tol) {
                    st.h_current = accepted_next_h(st.h_try, err, tol, st.ctl_min, st.ctl_max, st.req_h);
                } else {
                    accepted = false;
                    if (rejected_attempt(st, err, tol)) {
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
                const double next_r = SC::radius(c, next.x);
                const double old_r = st.old_r;
                if (!st.entered && next_r <= c.outer_radius) {
                    st.entered = 1;
                    st.inside = 0;
                } else if (!st.entered && next_r >= old_r) {
                    S = next;
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
                        atomicExch(W.status, 3);  // surfaces lie inside the near phase
                        st.reason = kInvalidState;
                        st.mode = kDone;
                    } else {
                        S = next;
                        st.pa_steps += 1;
                        if (st.entered) st.inside += 1;
                        st.n += 1;
                    }
                }
            }
        } else if (run && (st.mode == kBStep || st.mode == kBCamCross)) {
            const ImageConsts& c = J->c;
            const bool cam = st.mode == kBCamCross;
            bool proceed = true;
            double h = st.hB;
            if (st.rk_kind != kRkRK4) {
                const double tol = max_val(c.tolerance, kTolFloor);
                if (err <= tol) {
                    h = abs_val(st.h_try);
                    if (!cam) st.h_current = abs_val(accepted_next_h(st.h_try, err, tol, st.ctl_min, st.ctl_max, st.req_h));
                } else {
                    proceed = false;
                    if (rejected_attempt(st, err, tol)) {
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
            if (proceed) {
                Ray sample = st.rk_kind == kRkSD ? mid : next;
                int crosses = 1;
                if (!cam) {
                    // camera surface (pass_b.hpp:999-1028)
                    const double s0 = st.start_r - c.cam_radius;
                    const double s1 = SC::radius(c, next.x) - c.cam_radius;
                    crosses = (s0 == 0.0 || s1 == 0.0) ? 1 : ((s0 < 0.0 && s1 > 0.0) || (s0 > 0.0 && s1 < 0.0));
                    if (crosses) {
                        const double denom = s0 - s1;
                        const double frac = abs_val(denom) <= kTiny ? 1.0 : min_val(1.0, max_val(0.0, s0 / denom));
                        const double h_cross = h * frac;
                        if (abs_val(h_cross) <= 1e-14) {
                            h = 0.0;
                            next = S;
                            sample = S;
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
                if (proceed) {
                    // The sample lies outside the radiating sphere: every
                    // coefficient is zero, the transfer step leaves the Stokes
                    // vector unchanged and the step cap resolves to max_step
                    // (pass_b.hpp:1414-1496).
                    const double sample_r = SC::radius(c, sample.x);
                    const double next_r = SC::radius(c, next.x);
                    if ((c.max_radiation_step > 0.0 &&
                         (st.start_r <= c.outer_radius || sample_r <= c.outer_radius || next_r <= c.outer_radius)) ||
                        (sample_r - c.inner_radius > 0.0 && sample_r < c.outer_radius))
                        atomicExch(W.status, 3);
                    st.cap = c.max_step;
                    S = next;
                    st.steps += 1;
                    if (crosses) st.reached = 1;
                    st.mode = kBStep;
                    st.rk_kind = -1;
                }
            }
        }

        // ------------------------------------------------------------ finish
        if (!park && st.mode == kDone) {
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
            double obs[NF][4];
            Stokes4<double> sd[NF];
            // only the radiating phase carries the Stokes vector: it is in the record
            if (st.in_b) memcpy(&stokes[0], W.pool[my_id].stokes, sizeof(stokes));
#pragma unroll
            for (int f = 0; f < NF; ++f)
                sd[f] = st.in_b ? RT::result(stokes[f], c, f) : Stokes4<double>{0.0, 0.0, 0.0, 0.0};
            finish_ray_scene<SC, NF>(c, cam, S, st.in_b, sd, o, obs);
            store_stokes_n<NF>(J->out, st.pixel, J->npix, c.nfreq, obs);
            store_diagnostics(J->out, st.pixel, o);
            if constexpr (SC::kSlowLight) {
                if (!st.in_b) J->out.basis_identity_error[st.pixel] = 0.0;
            }
            if (W.job_done) atomicAdd(&W.job_done[st.job], 1u);
            st.mode = kIdle;
        }
    }
}

}  // namespace kp
