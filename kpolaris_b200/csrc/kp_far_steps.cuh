// kp_far_steps.cuh -- what the step control will do, known without asking it:
// how many of its steps the mixed policy's far phase bridges at once
// (quad_macro_step in kp_quad.cuh), and which steps need no error estimate.
#pragma once

#include "kp_common.cuh"

namespace kp {

// One row of the extrapolation that bridges a run, for one component: the
// modified midpoint rule with n_j = 2 j + 2 substeps gave v; c0, c1, c2 hold
// the columns of the row before and take this row's.  Neville's scheme in the
// step squared: column k from column k - 1 and the row before, with q = 1 /
// ((n_j / n_(j-k))^2 - 1).  Returns the row's last column.
KP_HD double macro_row(int j, double v, double& c0, double& c1, double& c2) {
    const double q[3] = {j == 1 ? 1.0 / 3.0 : (j == 2 ? 0.8 : 9.0 / 7.0), j == 2 ? 0.125 : 1.0 / 3.0, 1.0 / 15.0};
    double* const c[3] = {&c0, &c1, &c2};
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 3; ++k) {
        const double w = v + (v - *c[k]) * q[k];
        if (k <= j) *c[k] = v;
        if (k < j) v = w;
    }
    return v;
}

// A run of accepted steps: their number, the affine distance they cover and
// the size of the step after them (all positive; count 0: none).
struct MacroRun {
    int count;
    double length, next_h;
};

// The run of steps the step control would take from a ray at radius r whose
// next step has size h (at most `cap`, the step's own size for fixed steps),
// where each of them is sure to be accepted:
// * The step-doubling error of a step of size h at radius r is below
//   (16 + r / 4) M h^5 / r^6 beyond the sphere (k, e1 and e2 in the first
//   term; the position, whose components near zero are measured absolutely,
//   in the second) plus rounding.  The two factors are fitted: over the rays of
//   tests/native/far_steps.cpp the error is at most 0.4 of it.  At tol / 64 or less the control doubles a step below the cap,
//   at tol / 4 or less a step at the cap stays there, so the run's sizes are
//   known: h, 2h, 4h, ... cap, cap, ...  (At the cap a sixteenth is asked
//   for: the run has none of its steps' truncation errors, whose sum grows as
//   the fourth power of 1 / r and at a quarter moved five pixels in 400,000
//   across a substep decision, against one without runs; the far phase of
//   8 x 256^2 pays 26 -> 45 ms for it.)
// * No step of the run starts in the near phase, reaches the camera's radius
//   or, in pass A, the turning point.  xk is x.k (spatial), v the spatial
//   speed |dx/dlambda|, dir the sign of the step; over a run the speed and the
//   direction change by a few M / r, which the margins cover.
// * The run covers at most a fifth of the radius, where quad_macro_step is off
//   by at most 3e-12 on the same rays (against eight bridges of an eighth).
KP_HD MacroRun macro_run(const ImageConsts& c, double r, double xk, double v, double h, double cap, double dir,
                         bool pass_a, int left) {
    MacroRun none = {0, 0.0, 0.0};
    const double rmin = 0.8 * r;
    const double r2 = rmin * rmin, c2 = cap * cap;
    const double bound = (16.0 + 0.25 * rmin) * c.mass * c2 * c2 * cap / (r2 * r2 * r2) + 1e-14;
    const double tol = max_val(c.tolerance, kTolFloor) * (h < cap ? 1.0 / 64.0 : 1.0 / 16.0);
    if (!(bound <= (c.adaptive ? tol : 1e-11))) return none;
    double reach = 0.2 * r;
    const double along = dir * xk;  // > 0: outward
    if (pass_a) {
        if (along >= 0.0) return none;
        reach = min_val(reach, 0.8 * (-along / v) - 16.0 * c.mass);
    } else {
        reach = min_val(reach, abs_val(r - c.cam_radius) - 1.1 * v * cap);
    }
    if (!(along > 0.1 * r * v)) reach = min_val(reach, r - c.far_radius - 0.1 * v * cap);
    const double span = reach / (v * (1.0 + 4.0 * c.mass / rmin));
    if (!(span >= h) || !(span < 1e300) || left < 1) return none;
    MacroRun run = {0, 0.0, h};
    while (run.next_h < cap && run.count < left && run.length + run.next_h <= span) {
        run.length += run.next_h;
        run.next_h = min_val(cap, 2.0 * run.next_h);
        ++run.count;
    }
    if (run.next_h >= cap) {
        const double m = (span - run.length) / cap;
        const int more = m < double(left - run.count) ? int(m) : left - run.count;
        run.length += cap * double(more);
        run.count += more;
    }
    return run;
}

// Whether the step-doubling error of a step of size h at radius r is sure to
// be at most `lim`, from a bound on the Kerr-Schild transport: km the largest
// |k^mu| (k near the null cone), w the largest component of k, e1 and e2.  With
// `lim` a quarter of the tolerance for a step at the cap and 1/64 of it
// otherwise the step control accepts the step and the next one's size is known
// (the cap, or twice the size): the attempt needs no full-step chain.  The
// bound's factors are fitted, with a margin: the error found by
// tests/native/far_steps.cpp is at most 0.1 of it along camera rays past the
// hole, down to r = 2 M, and 0.4 for random vectors up to half off the cone.
// The last term covers rounding.
KP_HD bool certain_step(double mass, double r, double km, double w, double h, double lim) {
    const double ah = abs_val(h), rl = r - 3.5 * ah * km;
    if (!(rl > 2.0 * mass) || !(w < 1e4)) return false;
    const double hk = ah * km, hk2 = hk * hk, r2 = rl * rl;
    return (24.0 + 0.375 * rl) * mass * (hk2 * hk2 * ah * w) <= (lim - 1e-13 * max_val(1.0, w)) * (r2 * r2 * r2);
}

}  // namespace kp
