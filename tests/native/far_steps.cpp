// Host check of the far field's bridged runs of steps (macro_run in
// kpolaris_b200/csrc/kp_far_steps.cuh) against the step control itself, in
// FP64 with the reference's transport.  Rays of a pinhole camera at several
// radii, seeded.  Prints
//   the largest step-doubling error of a run's steps over the bound macro_run
//   takes for it,
//   the number of runs, and of runs that the step control does not take
//   (another step size, a step from or into the near phase, past the camera
//   or, in pass A, outward),
//   the largest distance (over max(1, |.|)) between the extrapolated midpoint
//   rule over a run and the steps themselves,
//   how many steps certain_step promised, and the largest error of one of
//   them over the error it was promised to stay under,
//   the largest distance between a run bridged at once and in eight parts,
//   and the largest such error of random vectors.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#include "kp_camera.cuh"
#include "kp_far_steps.cuh"
#include "kp_geometry.cuh"

using namespace kp;

static Ray axpy(const Ray& y, double a, const Ray& x) {
    Ray o;
    const double* p = reinterpret_cast<const double*>(&y);
    const double* q = reinterpret_cast<const double*>(&x);
    double* r = reinterpret_cast<double*>(&o);
    for (int i = 0; i < 16; ++i) r[i] = p[i] + a * q[i];
    return o;
}

static Ray rk4(double M, double a, const Ray& s, double h) {
    const Ray k1 = ks_rhs(M, a, s), k2 = ks_rhs(M, a, axpy(s, 0.5 * h, k1));
    const Ray k3 = ks_rhs(M, a, axpy(s, 0.5 * h, k2)), k4 = ks_rhs(M, a, axpy(s, h, k3));
    return axpy(axpy(axpy(axpy(s, h / 6.0, k1), h / 3.0, k2), h / 3.0, k3), h / 6.0, k4);
}

static double distance(const Ray& a, const Ray& b) {
    const double* p = reinterpret_cast<const double*>(&a);
    const double* q = reinterpret_cast<const double*>(&b);
    double d = 0.0;
    for (int i = 0; i < 16; ++i)
        d = std::fmax(d, std::fabs(p[i] - q[i]) / std::fmax(1.0, std::fmax(std::fabs(p[i]), std::fabs(q[i]))));
    return d;
}

// Gragg's midpoint rule with 2, 4, 6, 8 substeps, extrapolated by the
// library's macro_row.
static Ray midpoint(double M, double a, const Ray& s, double H) {
    const Ray f0 = ks_rhs(M, a, s);
    Ray t, C[3];
    double* const v = reinterpret_cast<double*>(&t);
    double* const c[3] = {reinterpret_cast<double*>(&C[0]), reinterpret_cast<double*>(&C[1]),
                          reinterpret_cast<double*>(&C[2])};
    for (int j = 0; j < 4; ++j) {
        const int n = 2 * j + 2;
        const double h = H / n;
        Ray z0 = s, z1 = axpy(s, h, f0);
        for (int i = 1; i < n; ++i) {
            const Ray z2 = axpy(z0, 2.0 * h, ks_rhs(M, a, z1));
            z0 = z1;
            z1 = z2;
        }
        t = axpy(axpy(z1, h, ks_rhs(M, a, z1)), 1.0, z0);
        for (int i = 0; i < 16; ++i) v[i] = macro_row(j, 0.5 * v[i], c[0][i], c[1][i], c[2][i]);
    }
    return t;
}

int main() {
    std::mt19937_64 rng(20260101);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    double worst_const = 0.0, worst_dist = 0.0, worst_rule = 0.0;
    int runs = 0, wrong = 0;
    for (int ray = 0; ray < 600; ++ray) {
        ImageConsts c;
        std::memset(&c, 0, sizeof(c));
        c.mass = 1.0;
        c.spin = 0.99 * u(rng);
        c.adaptive = ray % 4 != 3;
        c.max_step = ray % 4 == 1 ? 0.7 : (ray % 4 == 2 ? 5.0 : 2.0);
        c.step = ray % 4 == 3 ? 1.0 : 0.025;
        c.tolerance = ray % 4 == 2 ? 1e-6 : 1e-8;
        c.outer_radius = 50.0 + 65.0 * u(rng);
        if (ray >= 400) {  // small spheres, short steps, near cameras
            c.max_step = 0.025 + 0.475 * u(rng);
            c.outer_radius = 4.0 + 46.0 * u(rng);
        }
        c.far_radius = c.outer_radius + 2.0 * std::fmax(c.max_step, c.step);
        c.cam_radius = ray < 400 ? 200.0 + 1800.0 * u(rng) : 60.0 + 300.0 * u(rng);
        // a ray through the camera's radius at some impact parameter, its
        // wavevector null in the Kerr-Schild metric to first order
        const double r = c.cam_radius, b = (ray < 400 ? 400.0 : 0.8 * c.cam_radius) * (u(rng) - 0.5), th = std::acos(2.0 * u(rng) - 1.0), ph = 6.28 * u(rng);
        const double n[3] = {std::sin(th) * std::cos(ph), std::sin(th) * std::sin(ph), std::cos(th)};
        double e[3] = {n[1], -n[0], 0.0};
        const double en = std::sqrt(e[0] * e[0] + e[1] * e[1]) + 1e-300;
        Ray s;
        const double out = std::sqrt(r * r - b * b);
        for (int i = 0; i < 3; ++i) {
            s.x.v[i + 1] = out * n[i] + b * e[i] / en;
            s.k.v[i + 1] = n[i];
            s.e1.v[i + 1] = e[i] / en;
        }
        s.x.v[0] = 0.0;
        s.k.v[0] = 1.0 + 2.0 / r;
        s.e1.v[0] = s.e2.v[0] = 0.0;
        for (int i = 0; i < 3; ++i) {
            const int p = (i + 1) % 3, q = (i + 2) % 3;
            s.e2.v[i + 1] = n[p] * s.e1.v[q + 1] - n[q] * s.e1.v[p + 1];
        }
        for (int pass = 0; pass < 2; ++pass) {
            // pass A: backward from the camera; pass B: forward from where A stopped
            const double dir = pass == 0 ? -1.0 : 1.0;
            const double cap = c.adaptive ? c.max_step : c.step;
            double h = c.step;
            if (pass == 1) h = cap;
            const double rr = ks_radius(c.spin, s.x);
            if (pass == 1 && !(rr > c.far_radius)) break;
            for (int guard = 0; guard < 60; ++guard) {
                const double r0 = ks_radius(c.spin, s.x);
                if (!(r0 > c.far_radius)) break;
                double xk = 0.0, kk = 0.0;
                for (int i = 1; i < 4; ++i) {
                    xk += s.x.v[i] * s.k.v[i];
                    kk += s.k.v[i] * s.k.v[i];
                }
                const MacroRun run = macro_run(c, r0, xk, std::sqrt(kk), h, cap, dir, pass == 0, 100000);
                if (run.count < 3) break;
                ++runs;
                const Ray far = midpoint(c.mass, c.spin, s, dir * run.length);
                Ray parts = s;
                for (int k = 0; k < 8; ++k) parts = midpoint(c.mass, c.spin, parts, 0.125 * dir * run.length);
                worst_rule = std::fmax(worst_rule, distance(far, parts));
                double len = 0.0, hh = h, old = r0;
                bool ok = true;
                for (int k = 0; k < run.count; ++k) {
                    const double rk = ks_radius(c.spin, s.x);
                    ok = ok && rk > c.far_radius;
                    const Ray full = rk4(c.mass, c.spin, s, dir * hh);
                    const Ray half = rk4(c.mass, c.spin, s, 0.5 * dir * hh);
                    const Ray two = rk4(c.mass, c.spin, half, 0.5 * dir * hh);
                    const double err = distance(full, two);
                    worst_const = std::fmax(
                        worst_const, err / ((16.0 + 0.25 * rk) * std::pow(hh, 5) / std::pow(rk, 6) + 1e-14));
                    s = c.adaptive ? two : full;
                    len += hh;
                    if (c.adaptive) {
                        ok = ok && err <= c.tolerance;
                        double f = err > 0.0 ? 0.9 * std::pow(c.tolerance / err, 0.2) : 2.0;
                        f = std::fmin(2.0, std::fmax(0.2, f));
                        hh = std::fmin(c.max_step, hh * f);
                    }
                    const double r1 = ks_radius(c.spin, s.x);
                    if (pass == 0) ok = ok && r1 < old;
                    if (pass == 1) ok = ok && (old - c.cam_radius) * (r1 - c.cam_radius) > 0.0;
                    old = r1;
                }
                ok = ok && old > c.far_radius && std::fabs(len - run.length) <= 1e-9 * len &&
                     std::fabs(hh - run.next_h) <= 1e-12 * hh;
                if (!ok) ++wrong;
                worst_dist = std::fmax(worst_dist, distance(far, s));
                h = run.next_h;
            }
        }
    }
    // certain_step: the error of a step against the bound it is promised by,
    // along camera rays past the hole, backward and forward
    double worst_certain = 0.0;
    long certain = 0;
    for (int ray = 0; ray < 150; ++ray) {
        ImageConsts c;
        std::memset(&c, 0, sizeof(c));
        c.mass = 1.0;
        c.spin = 0.998 * u(rng);
        c.nx = c.ny = 64;
        c.cam_radius = u(rng) < 0.5 ? 1000.0 : 50.0 + 1000.0 * u(rng);
        const double inc = 0.1 + 2.9 * u(rng);
        c.sin_inc = std::sin(inc);
        c.cos_inc = std::cos(inc);
        c.fov = c.fov_y = (u(rng) < 0.6 ? 24.0 : 160.0) / c.cam_radius;
        const CameraFrame f = camera_frame(c);
        Ray s = camera_ray(c, f, int(4096 * u(rng)));
        const double rh = 1.0 + std::sqrt(1.0 - c.spin * c.spin);
        double dir = -1.0;
        for (int n = 0; n < 6000; ++n) {
            const double r = ks_radius(c.spin, s.x);
            if (dir < 0.0 ? (r < rh * 1.05 || (r > 1200.0 && n > 100)) : (r > 1100.0 || r < rh * 1.01)) {
                if (dir > 0.0) break;
                dir = 1.0;
            }
            double km = 0.0, w = 0.0;
            for (int i = 0; i < 4; ++i) {
                km = std::fmax(km, std::fabs(s.k.v[i]));
                w = std::fmax(w, std::fmax(std::fabs(s.e1.v[i]), std::fabs(s.e2.v[i])));
            }
            w = std::fmax(km, w);
            for (const double h : {8.0, 4.0, 2.0, 0.7, 0.2, 0.03}) {
                for (const double lim : {2.5e-9, 2.5e-11, 1e-8 / 64.0, 1e-6 / 64.0}) {
                    if (!certain_step(c.mass, r, km, w, h, lim)) continue;
                    ++certain;
                    const Ray half = rk4(c.mass, c.spin, s, 0.5 * dir * h);
                    const double err = distance(rk4(c.mass, c.spin, s, dir * h), rk4(c.mass, c.spin, half, 0.5 * dir * h));
                    worst_certain = std::fmax(worst_certain, err / lim);
                }
            }
            s = rk4(c.mass, c.spin, s, dir * (r > 130.0 ? 4.0 : std::fmin(2.0, 0.05 * r * (0.3 + u(rng)))));
            if (!(std::fabs(s.x.v[1]) < 1e9)) break;
        }
    }
    // and of random vectors: k on the null cone with its spatial part up to half
    // as long again, of any size and direction, e1 and e2 of any
    double worst_random = 0.0;
    for (int i = 0; i < 30000; ++i) {
        const double spin = 0.998 * u(rng), r = 2.2 * std::pow(700.0, u(rng)), size = std::pow(3.0, 2.0 * u(rng) - 1.0);
        Ray s;
        double n[3], d[3];
        for (double* v : {n, d}) {
            const double th = std::acos(2.0 * u(rng) - 1.0), ph = 6.283185307 * u(rng);
            v[0] = std::sin(th) * std::cos(ph);
            v[1] = std::sin(th) * std::sin(ph);
            v[2] = std::cos(th);
        }
        s.x.v[0] = 0.0;
        for (int k = 0; k < 3; ++k) s.x.v[k + 1] = std::sqrt(r * r + spin * spin) * n[k];
        const KSMetricPoint g = ks_point(1.0, spin, s.x);
        const double ld = g.l[1] * d[0] + g.l[2] * d[1] + g.l[3] * d[2];
        const double qa = g.amp - 1.0, qb = 2.0 * g.amp * ld, qc = 1.0 + g.amp * ld * ld, disc = qb * qb - 4.0 * qa * qc;
        if (!(disc > 0.0) || !(qa < 0.0)) continue;
        s.k.v[0] = size * std::fmax((-qb - std::sqrt(disc)) / (2.0 * qa), (-qb + std::sqrt(disc)) / (2.0 * qa));
        const double off = size * (0.8 + 0.7 * u(rng));
        double km = std::fabs(s.k.v[0]), w = 0.0;
        for (int k = 0; k < 3; ++k) km = std::fmax(km, std::fabs(s.k.v[k + 1] = off * d[k]));
        for (int k = 0; k < 4; ++k) {
            s.e1.v[k] = 2.0 * u(rng) - 1.0;
            s.e2.v[k] = 2.0 * u(rng) - 1.0;
            w = std::fmax(w, std::fmax(std::fabs(s.e1.v[k]), std::fabs(s.e2.v[k])));
        }
        w = std::fmax(km, w);
        const double rb = ks_radius(spin, s.x);
        for (const double h : {16.0, 8.0, 4.0, 2.0, 0.7, 0.2, 0.03}) {
            for (const double lim : {2.5e-9, 2.5e-11, 1e-8 / 64.0, 1e-6 / 64.0, 2.5e-7}) {
                if (!certain_step(1.0, rb, km, w, h, lim)) continue;
                const Ray half = rk4(1.0, spin, s, 0.5 * h);
                worst_random = std::fmax(worst_random, distance(rk4(1.0, spin, s, h), rk4(1.0, spin, half, 0.5 * h)) / lim);
            }
        }
    }
    std::printf("%.3f %d %d %.3e %ld %.3f %.3e %.3f\n", worst_const, runs, wrong, worst_dist, certain, worst_certain,
                worst_rule, worst_random);
    return 0;
}
