// Host check of the mixed policy's factored transport RHS
// (kpolaris_b200/csrc/kp_geometry_mixed.cuh) against the reference-order FP64
// RHS (kp_geometry.cuh) on seeded states around a Kerr black hole, and of the
// FMKS one (fmks_rhs_factored against fmks_rhs in kp_fmks.cuh).  Prints the
// largest normwise relative deviation of each.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#include "kp_fmks.cuh"

// The largest deviation of dk, de1 and de2, each against its own largest component.
static double deviation(const kp::Ray& ref, const kp::Ray& got) {
    const kp::D4* R[3] = {&ref.k, &ref.e1, &ref.e2};
    const kp::D4* A[3] = {&got.k, &got.e1, &got.e2};
    double worst = 0.0;
    for (int w = 0; w < 3; ++w) {
        double scale = 0.0, d = 0.0;
        for (int k = 0; k < 4; ++k) {
            scale = std::fmax(scale, std::fabs(R[w]->v[k]));
            d = std::fmax(d, std::fabs(A[w]->v[k] - R[w]->v[k]));
        }
        if (scale > 0.0) worst = std::fmax(worst, d / scale);
    }
    return worst;
}

int main() {
    std::mt19937_64 rng(12345);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    double worst_ks = 0.0, worst_fmks = 0.0;
    for (int i = 0; i < 20000; ++i) {
        const double spin = 0.99 * std::fabs(u(rng));
        const double rad = 1.5 + std::pow(10.0, 3.0 * std::fabs(u(rng)));
        double dir[3] = {u(rng), u(rng), u(rng)};
        const double n = std::sqrt(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]) + 1e-12;
        kp::Ray s;
        s.x.v[0] = 0.0;
        for (int k = 0; k < 3; ++k) s.x.v[k + 1] = rad * dir[k] / n;
        for (int k = 0; k < 4; ++k) {
            s.k.v[k] = u(rng);
            s.e1.v[k] = u(rng);
            s.e2.v[k] = u(rng);
        }
        s.k.v[0] = 1.0 + std::fabs(u(rng));
        worst_ks = std::fmax(worst_ks, deviation(kp::ks_rhs(1.0, spin, s), kp::ks_rhs_factored(1.0, spin, s)));
        kp::FmksParams m;
        std::memset(&m, 0, sizeof(m));
        m.mass = 1.0;
        m.spin = spin;
        m.startx1 = std::log(1.2);
        m.hslope = 0.3;
        m.mks_smooth = 0.5;
        m.poly_alpha = 14.0;
        m.poly_xt = 0.82;
        m.poly_norm = 0.5 * 3.141592653589793 / (1.0 + 1.0 / 15.0 / std::pow(0.82, 14.0));
        s.x.v[1] = std::log(rad);
        s.x.v[2] = 0.5 + 0.49 * u(rng);
        s.x.v[3] = 3.0 * u(rng);
        worst_fmks = std::fmax(worst_fmks, deviation(kp::fmks_rhs(m, s), kp::fmks_rhs_factored(m, s)));
    }
    std::printf("%.3e %.3e\n", worst_ks, worst_fmks);
    return 0;
}
