// Host build of the mixed policy's thermal-synchrotron fits
// (kpolaris_b200/csrc/kp_radiation_mixed.cuh), for tests/test_mixed_coefficients.py.
// Reads lines "fit nu ne thetae b theta sin cos" on stdin and prints the
// unscaled invariant coefficients jI jQ jV aI aQ aV rQ rV (magnetic basis).
#include <cmath>
#include <cstdio>
#include <cstring>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#include "kp_radiation_mixed.cuh"

int main() {
    int fit;
    double nu, ne, te, b, th, s, c;
    while (std::scanf("%d %lf %lf %lf %lf %lf %lf %lf", &fit, &nu, &ne, &te, &b, &th, &s, &c) == 8) {
        kp::ImageConsts k;
        std::memset(&k, 0, sizeof(k));
        k.fit = fit;
        k.min_sin_theta = 1e-4;
        k.max_pol_frac = 0.99;
        k.emission_scale = k.absorption_scale = k.faraday_scale = 1.0;
        kp::RiafSampleM p;
        std::memset(&p, 0, sizeof(p));
        p.emitting = 1;
        p.ne = ne;
        p.thetae = te;
        p.b = b;
        p.nu_fluid = 1.0;
        p.sin_theta = s;
        p.cos_theta = c;
        p.has_chi = 1;
        p.cos2chi = 1.0;
        p.sin2chi = 0.0;
        kp::riaf_sample_thermal_m(k, p);
        // scale the emission as the images do and undo it
        const double j0 = ne * 2.3e-19 * 2.8e6 * b / 3e10 / (nu * nu);
        const int e = int(std::floor(std::log2(1.0 / std::max(j0, 1e-300))));
        const double escale = std::ldexp(1.0, std::max(-120, std::min(120, e)));
        const kp::CoeffsM o = kp::riaf_coefficients_m(k, p, nu * 1e-9, escale);
        const double inv = 1.0 / escale;
        std::printf("%.17e %.17e %.17e %.17e %.17e %.17e %.17e %.17e\n", o.jI * inv, o.jQ * inv, o.jV * inv, o.aI, o.aQ,
                    o.aV, o.rQ, o.rV);
    }
    return 0;
}
