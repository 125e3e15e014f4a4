// kp_lanes.cu -- the phase kernels with one ray per lane (lane_body in
// kp_persistent.cuh), for images and launches with rays enough to fill the
// device.  Compiled once per policy and scene (KP_LANES_POLICY,
// KP_LANES_SCENE) with the floating-point flags of that policy's quad kernels,
// but with exp, log and pow inlined (near-B of 8 x 256^2 FP64, four
// frequencies: 491 ms, as calls 513 ms).  Near-A and near-B run as one CTA of
// 256 threads per SM, whose warps step through the same code region (near-A of
// 8 x 256^2 FP64: 85 ms, as two CTAs of 128 95 ms).
#include <cuda_runtime.h>

#include "kp_launch.h"
#include "kp_persistent.cuh"

namespace kp {

template<class P, int NF, class SC>
__global__ void __launch_bounds__(kFarThreads, kFarBlocks) lanes_far(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) > quad_rays) lane_body<P, NF, kPhaseFar, SC>(W);
}

template<class P, class SC>
__global__ void __launch_bounds__(kLaneNearThreads, 1) lanes_near_a(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) > quad_rays) lane_body<P, kMaxFreq, kPhaseNearA, SC>(W);
}

template<class P, int NF, class SC>
__global__ void __launch_bounds__(kLaneNearThreads, 1) lanes_near_b(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) > quad_rays) lane_body<P, NF, kPhaseNearB, SC>(W);
}

template<class P, class SC>
cudaError_t launch_lanes(int phase, const WaveDesc& W, int nf_max, long long lanes, long long quad_rays,
                         cudaStream_t stream) {
    // the mixed policy has far kernels of its own, and one form of its
    // arithmetic whatever shares the launch
    constexpr int kOne = P::kMixed ? kMaxFreq : 1;
    const void* fn = reinterpret_cast<const void*>(lanes_near_a<P, SC>);
    if (phase == kPhaseFar) {
        if constexpr (P::kMixed) return cudaErrorInvalidValue;
        else fn = nf_max == 1 ? reinterpret_cast<const void*>(lanes_far<P, 1, SC>)
                              : reinterpret_cast<const void*>(lanes_far<P, kMaxFreq, SC>);
    } else if (phase == kPhaseNearB) {
        fn = nf_max == 1 ? reinterpret_cast<const void*>(lanes_near_b<P, kOne, SC>)
                         : reinterpret_cast<const void*>(lanes_near_b<P, kMaxFreq, SC>);
    }
    const int threads = phase == kPhaseFar ? kFarThreads : kLaneNearThreads;
    void* args[] = {const_cast<WaveDesc*>(&W), &quad_rays};
    return cudaLaunchKernel(fn, dim3(unsigned((lanes + threads - 1) / threads)), dim3(threads), args, 0, stream);
}

template cudaError_t launch_lanes<KP_LANES_POLICY, KP_LANES_SCENE>(int, const WaveDesc&, int, long long, long long,
                                                                   cudaStream_t);

#ifdef KP_LANES_IMAGE
// Pass B (pass_b.hpp:940-1114, :1312-1501) of an image with fixed steps, as a
// loop over the steps: with nothing to retry and no step control the ray needs
// none of lane_body's state machine (256^2: 114 -> 87 ms).
template<int NF>
__device__ __forceinline__ void trace_pass_b_fixed(const ImageConsts& c, Ray& state, Stokes4<double> (&stokes)[NF],
                                                   int& steps, int& reason) {
    using RT = RadTraits<PolicyFP64, SceneRiaf>;
    const int nf = c.nfreq < NF ? c.nfreq : NF;
#pragma unroll
    for (int f = 0; f < NF; ++f) RT::zero(stokes[f]);
    steps = 0;
    int reached = 0;
    double h_current = c.step;
    double cap = c.max_radiation_step > 0.0 ? c.max_radiation_step : c.max_step;
    double start_r = ks_radius(c.spin, state.x);
#pragma unroll 1
    while (!reached && steps < c.max_steps) {
        double h = h_current;
        if (start_r <= c.outer_radius && cap > 0.0) h = min_val(h, cap);
        Ray next = rk4_step(c.mass, c.spin, state, h);
        double next_r = ks_radius(c.spin, next.x);
        // camera surface (pass_b.hpp:999-1028)
        const double s0 = start_r - c.cam_radius, s1 = next_r - c.cam_radius;
        const int crosses = (s0 == 0.0 || s1 == 0.0) ? 1 : ((s0 < 0.0 && s1 > 0.0) || (s0 > 0.0 && s1 < 0.0));
        if (crosses) {
            const double denom = s0 - s1;
            const double frac = abs_val(denom) <= kTiny ? 1.0 : min_val(1.0, max_val(0.0, s0 / denom));
            const double h_cross = h * frac;
            if (abs_val(h_cross) <= 1e-14) {
                h = 0.0;
                next = state;
                next_r = start_r;
            } else if (frac < 0.999999999999) {
                h = h_cross;
                next = rk4_step(c.mass, c.spin, state, h);
                next_r = ks_radius(c.spin, next.x);
            }
        }
        // radiation at the step's end (pass_b.hpp:1414-1496)
        const double local_max_rs =
            c.max_radiation_step > 0.0 && (start_r <= c.outer_radius || next_r <= c.outer_radius) ? c.max_radiation_step : 0.0;
        const bool radiating = next_r - c.inner_radius > 0.0 && next_r < c.outer_radius;
        int required = 1, pred = 1;
        Coeffs<double> co[NF];
        auto count = [&](const RadDepths& depth) {
            required = max(required, substeps_for(depth, h, local_max_rs, c));
            pred = max(pred, substeps_for(depth, h_current, local_max_rs, c));
        };
        if (!radiating) {
            count(RadDepths{0.0, 0.0, 0.0});
        } else {
            const RiafSample ps = riaf_sample(c, next);
#pragma unroll 1
            for (int f = 0; f < nf; ++f) {
                co[f] = RT::coeffs(c, ps, f);
                if (!c.faraday_rotation) co[f].rV = 0.0;
                if (c.nctl == 0) count(RT::depths(co[f], c.dlambda_scale[f]));
            }
#pragma unroll 1
            for (int g = 0; g < c.nctl; ++g) {
                Coeffs<double> cg = RT::coeffs_ctl(c, ps, g);
                if (!c.faraday_rotation) cg.rV = 0.0;
                count(RT::depths(cg, c.ctl_dlambda_scale[g]));
            }
        }
        if (required > 1 && h > c.min_step_abs * 1.0001) {
            h_current = max_val(c.min_step_abs, over_pow2(h, required));
            cap = h_current;
            continue;
        }
        cap = c.max_step;
        if (pred > 1 && (local_max_rs > 0.0 || c.max_radiation_depth > 0.0 || c.max_absorption_depth > 0.0 ||
                         c.max_faraday_depth > 0.0))
            cap = max_val(c.min_step_abs, over_pow2(h_current, pred));
        if (!radiating) {
#pragma unroll
            for (int f = 0; f < NF; ++f) RT::add_zero(stokes[f]);
        } else if (h > 0.0) {
#pragma unroll 1
            for (int f = 0; f < nf; ++f) RT::step(stokes[f], co[f], h, c, f);
        }
        state = next;
        start_r = next_r;
        steps += 1;
        if (crosses) reached = 1;
    }
    reason = reached ? kReachedCamera : kMaxSteps;
}

// The plain FP64 kernel with one thread per pixel, fixed steps.
template<int NF>
__global__ void __launch_bounds__(kImageThreads, kImageBlocks) image_fp64_fixed(const __grid_constant__ JobDesc job) {
    const int pixel = blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= job.npix) return;
    const ImageConsts& c = job.c;
    const Ray cam = camera_ray(c, job.frame, pixel);
    Ray state = cam;
    PixelOut o;
    o.steps = 0;
    int reason = kMaxSteps;
    const int valid = trace_pass_a(c, state, o.pass_a_steps, reason);
    Stokes4<double> stokes[NF];
#pragma unroll
    for (int f = 0; f < NF; ++f) stokes[f] = Stokes4<double>{0.0, 0.0, 0.0, 0.0};
    if (valid) trace_pass_b_fixed<NF>(c, state, stokes, o.steps, reason);
    o.reason = reason;
    double obs[NF][4];
    finish_ray<double, NF>(c, cam, state, valid, stokes, o, obs);
    store_stokes_n<NF>(job.out, pixel, job.npix, c.nfreq, obs);
    store_diagnostics(job.out, pixel, o);
}

// The plain FP64 kernel with one thread per pixel, adaptive steps.
template<int NF>
__global__ void __launch_bounds__(kImageThreads, kImageBlocks) image_fp64_per_lane(const __grid_constant__ JobDesc job) {
    WaveDesc W = {};
    W.jobs = &job;
    W.njobs = 1;
    W.fresh_end = job.npix;
    lane_body<PolicyFP64, NF, kPhaseAll>(W);
}

cudaError_t launch_image_lanes(const JobDesc& job, cudaStream_t stream) {
    const int grid = (job.npix + kImageThreads - 1) / kImageThreads;
    if (!job.c.adaptive) {
        if (job.c.nfreq == 1) image_fp64_fixed<1><<<grid, kImageThreads, 0, stream>>>(job);
        else image_fp64_fixed<kMaxFreq><<<grid, kImageThreads, 0, stream>>>(job);
    } else if (job.c.nfreq == 1) image_fp64_per_lane<1><<<grid, kImageThreads, 0, stream>>>(job);
    else image_fp64_per_lane<kMaxFreq><<<grid, kImageThreads, 0, stream>>>(job);
    return cudaGetLastError();
}
#endif

}  // namespace kp
