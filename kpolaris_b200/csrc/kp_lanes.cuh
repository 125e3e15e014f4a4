// kp_lanes.cuh -- the phase kernels with one ray per lane (lane_body in
// kp_persistent.cuh), for images and launches with rays enough to fill the
// device.  Near-A and near-B run as one CTA of 256 threads per SM, whose warps
// step through the same code region (near-A of 8 x 256^2 FP64: 85 ms, as two
// CTAs of 128 95 ms).
#pragma once

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

}  // namespace kp
