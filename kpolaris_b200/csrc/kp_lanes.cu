// kp_lanes.cu -- the phase kernels with one ray per lane (lane_body in
// kp_persistent.cuh), for launches with rays enough to fill the device.
// Compiled once per policy and scene: KP_LANES_POLICY, KP_LANES_SCENE, with the
// floating-point flags of that policy's quad kernels.  Near-A and near-B run
// as one CTA of 256 threads per SM, whose warps step through the same code
// region (near-A of 8 x 256^2 FP64: 85 ms, as two CTAs of 128 95 ms), with
// exp, log and pow inlined (near-B, four frequencies: 491 ms, as calls 513 ms).
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
    const void* fn = reinterpret_cast<const void*>(lanes_near_a<P, SC>);
    if (phase == kPhaseFar)
        fn = nf_max == 1 ? reinterpret_cast<const void*>(lanes_far<P, 1, SC>)
                         : reinterpret_cast<const void*>(lanes_far<P, kMaxFreq, SC>);
    else if (phase == kPhaseNearB)
        fn = nf_max == 1 ? reinterpret_cast<const void*>(lanes_near_b<P, 1, SC>)
                         : reinterpret_cast<const void*>(lanes_near_b<P, kMaxFreq, SC>);
    const int threads = phase == kPhaseFar ? kFarThreads : kLaneNearThreads;
    void* args[] = {const_cast<WaveDesc*>(&W), &quad_rays};
    return cudaLaunchKernel(fn, dim3(unsigned((lanes + threads - 1) / threads)), dim3(threads), args, 0, stream);
}

template cudaError_t launch_lanes<KP_LANES_POLICY, KP_LANES_SCENE>(int, const WaveDesc&, int, long long, long long,
                                                                   cudaStream_t);

#ifdef KP_LANES_IMAGE
// The plain FP64 kernel with one thread per pixel.
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
    if (job.c.nfreq == 1) image_fp64_per_lane<1><<<grid, kImageThreads, 0, stream>>>(job);
    else image_fp64_per_lane<kMaxFreq><<<grid, kImageThreads, 0, stream>>>(job);
    return cudaGetLastError();
}
#endif

}  // namespace kp
