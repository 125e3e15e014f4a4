// kp_kernels_grmhd_slow.cu -- slow-light GRMHD images (FMKS metric, grid plasma interpolated
// in time between resident snapshots) on the wavefront engine with
// the FP64 policy. Compiled without FMA contraction, as the fast-light GRMHD kernels.
#include <cuda_runtime.h>

#define KP_MATH_CALLS 1  // kp_radiation.cuh
#include "kp_launch.h"
#include "kp_quad.cuh"

namespace kp {

__global__ void __launch_bounds__(kFarThreads, kFarBlocks) wave_far_grmhd_slow(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseFar, SceneGrmhdSlow>(W);
}

__global__ void __launch_bounds__(kNearAThreads, kNearABlocks) wave_near_a_grmhd_slow(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseNearA, SceneGrmhdSlow>(W);
}

__global__ void __launch_bounds__(kNearBThreads, kNearBBlocks) wave_near_b_grmhd_slow(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseNearB, SceneGrmhdSlow>(W);
}

static const void* wave_kernel_grmhd_slow(int phase) {
    if (phase == kPhaseFar) return reinterpret_cast<const void*>(wave_far_grmhd_slow);
    if (phase == kPhaseNearA) return reinterpret_cast<const void*>(wave_near_a_grmhd_slow);
    return reinterpret_cast<const void*>(wave_near_b_grmhd_slow);
}

cudaError_t launch_wave_grmhd_slow(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                              cudaStream_t stream) {
    return launch_wave<PolicyFP64, SceneGrmhdSlow>(wave_kernel_grmhd_slow(phase), phase, W, nf_max, true, blocks, threads, stream);
}

int wave_occupancy_grmhd_slow(int phase, int nf_max, int threads) {
    if (phase < 0 || phase >= kPhases) return 0;
    const void* fn = wave_kernel_grmhd_slow(phase);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, 0);
    return n;
}

}  // namespace kp
