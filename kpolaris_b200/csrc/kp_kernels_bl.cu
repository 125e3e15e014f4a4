// kp_kernels_bl.cu -- the RIAF in Boyer-Lindquist coordinates (SceneRiafBL)
// on the wavefront engine with the FP64 policy, compiled without FMA contraction so the arithmetic stays closest to the reference's CPU rounding.
#include <cuda_runtime.h>

#define KP_MATH_CALLS 1  // kp_radiation.cuh
#include "kp_launch.h"
#include "kp_quad.cuh"

namespace kp {

__global__ void __launch_bounds__(kFarThreads, kFarBlocks) wave_bl_far(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseFar, SceneRiafBL>(W);
}

__global__ void __launch_bounds__(kNearAThreads, kNearABlocks) wave_bl_near_a(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseNearA, SceneRiafBL>(W);
}

__global__ void __launch_bounds__(kNearBThreads, kNearBBlocks) wave_bl_near_b(const WaveDesc W, long long quad_rays) {
    if (wave_rays(W) <= quad_rays) quad_body<PolicyFP64, kPhaseNearB, SceneRiafBL>(W);
}

static const void* wave_bl_kernel(int phase) {
    if (phase == kPhaseFar) return reinterpret_cast<const void*>(wave_bl_far);
    if (phase == kPhaseNearA) return reinterpret_cast<const void*>(wave_bl_near_a);
    return reinterpret_cast<const void*>(wave_bl_near_b);
}

cudaError_t launch_wave_bl(int phase, const WaveDesc& W, int nf_max, int blocks, int threads, cudaStream_t stream) {
    return launch_wave<PolicyFP64, SceneRiafBL>(wave_bl_kernel(phase), phase, W, nf_max, false, blocks, threads, stream);
}

int wave_occupancy_bl(int phase, int nf_max, int threads) {
    if (phase < 0 || phase >= kPhases) return 0;
    const void* fn = wave_bl_kernel(phase);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, 0);
    return n;
}

}  // namespace kp
