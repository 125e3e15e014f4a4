// kp_kernels_grmhd_slow_mixed.cu -- slow-light GRMHD images (FMKS metric, grid plasma interpolated
// in time between resident snapshots) on the wavefront engine with
// the mixed policy (factored geodesic, fits and transfer, all of it FP64).  Compiled with FMA contraction.
#include <cuda_runtime.h>

#include "kp_launch.h"
#include "kp_quad.cuh"

namespace kp {

__global__ void __launch_bounds__(kFarThreads, kFarBlocks) wave_far_grmhd_slow_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseFar, SceneFarCks<SceneGrmhdSlow>>(W);
}

__global__ void __launch_bounds__(kNearAThreads, kNearABlocks) wave_near_a_grmhd_slow_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearA, SceneGrmhdSlow>(W);
}

__global__ void __launch_bounds__(kNearBThreads, kNearBBlocks) wave_near_b_grmhd_slow_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearB, SceneGrmhdSlow>(W);
}

static const void* wave_kernel_grmhd_slow_mixed(int phase) {
    if (phase == kPhaseFar) return reinterpret_cast<const void*>(wave_far_grmhd_slow_mixed);
    if (phase == kPhaseNearA) return reinterpret_cast<const void*>(wave_near_a_grmhd_slow_mixed);
    return reinterpret_cast<const void*>(wave_near_b_grmhd_slow_mixed);
}

cudaError_t launch_wave_grmhd_slow_mixed(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                              cudaStream_t stream) {
    const void* const fn[2] = {wave_kernel_grmhd_slow_mixed(phase), nullptr};  // one image to a launch
    return launch_forms<PolicyMixed, SceneGrmhdSlow>(fn, phase, W, nf_max, blocks, threads, stream);
}

int wave_occupancy_grmhd_slow_mixed(int phase, int nf_max, int threads) {
    if (phase < 0 || phase >= kPhases) return 0;
    const void* fn = wave_kernel_grmhd_slow_mixed(phase);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, 0);
    return n;
}

}  // namespace kp
