// kp_kernels_bl_mixed.cu -- the RIAF in Boyer-Lindquist coordinates (SceneRiafBL)
// on the wavefront engine with the mixed policy (FP64 BL geodesic, factored fits), compiled with FMA contraction.
#include <cuda_runtime.h>

#include "kp_launch.h"
#include "kp_quad.cuh"

namespace kp {

// one form whatever shares the launch: compiled for one frequency, the end of
// a ray rounds differently
__global__ void __launch_bounds__(kFarThreads, 2) wave_bl_mixed_far(const WaveDesc W) {
    lane_body<PolicyMixed, kMaxFreq, kPhaseFar, SceneRiafBL>(W);
}

template<bool SHARED>
__global__ void __launch_bounds__(kNearAThreads, kNearABlocks) wave_bl_mixed_near_a(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearA, SceneRiafBL, SHARED>(W);
}

template<bool SHARED>
__global__ void __launch_bounds__(kNearBThreads, kNearBBlocks) wave_bl_mixed_near_b(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearB, SceneRiafBL, SHARED>(W);
}

template<bool SHARED>
static const void* wave_bl_mixed_kernel(int phase) {
    if (phase == kPhaseFar) return reinterpret_cast<const void*>(wave_bl_mixed_far);
    if (phase == kPhaseNearA) return reinterpret_cast<const void*>(wave_bl_mixed_near_a<SHARED>);
    return reinterpret_cast<const void*>(wave_bl_mixed_near_b<SHARED>);
}

cudaError_t launch_wave_bl_mixed(int phase, const WaveDesc& W, int nf_max, int blocks, int threads, cudaStream_t stream) {
    const void* const fn[2] = {wave_bl_mixed_kernel<false>(phase), wave_bl_mixed_kernel<true>(phase)};
    return launch_forms<PolicyMixed, SceneRiafBL>(fn, phase, W, nf_max, blocks, threads, stream);
}

int wave_occupancy_bl_mixed(int phase, int nf_max, int threads) {
    if (phase < 0 || phase >= kPhases) return 0;
    const void* fn = wave_bl_mixed_kernel<false>(phase);
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, 0);
    return n;
}

}  // namespace kp
