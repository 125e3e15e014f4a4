// kp_kernels_mixed.cu -- the mixed policy's wavefront kernels: FP64 in
// factored, contracted forms that round differently from the reference, and
// many far-field steps at once.  Compiled with FMA contraction enabled.
#include <cuda_runtime.h>

#include "kp_launch.h"
#include "kp_quad.cuh"

namespace kp {

__global__ void __launch_bounds__(kFarThreads, kFarBlocks) wave_far_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseFar>(W);
}

__global__ void __launch_bounds__(kNearAThreads, kNearABlocks) wave_near_a_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearA>(W);
}

__global__ void __launch_bounds__(kNearBThreads, kNearBBlocks) wave_near_b_mixed(const WaveDesc W) {
    quad_body<PolicyMixed, kPhaseNearB>(W);
}

static const void* wave_kernel_mixed(int phase) {
    if (phase == kPhaseFar) return reinterpret_cast<const void*>(wave_far_mixed);
    if (phase == kPhaseNearA) return reinterpret_cast<const void*>(wave_near_a_mixed);
    return reinterpret_cast<const void*>(wave_near_b_mixed);
}

cudaError_t launch_wave_mixed(int phase, const WaveDesc& W, int blocks, int threads, cudaStream_t stream) {
    if (phase < 0 || phase >= kPhases) return cudaErrorInvalidValue;
    void* args[] = {const_cast<WaveDesc*>(&W)};
    return cudaLaunchKernel(wave_kernel_mixed(phase), dim3(blocks), dim3(threads), args, 0, stream);
}

__global__ void __launch_bounds__(128) seed_mixed(const JobDesc* jobs, const SeedEntry* entries,
                                                 const long long* prefix, int nentries, RayRecord* pool,
                                                 unsigned* far_ids, unsigned* far_count) {
    seed_body<SceneRiaf>(jobs, entries, prefix, nentries, pool, far_ids, far_count);
}

cudaError_t launch_seed_mixed(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix, int nentries,
                              long long total, RayRecord* pool, unsigned* far_ids, unsigned* far_count,
                              cudaStream_t stream) {
    if (total <= 0) return cudaSuccess;
    const int grid = int((total + 127) / 128);
    seed_mixed<<<grid, 128, 0, stream>>>(jobs, entries, prefix, nentries, pool, far_ids, far_count);
    return cudaGetLastError();
}

int wave_occupancy_mixed(int phase, int threads) {
    if (phase < 0 || phase >= kPhases) return 0;
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wave_kernel_mixed(phase), threads, 0);
    return n;
}

}  // namespace kp
