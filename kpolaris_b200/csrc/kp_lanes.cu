// kp_lanes.cu -- the FP64 policy's kernels with one ray per lane
// (kp_lanes.cuh).  Compiled once per scene (KP_LANES_SCENE), without FMA
// contraction, with exp, log and pow inlined (near-B of 8 x 256^2, four
// frequencies: 491 ms, as the calls of the quad kernels 513 ms).
#include <cuda_runtime.h>

#include "kp_lanes.cuh"

namespace kp {

template cudaError_t launch_lanes<PolicyFP64, KP_LANES_SCENE>(int, const WaveDesc&, int, long long, long long,
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
