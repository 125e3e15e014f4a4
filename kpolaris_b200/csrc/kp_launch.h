// kp_launch.h -- internal launch interface between the C-ABI host code
// (kp_capi.cu) and the kernel translation units.
#pragma once

#include <cuda_runtime.h>

#include "kp_common.cuh"

namespace kp {

// Plain FP64 kernel, one image: one quad per pixel (kp_kernels_fp64.cu), or
// one thread (kp_lanes.cu).
cudaError_t launch_image_fp64(const ImageConsts& c, const ImageOutPtrs& out, int sms, cudaStream_t stream);
cudaError_t launch_image_lanes(const JobDesc& job, cudaStream_t stream);
// Analysis mode: the per-pixel FP64 image with the line-of-sight
// diagnostics (one frequency; radial_bins in 1..24).
constexpr int kMaxRadialBins = 24;  // KPOLARIS_MAX_ANALYSIS_RADIAL_BINS

struct AnalysisConsts {
    int radial_bins;
    double radial_min, radial_max, formation_fraction;
};

// Device arrays of the analysis outputs: scalars [npix]; radial arrays
// [radial_bins][npix].
struct AnalysisPtrs {
    double* radiating_path_length;
    double* emission_weight;
    double* emission_weighted_radius;
    double* emission_weighted_optical_depth_to_camera;
    double* absorption_depth;
    double* absorption_operator_depth;
    double* faraday_rotation_depth;
    double* faraday_conversion_depth;
    double* faraday_operator_depth;
    double* dominant_emission_radius;
    int32_t* dominant_emission_region;
    double* dominant_ne_cgs;
    double* dominant_thetae;
    double* dominant_b_cgs;
    double* dominant_beta;
    double* dominant_sigma;
    double* emission_weighted_ne_cgs;
    double* emission_weighted_thetae;
    double* emission_weighted_b_cgs;
    double* emission_weighted_beta;
    double* emission_weighted_sigma;
    double* photon_ring_winding_estimate;
    int32_t* radiation_substeps;
    double* radial_stokes_i;
    double* radial_stokes_q;
    double* radial_stokes_u;
    double* radial_stokes_v;
    double* radial_absorption_depth;
    double* radial_faraday_rotation_depth;
    double* radial_faraday_conversion_depth;
    double* radial_faraday_operator_depth;
    double* observer_weighted_radius_i;
    double* observer_weighted_radius_linear;
    double* observer_weighted_radius_circular;
    double* intensity_formation_radius_low;
    double* intensity_formation_radius_median;
    double* intensity_formation_radius_high;
    double* linear_formation_radius_low;
    double* linear_formation_radius_median;
    double* linear_formation_radius_high;
    double* circular_formation_radius_low;
    double* circular_formation_radius_median;
    double* circular_formation_radius_high;
    double* los_linear_coherence;
    double* los_circular_coherence;
    double* contribution_closure_max_abs;
    double* contribution_closure_relative_l1;
    double* foreground_absorption_depth;
    double* foreground_faraday_rotation_depth;
    double* foreground_faraday_conversion_depth;
    double* foreground_faraday_operator_depth;
    double* foreground_faraday_operator_fraction;
};

cudaError_t launch_image_fp64_analysis(const ImageConsts& c, const AnalysisConsts& k, const ImageOutPtrs& out,
                                       const AnalysisPtrs& an, const kp_response_config* resp, double* resp_data,
                                       cudaStream_t stream);

// Camera tetrad of an image, evaluated on the host (bit-identical to the
// reference's CPU evaluation): Cartesian Kerr-Schild, or Boyer-Lindquist for
// a kSceneRiafBL image.
void host_camera_frame(const ImageConsts& c, double frame[5][4]);

// Wavefront engine: one launch of `phase` (kPhaseFar / kPhaseNear) over the
// inputs described by `W` (a host copy whose pointers are device pointers).
// nf_max: the largest frequency count of the launch's jobs.
cudaError_t launch_wave_fp64(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                             cudaStream_t stream);
cudaError_t launch_wave_mixed(int phase, const WaveDesc& W, int blocks, int threads, cudaStream_t stream);
// Resident CTAs per SM of a phase kernel at `threads` per CTA.
int wave_occupancy_fp64(int phase, int nf_max, int threads);
int wave_occupancy_mixed(int phase, int threads);

// Seed kernels of the serving loop (same translation unit, hence the same
// camera-ray arithmetic, as the policy's phase kernels): initial records of
// the rays of newly admitted jobs, appended to the far queue.
cudaError_t launch_seed_fp64(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix, int nentries,
                             long long total, RayRecord* pool, unsigned* far_ids, unsigned* far_count,
                             cudaStream_t stream);
cudaError_t launch_seed_mixed(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix, int nentries,
                              long long total, RayRecord* pool, unsigned* far_ids, unsigned* far_count,
                              cudaStream_t stream);

// The GRMHD scene (FMKS metric, grid plasma), FP64 policy
// (kp_kernels_grmhd.cu), its seed kernel and the derived-scalar precompute
// (derived: [5][n1][n2][n3] device array).
cudaError_t launch_wave_grmhd(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                              cudaStream_t stream);
int wave_occupancy_grmhd(int phase, int nf_max, int threads);
// The same scene under the mixed policy (kp_kernels_grmhd_mixed.cu).
cudaError_t launch_wave_grmhd_mixed(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                                    cudaStream_t stream);
int wave_occupancy_grmhd_mixed(int phase, int nf_max, int threads);
cudaError_t launch_seed_grmhd_mixed(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix,
                                    int nentries, long long total, RayRecord* pool, unsigned* far_ids,
                                    unsigned* far_count, cudaStream_t stream);
// The RIAF in Boyer-Lindquist coordinates, FP64 policy (kp_kernels_bl.cu)
// and mixed policy (kp_kernels_bl_mixed.cu).
cudaError_t launch_wave_bl(int phase, const WaveDesc& W, int nf_max, int blocks, int threads, cudaStream_t stream);
int wave_occupancy_bl(int phase, int nf_max, int threads);
cudaError_t launch_wave_bl_mixed(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                                 cudaStream_t stream);
int wave_occupancy_bl_mixed(int phase, int nf_max, int threads);
// Longest-first order of a near-B queue (kp_reorder.cu): `count` ids from
// `ids` into `out`, grouped by pass-A steps, most first; `scratch` holds 512
// unsigned counters.
cudaError_t launch_lpt_order(const unsigned* ids, const unsigned* count, const RayRecord* pool, unsigned* scratch,
                             unsigned* out, int sms, cudaStream_t stream);
// Slow-light GRMHD (kp_kernels_grmhd_slow.cu, kp_kernels_grmhd_slow_mixed.cu).
cudaError_t launch_wave_grmhd_slow(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                                   cudaStream_t stream);
int wave_occupancy_grmhd_slow(int phase, int nf_max, int threads);
cudaError_t launch_wave_grmhd_slow_mixed(int phase, const WaveDesc& W, int nf_max, int blocks, int threads,
                                         cudaStream_t stream);
int wave_occupancy_grmhd_slow_mixed(int phase, int nf_max, int threads);
cudaError_t launch_seed_grmhd(const JobDesc* jobs, const SeedEntry* entries, const long long* prefix, int nentries,
                              long long total, RayRecord* pool, unsigned* far_ids, unsigned* far_count,
                              cudaStream_t stream);
// Reference-layout primitives [8][ncell] into the cell-major device grid.
cudaError_t launch_grid_to_cells(const float* soa, float* cells, long long ncell, int sms, cudaStream_t stream);
cudaError_t launch_grid_derived(const GridConsts& g, double* derived, int sms, cudaStream_t stream);

// Launches of one wavefront batch run in cycles of (far, near-A, near-B)
// until no ray is left; a batch whose rays still move between phases after
// this many cycles ends with KP_ERR_TIMEOUT (a 256x256 image takes 2 cycles,
// rays grazing the radiating sphere a few more).
constexpr int kMaxWaveCycles = 24;

// Threads per CTA of each phase kernel and resident CTAs per SM they are
// compiled for: 8 warps of 255 registers per SM.  Near-B's one large CTA keeps
// all of them in step (8 x 256^2 mixed: 189 ms against 197 ms for two CTAs);
// near-A and the far phase are faster in two (57 against 62 ms).  12 warps of
// 168 registers spill: a 128^2 image at 60 degrees took 293 instead of 219 ms.
constexpr int kFarThreads = 128, kFarBlocks = 2;
constexpr int kNearAThreads = 128, kNearABlocks = 2;
constexpr int kNearBThreads = 256, kNearBBlocks = 1;
constexpr int kImageThreads = 32, kImageBlocks = 8;  // the plain FP64 kernel: a warp's slot is free when its own rays end
constexpr int kLaneNearThreads = 256;  // near-A and near-B with one ray per lane
inline int wave_threads(int phase) {
    return phase == kPhaseFar ? kFarThreads : (phase == kPhaseNearA ? kNearAThreads : kNearBThreads);
}
// CTAs that give every ray a warp: more would only idle.
inline long long wave_blocks_needed(int phase, long long rays) {
    const int warps = wave_threads(phase) / 32;
    return (rays + warps - 1) / warps;
}

// Rays up to which a phase of the FP64 policy runs on quads; beyond, on lanes
// (kp_lanes.cu).  `quads`: those of the phase's grid (9,472 on a B200).  The
// lanes of a quad repeat the connection, so where rays fill the device lanes
// are faster; near-B's quads share out the frequencies, which moves the line
// up with their number unless FMKS makes the connection the larger part.
// Measured, quads / lanes (ms), which agree bit for bit:
//   far     128^2 26 / 26, 256^2 116 / 50
//   near-A  256^2 16.6 / 17.7, 320^2 24.2 / 22.7, 512^2 61 / 37, 8 x 256^2 124 / 82
//   near-B  1 frequency: 256^2 at 60 degrees 70 / 71, 512^2 166 / 72, 8 x 256^2 331 / 137
//           2: 320^2 161 / 168, 512^2 338 / 282, 8 x 256^2 670 / 330
//           4: 384^2 202 / 217, 512^2 344 / 343, 4 x 320^2 at 10 to 70 degrees 1655 / 1870,
//              8 x 256^2 678 / 472
//   fixed steps, which are much of a length: near-B 192^2 32 / 11
//   GRMHD   256^2 177 / 185, 320^2 266 / 263, 512^2 628 / 474; four frequencies 720 / 582
// (near-B: lanes until its input runs out, the rest on quads.  Without that
// 4 x 320^2 took 3243, 8 x 256^2 492.)
inline long long quad_rays(int phase, int nf_max, bool fmks, bool fixed_steps, long long quads) {
    if (phase == kPhaseFar || fixed_steps) return quads;
    if (phase == kPhaseNearA || nf_max == 1 || fmks) return 8 * quads;
    return (nf_max == 2 ? 24 : 48) * quads;
}

// Pixels up to which the plain FP64 kernel gives each a quad: with fixed
// steps, whose rays are much of a length, while every ray gets one of its own
// (96^2 32 / 31 ms, 128^2 56 / 31, 256^2 209 / 87); with adaptive steps until the longest rays no longer
// set the time (quads / lanes: one frequency 192^2 122 / 131, 256^2 217 / 165,
// 1024^2 3205 / 1873; two 256^2 378 / 381, 512^2 1313 / 1075; four 512^2 1336
// / 1439, 768^2 2900 / 2510).
inline long long image_quad_pixels(int nfreq, bool adaptive, int sms) {
    return (!adaptive ? 1 : (nfreq == 1 ? 5 : (nfreq == 2 ? 24 : 48))) * 64ll * sms;
}

// One launch of a phase: the quad kernel and, where there can be more rays
// than it takes, the lane kernel; whichever the launch's ray count is not for
// returns at once.  The lane kernel of near-B hands at most its `lanes` rays
// on, 4 per quad, which the next launch takes on quads (their line is above).
template<class P, class SC>
cudaError_t launch_lanes(int phase, const WaveDesc& W, int nf_max, long long lanes, long long quad_rays,
                         cudaStream_t stream);

template<class P, class SC>
inline cudaError_t launch_wave(const void* quad_kernel, int phase, const WaveDesc& W, int nf_max, bool fmks,
                               int blocks, int threads, cudaStream_t stream) {
    if (nf_max < 1 || nf_max > kMaxFreq || phase < 0 || phase >= kPhases) return cudaErrorInvalidValue;
    const long long lanes = (long long)blocks * threads;
    long long rays = quad_rays(phase, nf_max, fmks, W.fixed_steps, lanes / 4);
    if (W.fresh_end - W.fresh_begin <= rays) {
        void* args[] = {const_cast<WaveDesc*>(&W), &rays};
        const cudaError_t e = cudaLaunchKernel(quad_kernel, dim3(blocks), dim3(threads), args, 0, stream);
        if (e != cudaSuccess || W.rays_max <= rays) return e;
    }
    return launch_lanes<P, SC>(phase, W, nf_max, lanes, rays, stream);
}

// Whether an image's near phases run with one ray per lane under the mixed
// policy.  The forms round differently, so the line is drawn by the image
// alone: an image is the same in a batch, in a server and by itself.  Measured,
// quads / lanes (ms per image):
//   GRMHD           256^2 69 / 89, 320^2 108 / 130, 384^2 152 / 142, 512^2 270 / 206;
//                   four frequencies 384^2 184 / 180, 512^2 322 / 263
//   slow light      320^2 106 / 106, 512^2 262 / 169
//   Boyer-Lindquist one frequency 256^2 102 / 104, 320^2 152 / 136, 512^2 356 / 287; four
//                   512^2 482 / 537 (the longest rays of a Faraday-thick image set the time,
//                   and a quad steps them faster)
// Cartesian Kerr-Schild images keep the quads: one of 512^2 at one frequency takes
// 103 / 71, but images of many sizes share launches there, and 64 of 32^2 to
// 512^2 take 2.62 s on quads, 2.78 s with the larger ones on lanes, whose
// kernels end with their own longest rays after those of the quads.
inline int lane_image(const ImageConsts& c, int npix) {
    if (c.scene == kSceneRiafCks) return 0;
    if (c.scene == kSceneRiafBL) return npix > (c.nfreq == 1 ? 80000 : 800000);
    return npix > 120000;
}

// A launch of a phase under the mixed policy: one kernel for each form that
// its images take.  `quad_kernel`: of the phase, and of the phase where it
// shares its launch with lanes (the test of every ray's form costs an
// image alone 2% of its time).
template<class P, class SC>
inline cudaError_t launch_forms(const void* const (&quad_kernel)[2], int phase, const WaveDesc& W, int nf_max,
                                int blocks, int threads, cudaStream_t stream) {
    if (nf_max < 1 || nf_max > kMaxFreq || phase < 0 || phase >= kPhases) return cudaErrorInvalidValue;
    const bool lanes = phase != kPhaseFar && (W.forms & kFormLanes);
    if (!lanes || (W.forms & kFormQuads)) {
        void* args[] = {const_cast<WaveDesc*>(&W)};
        const cudaError_t e = cudaLaunchKernel(quad_kernel[lanes], dim3(blocks), dim3(threads), args, 0, stream);
        if (e != cudaSuccess || !lanes) return e;
    }
    return launch_lanes<P, SC>(phase, W, nf_max, (long long)blocks * threads, -1, stream);
}

}  // namespace kp
