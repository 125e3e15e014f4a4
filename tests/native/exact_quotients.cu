// Test probe (test infrastructure, not part of the library): the quotients
// and square roots of kpolaris_b200/csrc/kp_exact.cuh on the GPU against
// CUDA's own operators, and the errors of the mixed policy's reciprocals and
// roots.  Built by tests/test_exact_quotients.py with the FP64 kernels' flags.
#include <cuda_runtime.h>

#include "kp_exact.cuh"
#include "exact_quotients.h"
#include "kp_radiation_mixed.cuh"

namespace {

__global__ void check_kernel(int draws, xq::Counts* out) {
    uint64_t s = 0x9E3779B97F4A7C15ull * uint64_t(blockIdx.x * blockDim.x + threadIdx.x + 1);
    for (int i = 0; i < 8; ++i) xq::next(s);
    xq::Counts n = {};
    for (int i = 0; i < draws; ++i) xq::check(s, n);
    atomicAdd(&out->quots, n.quots);
    atomicAdd(&out->over, n.over);
    atomicAdd(&out->quot, n.quot);
    atomicAdd(&out->recip, n.recip);
    atomicAdd(&out->root, n.root);
}

__device__ void largest(double* out, double got, double want) {
    atomicMax(reinterpret_cast<unsigned long long*>(out), (unsigned long long)__double_as_longlong(fabs(got - want) / want));
}

// Relative errors of kp_recip, both results of kp_sqrt_pair, and cube_root in
// x = 1..1e7 and over its whole range.
__global__ void mixed_kernel(int draws, double* out) {
    uint64_t s = 0x9E3779B97F4A7C15ull * uint64_t(blockIdx.x * blockDim.x + threadIdx.x + 1);
    for (int i = 0; i < 8; ++i) xq::next(s);
    for (int i = 0; i < draws; ++i) {
        const double v = xq::number(s, 900, false);
        double root, inv;
        kp::kp_sqrt_pair(v, root, inv);
        largest(out, kp::kp_recip(v), 1.0 / v);
        largest(out + 1, root, sqrt(v));
        largest(out + 2, inv, 1.0 / sqrt(v));
        const double x = xq::number(s, 200, false);
        largest(out + (x >= 1.0 && x <= 1e7 ? 3 : 4), kp::cube_root(x), cbrt(x));
    }
}

}  // namespace

// 148 * 128 threads, `draws` draws each; returns 0 or a cudaError_t.
extern "C" int kp_probe_mixed_roots(int draws, double* errors) {
    double* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 5 * sizeof(double));
    if (e == cudaSuccess) e = cudaMemset(d, 0, 5 * sizeof(double));
    if (e == cudaSuccess) {
        mixed_kernel<<<148, 128>>>(draws, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(errors, d, 5 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}

// 148 * 128 threads, `draws` draws each; returns 0 or a cudaError_t.
extern "C" int kp_probe_exact_quotients(int draws, unsigned long long* counts) {
    xq::Counts* d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(xq::Counts));
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(xq::Counts));
    if (e == cudaSuccess) {
        check_kernel<<<148, 128>>>(draws, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(counts, d, sizeof(xq::Counts), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return int(e);
}
