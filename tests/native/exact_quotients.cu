// Test probe (test infrastructure, not part of the library): the quotients
// and square roots of kpolaris_b200/csrc/kp_exact.cuh on the GPU against
// CUDA's own operators.  Built by tests/test_exact_quotients.py with the FP64
// kernels' flags.
#include <cuda_runtime.h>

#include "kp_exact.cuh"
#include "exact_quotients.h"

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

}  // namespace

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
