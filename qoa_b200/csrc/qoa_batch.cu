// qoa_batch.cu — shots of sampled batch circuits.
#include <cuda_runtime.h>
#include <stdint.h>

#include "qoa_kernels.cuh"

namespace qoa {

// --------------------------------------------------------------------------
// Shots of sampled batch circuits: one CTA per circuit builds the marginal
// tree of its final state in global scratch (level k, 1 <= k < n, holds the
// 2^k sums over qubits k..n-1 at tree + 2^k - 2, each the sum of two values of
// level k + 1 that differ in their top bit), then each thread takes shots and
// walks the tree from qubit 0 by inverse CDF (bit q = 0 while the remaining mass
// is below the marginal of that prefix). The tree is not divided by the norm:
// the states of a batch are unit vectors up to rounding, and t = u x total
// scales with it.
__device__ __forceinline__ double samp_abs2(const double2* a, uint64_t i) {
    const double2 x = a[i];
    return fma(x.x, x.x, x.y * x.y);
}
__device__ __forceinline__ double samp_abs2(const float2* a, uint64_t i) {
    const float2 x = a[i];
    return (double)x.x * x.x + (double)x.y * x.y;
}

template <typename T>
__global__ void __launch_bounds__(1024) k_sample_jobs(const SampleJob* __restrict__ jobs, const double* __restrict__ u,
                                                      unsigned long long* __restrict__ out) {
    const SampleJob J = jobs[blockIdx.x];
    const T* a = reinterpret_cast<const T*>(J.amps);
    const uint32_t n = J.n;
    double* tree = J.tree;
    if (n >= 2) {
        const uint64_t half = 1ull << (n - 1);
        double* leaf = tree + (half - 2);
        for (uint64_t p = threadIdx.x; p < half; p += blockDim.x) leaf[p] = samp_abs2(a, p) + samp_abs2(a, p + half);
        __syncthreads();
        for (int k = (int)n - 2; k >= 1; --k) {
            const uint64_t cnt = 1ull << k;
            const double* hi = tree + ((2ull << k) - 2);
            double* lo = tree + (cnt - 2);
            for (uint64_t p = threadIdx.x; p < cnt; p += blockDim.x) lo[p] = hi[p] + hi[p + cnt];
            __syncthreads();
        }
    }
    auto h = [&](uint32_t k, uint64_t p) -> double {
        if (k == n) return samp_abs2(a, p);
        if (k == 0) return n == 1 ? samp_abs2(a, 0) + samp_abs2(a, 1) : tree[0] + tree[1];
        return tree[((1ull << k) - 2) + p];
    };
    for (uint32_t s = threadIdx.x; s < J.shots; s += blockDim.x) {
        double t = u[J.u_start + s] * h(0, 0);
        uint64_t pre = 0;
        for (uint32_t q = 0; q < n; ++q) {
            const double left = h(q + 1, pre);
            if (t < left) continue;
            t -= left;
            pre |= 1ull << q;
        }
        out[J.out_start + s] = pre;
    }
}

cudaError_t launch_sample_jobs(bool f32, const SampleJob* jobs, uint32_t njobs, const double* u,
                               unsigned long long* out, cudaStream_t st) {
    if (!njobs) return cudaSuccess;
    if (f32) k_sample_jobs<float2><<<njobs, 1024, 0, st>>>(jobs, u, out);
    else k_sample_jobs<double2><<<njobs, 1024, 0, st>>>(jobs, u, out);
    return cudaGetLastError();
}

}  // namespace qoa
