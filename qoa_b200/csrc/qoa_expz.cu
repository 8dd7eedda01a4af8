// qoa_expz.cu — <Z_mask> = sum_i (-1)^popcount(i & mask) |a_i|^2 for many masks
// in one sweep of the state.
//
// A CTA takes a tile of 4096 amplitudes: 16 squares a thread, and replaces
// them by their Walsh-Hadamard transform over index bits 4..11 (two rounds of
// four butterfly stages in registers with one exchange through shared memory
// between them). A mask's sum over the tile is then 16 of the 4096 values
// (the row its bits 4..11 name), signed by its bits 0..3 and by the parity of
// the tile's own index: one load and one add a tile for each of 16 lanes. The
// cost per amplitude is 2 + 8 FP64 instructions whatever the number of masks,
// up to 256 at once, where summing mask by mask costs a popcount, a select
// and an add per amplitude and mask, and a sweep of the state per 8 masks.
// It is bound by reading the state (HBM, or L2 where the state fits). Measured
// on B200 against sweeps of 8 masks: 27 qubits complex128, 16 masks 1573 ->
// 313 us (6.9 TB/s); 23 qubits complex64, 45 masks 288 -> 29 us (2.3 TB/s, in
// L2); 119 batch circuits of 13 to 20 qubits, 8 masks each 229 -> 82 us.
#include <cuda_runtime.h>

#include <stdint.h>

#include "qoa_kernels.cuh"
#include "qoa_launch.cuh"
#include "qoa_pass_dev.cuh"

namespace qoa {

namespace {

constexpr uint32_t TILE = EXPZ_CHUNK;  // 4096 = 256 threads x 16
constexpr int THREADS = 256;
static_assert(TILE == 16 * THREADS, "a thread holds 16 values of a tile");

// Shared-memory slot of tile value j: the low four bits XORed with the next
// four, so that all three access patterns below are free of bank conflicts.
__device__ __forceinline__ uint32_t zpos(uint32_t j) { return j ^ ((j >> 4) & 15u); }

__device__ __forceinline__ void wht16(double (&x)[16]) {
#pragma unroll
    for (int h = 1; h < 16; h <<= 1)
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (!(i & h)) {
                const double a = x[i], b = x[i | h];
                x[i] = a + b;
                x[i | h] = a - b;
            }
}

// Adds the tile at `base` (a multiple of TILE) to the thread's sums: lane
// group threadIdx.x / 16 + 16 i serves mask mk[i], each lane one value of its
// row.
template <typename T, int MI>
__device__ __forceinline__ void expz_tile(const T* __restrict__ a, uint64_t base, uint64_t len, const uint64_t (&mk)[MI],
                                          double (&acc)[MI], double* sm) {
    const uint32_t t = threadIdx.x;
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const uint64_t i = base + (uint32_t)r * THREADS + t;
        x[r] = i < len ? c_abs2(a[i]) : 0.0;
    }
    wht16(x);  // bits 8..11
    __syncthreads();  // the previous tile's rows have been read
#pragma unroll
    for (int r = 0; r < 16; ++r) sm[zpos((uint32_t)r * THREADS + t)] = x[r];
    __syncthreads();
    const uint32_t j0 = (t >> 4) * 256u + (t & 15u);
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = sm[zpos(j0 + 16u * m)];
    wht16(x);  // bits 4..7
#pragma unroll
    for (int m = 0; m < 16; ++m) sm[zpos(j0 + 16u * m)] = x[m];
    __syncthreads();
    const uint32_t v = t & 15u;
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const double y = sm[zpos(((uint32_t)mk[i] & 0xff0u) + v)];
        acc[i] += (__popcll(base & mk[i]) + __popc((uint32_t)mk[i] & v)) & 1 ? -y : y;
    }
}

__device__ __forceinline__ double sum16(double x) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Masks of one state: partial sums per CTA, added in CTA order by the CTA that
// finishes last (ticket returns to 0 by itself), divided by norm2.
template <typename T, int MI>
__global__ void __launch_bounds__(THREADS, MI <= 4 ? 4 : 2)
k_expz(const T* a, uint64_t len, const __grid_constant__ ExpzMasks M, uint32_t k,
       const double* norm2, double* __restrict__ partials, unsigned int* __restrict__ ticket,
       double* __restrict__ out) {
    grid_go();
    grid_wait();
    __shared__ double sm[TILE];
    __shared__ bool last;
    const uint32_t t = threadIdx.x, g = t >> 4;
    uint64_t mk[MI];
    double acc[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        mk[i] = g + 16u * i < k ? M.m[g + 16u * i] : 0ull;
        acc[i] = 0.0;
    }
    for (uint64_t base = (uint64_t)blockIdx.x * TILE; base < len; base += (uint64_t)gridDim.x * TILE)
        expz_tile(a, base, len, mk, acc, sm);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const double x = sum16(acc[i]);
        if ((t & 15u) == 0 && g + 16u * i < k) partials[(uint64_t)(g + 16u * i) * gridDim.x + blockIdx.x] = x;
    }
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double d = *norm2;
    for (uint32_t s = g; s < ((k + 15u) & ~15u); s += 16u) {
        double x = 0.0;
        if (s < k)
            for (uint32_t b = t & 15u; b < gridDim.x; b += 16u) x += __ldcg(partials + (uint64_t)s * gridDim.x + b);
        x = sum16(x);
        if ((t & 15u) == 0 && s < k) out[s] = d > 1e-12 ? x / d : 0.0;
    }
}

// Arena circuits: one CTA per tile of every circuit; slot mask_count is the
// squared norm (mask 0). Results do not depend on the launch shape: the final
// kernel adds each slot's tiles in a fixed order.
template <typename T, int MI>
__global__ void __launch_bounds__(THREADS, MI <= 4 ? 4 : 2)
k_arena_expz_partials(const ExpzJob* __restrict__ jobs, uint32_t njobs, const uint64_t* __restrict__ masks,
                      double* __restrict__ partials) {
    __shared__ double sm[TILE];
    const uint32_t b = blockIdx.x;
    uint32_t lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (jobs[mid].chunk_start <= b) lo = mid;
        else hi = mid - 1;
    }
    const ExpzJob J = jobs[lo];
    const uint32_t t = threadIdx.x, g = t >> 4, slots = J.mask_count + 1;
    uint64_t mk[MI];
    double acc[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        mk[i] = g + 16u * i < J.mask_count ? masks[J.mask_start + g + 16u * i] : 0ull;
        acc[i] = 0.0;
    }
    const uint64_t c = b - J.chunk_start;
    expz_tile(reinterpret_cast<const T*>(J.amps), c * TILE, 1ull << J.n, mk, acc, sm);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const double x = sum16(acc[i]);
        if ((t & 15u) == 0 && g + 16u * i < slots) partials[J.part_start + c * slots + g + 16u * i] = x;
    }
}

// One CTA per circuit, a warp per slot: lane l adds tiles l, l + 32, ...
__global__ void __launch_bounds__(256) k_arena_expz_final(const ExpzJob* __restrict__ jobs,
                                                          const double* __restrict__ partials, double* __restrict__ out) {
    __shared__ double sums[EXPZ_MAX_MASKS + 1];
    const ExpzJob J = jobs[blockIdx.x];
    const uint32_t slots = J.mask_count + 1;
    const uint32_t tiles = (uint32_t)(((1ull << J.n) + TILE - 1) / TILE);
    for (uint32_t s = threadIdx.x >> 5; s < slots; s += blockDim.x >> 5) {
        double x = 0.0;
        for (uint32_t c = threadIdx.x & 31; c < tiles; c += 32) x += partials[J.part_start + (uint64_t)c * slots + s];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) sums[s] = x;
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < J.mask_count; s += blockDim.x) out[J.out_start + s] = sums[s] / sums[J.mask_count];
}

template <typename T>
cudaError_t expz(const T* a, uint64_t len, const ExpzMasks& M, uint32_t k, const double* norm2, double* partials,
          unsigned int* ticket, double* out, uint32_t blocks, cudaStream_t st) {
    if (k <= 16) return launch_overlapped(k_expz<T, 1>, blocks, THREADS, 0, st, a, len, M, k, norm2, partials, ticket, out);
    if (k <= 64) return launch_overlapped(k_expz<T, 4>, blocks, THREADS, 0, st, a, len, M, k, norm2, partials, ticket, out);
    return launch_overlapped(k_expz<T, 16>, blocks, THREADS, 0, st, a, len, M, k, norm2, partials, ticket, out);
}

template <typename T>
void arena_partials(const ExpzJob* jobs, uint32_t njobs, uint32_t tiles, uint32_t max_masks, const uint64_t* masks,
                    double* partials, cudaStream_t st) {
    if (max_masks < 16) k_arena_expz_partials<T, 1><<<tiles, THREADS, 0, st>>>(jobs, njobs, masks, partials);
    else if (max_masks < 64) k_arena_expz_partials<T, 4><<<tiles, THREADS, 0, st>>>(jobs, njobs, masks, partials);
    else k_arena_expz_partials<T, 16><<<tiles, THREADS, 0, st>>>(jobs, njobs, masks, partials);
}

}  // namespace

// CTAs of the sweep: the tiles, or four for each of 148 SMs: resident at once
// up to 64 masks, in two waves above (two CTAs an SM, 128 registers).
uint32_t expz_blocks(uint64_t len) {
    const uint64_t tiles = (len + TILE - 1) / TILE;
    return (uint32_t)(tiles < 148 * 4 ? tiles : 148 * 4);
}

// k <= EXPZ_MASKS masks; partials: k * expz_blocks(len) doubles
cudaError_t launch_expz(const void* a, bool f32, uint64_t len, const ExpzMasks& M, uint32_t k, const double* norm2,
                        double* partials, unsigned int* ticket, double* out, cudaStream_t st) {
    if (k > EXPZ_MASKS) return cudaErrorInvalidValue;
    const uint32_t blocks = expz_blocks(len);
    return f32 ? expz((const float2*)a, len, M, k, norm2, partials, ticket, out, blocks, st)
               : expz((const double2*)a, len, M, k, norm2, partials, ticket, out, blocks, st);
}

cudaError_t launch_arena_expz(bool f32, const ExpzJob* jobs, uint32_t njobs, uint32_t chunks, uint32_t max_masks,
                              const uint64_t* masks, double* partials, double* out, cudaStream_t st) {
    if (!njobs) return cudaSuccess;
    if (f32) arena_partials<float2>(jobs, njobs, chunks, max_masks, masks, partials, st);
    else arena_partials<double2>(jobs, njobs, chunks, max_masks, masks, partials, st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_arena_expz_final<<<njobs, 256, 0, st>>>(jobs, partials, out);
    return cudaGetLastError();
}

}  // namespace qoa
