// qoa_small.cu — small states whole in one CTA's shared memory.
//
// A circuit is a list of sweeps (made by small_program in qoa_engine.cpp). A sweep names three qubits; each thread takes the 8
// amplitudes that differ in them into registers, applies the sweep's gates
// there — 2x2 gates on the three, diagonal gates anywhere — and puts them
// back; one barrier a sweep. Two kernels run them: k_small_state, one launch
// for a handle's op list, and k_small_batch, a persistent launch over many
// circuits, each starting in |0..0> and reduced to its Z strings in place.
//
// What bounds it: latency. A sweep is a shared-memory round trip and a
// barrier (~150 cycles), a gate ~40-100 cycles of FP64 and of reading its
// record; the state never leaves the SM. Three register qubits: a fourth
// would halve the sweeps of a layer but also the threads (2^n / 16), and
// states of up to 10 qubits have too few of those already. Gate records come
// from shared memory: read from global memory they cost ~600 cycles each.
// Diagonal gates are collected by the host, as one table over the register
// qubits and one factor per thread (58 -> 41 us for 10 qubits, 233 gates).
// Measured on B200, op lists on a handle against a launch per gate: 6 qubits,
// 61 gates 192 -> 48 us with the state read back; 10 qubits, 117 gates and 19
// Z strings 439 -> 61 us; against tile passes of one or two CTAs: 11 qubits,
// 258 gates 119 -> 79 us (complex64), 12 qubits 109 gates 54 -> 52 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdint.h>

#include "qoa_kernels.cuh"
#include "qoa_launch.cuh"
#include "qoa_pass_dev.cuh"

namespace qoa {

namespace {

// Shared-memory slot of amplitude i: the low three bits XORed with the folds
// of the others (linear), so that any three register qubits with distinct
// residues mod 3 leave a quarter-warp's 16-byte accesses free of conflicts.
__device__ __forceinline__ uint32_t small_pos(uint32_t i) {
    return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9) ^ (i >> 12)) & 7u);
}

template <int SUB, int K, typename T>
__device__ __forceinline__ void small_g1k(T (&a)[8], const double2* __restrict__ m) {
    const T z = CT<T>::mk(0, 0);
    const T m0 = CT<T>::from(m[0]);
    const T m1 = SUB == G1_GEN ? CT<T>::from(m[1]) : z, m2 = SUB == G1_GEN ? CT<T>::from(m[2]) : z,
            m3 = SUB == G1_GEN ? CT<T>::from(m[3]) : z;
#pragma unroll
    for (int v = 0; v < 8; ++v)
        if (!(v & (1 << K))) g1_pair<SUB>(a[v], a[v | (1 << K)], m0, m1, m2, m3);
}
template <int SUB, typename T>
__device__ __forceinline__ void small_g1(T (&a)[8], uint32_t k, const double2* __restrict__ m) {
    if (k == 0) small_g1k<SUB, 0>(a, m);
    else if (k == 1) small_g1k<SUB, 1>(a, m);
    else small_g1k<SUB, 2>(a, m);
}

// X / Y where the register-bit conditions cl hold (never the target's bit)
template <int SUB, int K, typename T>
__device__ __forceinline__ void small_xyk(T (&a)[8], uint32_t cl) {
    const T z = CT<T>::mk(0, 0);
#pragma unroll
    for (int v = 0; v < 8; ++v)
        if (!(v & (1 << K)) && ((uint32_t)v & cl) == cl) g1_pair<SUB>(a[v], a[v | (1 << K)], z, z, z, z);
}
template <int SUB, typename T>
__device__ __forceinline__ void small_xy(T (&a)[8], uint32_t k, uint32_t cl) {
    if (k == 0) small_xyk<SUB, 0>(a, cl);
    else if (k == 1) small_xyk<SUB, 1>(a, cl);
    else small_xyk<SUB, 2>(a, cl);
}

// 4x4 on register bits L < H: basis 2 * bit(H) + bit(L)
template <int L, int H, typename T>
__device__ __forceinline__ void small_u2(T (&a)[8], const double2* __restrict__ m) {
#pragma unroll
    for (int v = 0; v < 8; ++v)
        if (!(v & ((1 << L) | (1 << H)))) {
            T x[4] = {a[v], a[v | (1 << L)], a[v | (1 << H)], a[v | (1 << L) | (1 << H)]};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                T acc = c_mul(CT<T>::from(m[4 * r]), x[0]);
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    const T c = CT<T>::from(m[4 * r + k]);
                    acc.x = fma(c.x, x[k].x, acc.x); acc.x = fma(-c.y, x[k].y, acc.x);
                    acc.y = fma(c.x, x[k].y, acc.y); acc.y = fma(c.y, x[k].x, acc.y);
                }
                a[v | ((r & 1) << L) | ((r >> 1) << H)] = acc;
            }
        }
}

// One gate on a thread's 8 amplitudes; i0: their index with the register
// qubits 0; pend: the thread's phase. k: register bit (or register-bit pair); cl: register-bit
// conditions; co: conditions on the other qubits.
template <typename T>
__device__ __forceinline__ void small_gate(T (&a)[8], T& pend, uint32_t i0, const SmallOp op, const double2* __restrict__ coef) {
    if ((i0 & op.co) != op.co) return;
    const double2* m = coef + op.coef;
    const uint32_t k = op.k & 15u, cl = op.k >> 4;
    switch (op.code) {
        case SO_H: small_g1<G1_H>(a, k, m); break;
        case SO_RX: small_g1<G1_RX>(a, k, m); break;
        case SO_RY: small_g1<G1_RY>(a, k, m); break;
        case SO_GEN: small_g1<G1_GEN>(a, k, m); break;
        case SO_X: small_xy<G1_X>(a, k, cl); break;
        case SO_Y: small_xy<G1_Y>(a, k, cl); break;
        case SO_NEG:
#pragma unroll
            for (int v = 0; v < 8; ++v)
                if (((uint32_t)v & cl) == cl) a[v] = c_neg(a[v]);
            break;
        case SO_DIAG: {
            const T d = CT<T>::from(m[0]);
#pragma unroll
            for (int v = 0; v < 8; ++v)
                if (((uint32_t)v & cl) == cl) a[v] = c_mul(a[v], d);
            break;
        }
        case SO_SELR: {  // factor by register bit k
            const T d0 = CT<T>::from(m[0]), d1 = CT<T>::from(m[1]);
#pragma unroll
            for (int v = 0; v < 8; ++v)
                if (((uint32_t)v & cl) == cl) a[v] = c_mul(a[v], ((v >> k) & 1) ? d1 : d0);
            break;
        }
        case SO_TAB:
#pragma unroll
            for (int v = 0; v < 8; ++v) a[v] = c_mul(a[v], CT<T>::from(m[v]));
            break;
        case SO_PNEG: pend = c_neg(pend); break;
        case SO_PDIAG: pend = c_mul(pend, CT<T>::from(m[0])); break;
        case SO_PSEL: pend = c_mul(pend, CT<T>::from(m[(i0 >> k) & 1u])); break;
        case SO_U2:
            if (k == 0) small_u2<0, 1>(a, m);
            else if (k == 1) small_u2<0, 2>(a, m);
            else small_u2<1, 2>(a, m);
            break;
        default: break;
    }
}

// Copies chunk r of ops and coef into shared memory (16-byte words).
__device__ __forceinline__ void small_stage(SmallChunk* dst, const SmallChunkRef r, const SmallOp* ops, const double2* coef) {
    const uint4* so = reinterpret_cast<const uint4*>(ops + r.op_start);
    uint4* po = reinterpret_cast<uint4*>(dst->ops);
    for (uint32_t i = threadIdx.x; i < (r.nops + 1) / 2; i += blockDim.x) po[i] = so[i];
    for (uint32_t i = threadIdx.x; i < r.ncoef; i += blockDim.x) dst->coef[i] = coef[r.coef_start + i];
    __syncthreads();
}

// The sweeps of a staged chunk on the state s of n qubits (at least 2^3 slots).
template <typename T>
__device__ __forceinline__ void small_sweeps(T* s, uint32_t n, const SmallChunk* c, uint32_t nops) {
    const uint32_t groups = n > 3 ? 1u << (n - 3) : 1u;
    for (uint32_t oi = 0; oi < nops;) {
        const SmallOp sw = c->ops[oi];
        const uint32_t cnt = sw.coef, q0 = sw.co & 255u, q1 = (sw.co >> 8) & 255u, q2 = (sw.co >> 16) & 255u;
        const uint32_t p0 = small_pos(1u << q0), p1 = small_pos(1u << q1), p2 = small_pos(1u << q2);
        for (uint32_t p = threadIdx.x; p < groups; p += blockDim.x) {
            uint32_t i0 = ((p >> q0) << (q0 + 1)) | (p & ((1u << q0) - 1));
            i0 = ((i0 >> q1) << (q1 + 1)) | (i0 & ((1u << q1) - 1));
            i0 = ((i0 >> q2) << (q2 + 1)) | (i0 & ((1u << q2) - 1));
            const uint32_t b = small_pos(i0);
            T a[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) a[v] = s[b ^ ((v & 1) ? p0 : 0u) ^ ((v & 2) ? p1 : 0u) ^ ((v & 4) ? p2 : 0u)];
            T pend = CT<T>::mk(1, 0);
            for (uint32_t e = 1; e <= cnt; ++e) small_gate(a, pend, i0, c->ops[oi + e], c->coef);
            if (sw.k) {
#pragma unroll
                for (int v = 0; v < 8; ++v) a[v] = c_mul(a[v], pend);
            }
#pragma unroll
            for (int v = 0; v < 8; ++v) s[b ^ ((v & 1) ? p0 : 0u) ^ ((v & 2) ? p1 : 0u) ^ ((v & 4) ? p2 : 0u)] = a[v];
        }
        oi += 1 + cnt;
        __syncthreads();
    }
}

// A handle's op list: the state in (scaled by the pending 1/||psi||, or
// |0..0>), the sweeps, the state and its squared norm out.
template <typename T, int NC>
__global__ void __launch_bounds__(512) k_small_state(T* __restrict__ amps, uint32_t n, const double* __restrict__ norm2_in,
                                                     const __grid_constant__ SmallProgram<NC> P, double* __restrict__ norm2,
                                                     uint32_t* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    __shared__ double red[16];
    SmallChunk* c = reinterpret_cast<SmallChunk*>(small_smem);
    T* s = reinterpret_cast<T*>(small_smem + sizeof(SmallChunk));
    using R = typename CT<T>::R;
    const uint32_t len = 1u << n, slots = len < 8 ? 8 : len;
    grid_go();
    small_stage(c, P.ref[0], P.ops, P.coef);  // while the kernel before finishes
    grid_wait();
    const double nrm = read_after_wait(norm2_in);
    const bool valid = nrm > 1e-12;
    const R scale = valid ? (R)(1.0 / sqrt(nrm)) : (R)0;
    for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) {
        T x = CT<T>::mk(!valid && i == 0 ? (R)1 : (R)0, (R)0);
        if (valid && i < len) {
            x = amps[i];
            x = CT<T>::mk(x.x * scale, x.y * scale);
        }
        s[small_pos(i)] = x;
    }
    __syncthreads();
    for (uint32_t k = 0; k < P.nchunks; ++k) {
        if (k) small_stage(c, P.ref[k], P.ops, P.coef);
        small_sweeps(s, n, c, P.ref[k].nops);
    }
    double ss = 0.0;
    for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
        const T x = s[small_pos(i)];
        amps[i] = x;
        ss += c_abs2(x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
        *norm2 = t;
        if (t != t) atomicOr(&status[0], 1u);
        if (!(t > 1e-12)) atomicAdd(&status[2], 1u);
    }
}

template <typename T>
__global__ void k_small_batch(const SmallCircuit* __restrict__ circs, uint32_t count, const SmallChunkRef* __restrict__ chunks,
                              const SmallOp* __restrict__ ops, const double2* __restrict__ coef,
                              const uint64_t* __restrict__ masks, double* __restrict__ out,
                              unsigned int* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char small_smem[];
    SmallChunk* ch = reinterpret_cast<SmallChunk*>(small_smem);
    T* s = reinterpret_cast<T*>(small_smem + sizeof(SmallChunk));
    __shared__ uint32_t cidx;
    __shared__ double red[8 + 1][32];
    using R = typename CT<T>::R;
    while (true) {
        if (threadIdx.x == 0) cidx = atomicAdd(counter, 1u);
        __syncthreads();
        const uint32_t c = cidx;
        __syncthreads();
        if (c >= count) break;
        const SmallCircuit ci = circs[c];
        const uint32_t len = 1u << ci.n, slots = len < 8 ? 8 : len;
        for (uint32_t i = threadIdx.x; i < slots; i += blockDim.x) s[small_pos(i)] = CT<T>::mk(i == 0 ? (R)1 : (R)0, (R)0);
        for (uint32_t k = 0; k < ci.chunk_count; ++k) {
            const SmallChunkRef r = chunks[ci.chunk_start + k];
            small_stage(ch, r, ops, coef);
            small_sweeps(s, ci.n, ch, r.nops);
        }
        __syncthreads();
        if (ci.state_out)  // sampled after the run: the state goes to HBM
            for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) reinterpret_cast<T*>(ci.state_out)[i] = s[small_pos(i)];
        // <Z_mask> of the normalised state, 8 masks per sweep
        for (uint32_t m0 = 0; m0 < ci.mask_count; m0 += 8) {
            double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            uint32_t mk[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) mk[q] = (m0 + q < ci.mask_count) ? (uint32_t)masks[ci.mask_start + m0 + q] : 0;
            for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
                const T a = s[small_pos(i)];
                const double p = (double)a.x * a.x + (double)a.y * a.y;
                v[8] += p;
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] += (__popc(i & mk[q]) & 1) ? -p : p;
            }
            const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
            for (int q = 0; q < 9; ++q) {
                double x = v[q];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0) red[q][w] = x;
            }
            __syncthreads();
            if (threadIdx.x < 8 && m0 + threadIdx.x < ci.mask_count) {
                double t = 0.0, nrm = 0.0;
                for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { t += red[threadIdx.x][k]; nrm += red[8][k]; }
                out[ci.out_start + m0 + threadIdx.x] = t / nrm;
            }
            __syncthreads();
        }
    }
}

template <typename T>
size_t small_smem_bytes(uint32_t n) {
    return sizeof(SmallChunk) + (sizeof(T) << std::max<uint32_t>(n, 3));
}

template <typename T, int NC>
cudaError_t small_state(T* amps, uint32_t n, const double* norm2_in, const SmallProgram<NC>& P, double* norm2,
                        uint32_t* status, cudaStream_t st) {
    // the attribute allows the largest state, the same for every call (handles on several threads launch it)
    const cudaError_t e = cudaFuncSetAttribute(k_small_state<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)small_smem_bytes<T>(SMALL_STATE_MAX));
    if (e != cudaSuccess) return e;
    const uint32_t groups = n > 3 ? 1u << (n - 3) : 1u;
    const uint32_t threads = std::min(512u, std::max(32u, groups));
    return launch_overlapped(k_small_state<T, NC>, 1, threads, small_smem_bytes<T>(n), st, amps, n, norm2_in, P, norm2, status);
}

}  // namespace

template <int NC>
cudaError_t launch_small_state(void* amps, bool f32, uint32_t n, const double* norm2_in, const SmallProgram<NC>& P,
                               double* norm2, uint32_t* status, cudaStream_t st) {
    if (n > SMALL_STATE_MAX) return cudaErrorInvalidValue;
    return f32 ? small_state((float2*)amps, n, norm2_in, P, norm2, status, st)
               : small_state((double2*)amps, n, norm2_in, P, norm2, status, st);
}
template cudaError_t launch_small_state(void*, bool, uint32_t, const double*, const SmallProgram<1>&, double*, uint32_t*,
                                        cudaStream_t);
template cudaError_t launch_small_state(void*, bool, uint32_t, const double*, const SmallProgram<3>&, double*, uint32_t*,
                                        cudaStream_t);

cudaError_t launch_small_batch(bool f32, const SmallCircuit* circs, uint32_t count, const SmallChunkRef* chunks,
                               const SmallOp* ops, const double2* coef, const uint64_t* masks, double* out, unsigned int* counter, int max_n, int threads,
                               int ctas_per_sm, cudaStream_t st) {
    const size_t smem = f32 ? small_smem_bytes<float2>(max_n) : small_smem_bytes<double2>(max_n);
    // the attribute allows the largest state the kernel takes, the same for
    // every call: batches prepared on several host threads (the server's
    // workers) launch it concurrently with different sizes, and a smaller
    // setting made between another thread's set-up and launch fails that launch
    const size_t smem_cap = f32 ? small_smem_bytes<float2>(SMALL_MAX_F32) : small_smem_bytes<double2>(SMALL_MAX_F64);
    if (smem > smem_cap) return cudaErrorInvalidValue;
    // The tuning takes blocks of up to 1024 threads, the registers of a sweep
    // fewer (100 a thread in complex128: 640 do not fit); the loops stride by the block.
    // A launch bound instead would change the code for every block (512: 79 ->
    // 107 registers in complex64).
    cudaFuncAttributes fa;
    cudaError_t e = f32 ? cudaFuncGetAttributes(&fa, k_small_batch<float2>) : cudaFuncGetAttributes(&fa, k_small_batch<double2>);
    if (e != cudaSuccess) return e;
    threads = std::min(threads, fa.maxThreadsPerBlock & ~31);
    if (f32) e = cudaFuncSetAttribute(k_small_batch<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cap);
    else e = cudaFuncSetAttribute(k_small_batch<double2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cap);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(counter, 0, sizeof(unsigned int), st);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    unsigned grid = (unsigned)(sms * ctas_per_sm);
    if (grid > count) grid = count ? count : 1;
    if (f32) k_small_batch<float2><<<grid, threads, smem, st>>>(circs, count, chunks, ops, coef, masks, out, counter);
    else k_small_batch<double2><<<grid, threads, smem, st>>>(circs, count, chunks, ops, coef, masks, out, counter);
    return cudaGetLastError();
}

}  // namespace qoa
