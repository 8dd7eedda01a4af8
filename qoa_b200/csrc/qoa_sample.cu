// qoa_sample.cu — shots of a state: a radix marginal tree and one warp per shot.
//
// h_k[p] = sum over i with i mod 2^k == p of |a_i|^2 (the marginal of qubits
// 0..k-1) is what a shot walks from k = 0 to k = n. Only a few levels are
// stored (sample_levels): the state is read once into level K_1 = n - b_1,
// level K_2 = K_1 - b_2 comes from it, and so on down to at most 8 bits. A
// shot is one warp: at each stored level it gathers the up to 2^8 values
// below its prefix, folds them into the levels in between and walks those.
// Every sum pairs the top bit of its index first, at every level, whichever
// levels are stored, so a shot does not depend on the split.
//
// What bounds it: reading the state once (the fold of the amplitudes), and
// for small states the launches: 1 + ceil((n - 8) / 6) of them, where a
// level-by-level tree takes n. The stored levels take 1/64 (complex128) of
// the state instead of half of it. Measured on B200, a whole circuit with its
// shots, against level-by-level trees in scratch mapped on each call: 20
// qubits 3.3 -> 1.5 ms, 27 qubits 39.8 -> 24.1 ms, 29 qubits (complex64 QFT)
// 78.5 -> 19.9 ms.
#include <cuda_runtime.h>

#include <stdint.h>

#include "qoa_kernels.cuh"
#include "qoa_launch.cuh"
#include "qoa_pass_dev.cuh"

namespace qoa {

namespace {

constexpr uint32_t ROOT_BITS = 8;  // a warp's gather: 8 values a lane

// value j of a level: the amplitudes themselves, or a stored level
template <typename T>
struct AmpSrc {
    const T* a;
    double inv;
    bool valid;  // false: the logical state is |0..0>
    __device__ __forceinline__ double raw(uint64_t i) const {
        return valid ? c_abs2(a[i]) : (i == 0 ? 1.0 : 0.0);
    }
};

template <typename T>
__device__ __forceinline__ AmpSrc<T> amp_src(const T* a, const double* norm2) {
    const double nrm = read_after_wait(norm2);
    const bool valid = nrm > 1e-12;
    return AmpSrc<T>{a, valid ? 1.0 / nrm : 1.0, valid};
}

// Sum over j < 2^B of the values p + (j << lo), top bit of j paired first.
// From amplitudes, 1/norm2 is applied to the sums of two (level n - 1).
template <int B, int K, bool AMPS, typename S>
__device__ __forceinline__ double fold(const S& s, uint64_t p, uint32_t lo, uint32_t j) {
    if constexpr (K == B) {
        const uint64_t i = p + ((uint64_t)j << lo);
        if constexpr (AMPS) return s.raw(i);
        else return s[i];
    } else {
        const double x = fold<B, K + 1, AMPS>(s, p, lo, j) + fold<B, K + 1, AMPS>(s, p, lo, j + (1u << K));
        if constexpr (AMPS && K == B - 1) return x * s.inv;
        return x;
    }
}

template <int B, typename T>
__global__ void __launch_bounds__(128) k_fold_amps(const T* a, const double* norm2, uint32_t lo,
                                                   double* __restrict__ out) {
    grid_go();
    grid_wait();
    const AmpSrc<T> s = amp_src(a, norm2);
    const uint64_t cnt = 1ull << lo;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < cnt; p += (uint64_t)gridDim.x * blockDim.x)
        out[p] = fold<B, 0, true>(s, p, lo, 0);
}

template <int B>
__global__ void __launch_bounds__(128) k_fold_level(const double* in, uint32_t lo, double* __restrict__ out) {
    grid_go();
    grid_wait();
    const uint64_t cnt = 1ull << lo;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < cnt; p += (uint64_t)gridDim.x * blockDim.x)
        out[p] = fold<B, 0, false>(in, p, lo, 0);
}

// The levels between a prefix and the 2^b values below it, in one warp:
// lane l of v[r] holds value l + 32 r; x[k] holds level k (k <= 5) with
// value j on every lane l = j mod 2^k.
struct WarpTree {
    double v8[8], v7[4], v6[2], x[6];

    // v8[0 .. 2^(b-5)-1] loaded (b <= 5: v8[0] on lanes < 2^b). `leaf`: the
    // values are raw squares, scaled by inv once a level is a sum of two.
    __device__ __forceinline__ void build(uint32_t b, bool leaf, double inv) {
        const uint32_t full = 0xffffffffu;
        double s = leaf ? inv : 1.0;  // scale still owed by the next sum
        if (b == 8) {
#pragma unroll
            for (int r = 0; r < 4; ++r) v7[r] = (v8[r] + v8[r + 4]) * s;
            s = 1.0;
        } else if (b == 7) {
#pragma unroll
            for (int r = 0; r < 4; ++r) v7[r] = v8[r];
        }
        if (b >= 7) {
#pragma unroll
            for (int r = 0; r < 2; ++r) v6[r] = (v7[r] + v7[r + 2]) * s;
            s = 1.0;
        } else if (b == 6) {
            v6[0] = v8[0];
            v6[1] = v8[1];
        }
        if (b >= 6) {
            x[5] = (v6[0] + v6[1]) * s;
            s = 1.0;
        } else {
            x[5] = v8[0];  // b <= 5: level b's values (lanes < 2^b), copied down below
        }
#pragma unroll
        for (int k = 4; k >= 0; --k) {
            if ((uint32_t)k >= b) {
                x[k] = x[k + 1];
            } else {
                x[k] = (x[k + 1] + __shfl_xor_sync(full, x[k + 1], 1 << k)) * s;
                s = 1.0;
            }
        }
        if (leaf) {  // the values themselves as probabilities (level n)
#pragma unroll
            for (int r = 0; r < 8; ++r) v8[r] *= inv;
            if (b == 7) {
#pragma unroll
                for (int r = 0; r < 4; ++r) v7[r] *= inv;
            } else if (b == 6) {
                v6[0] *= inv;
                v6[1] *= inv;
            } else if (b <= 5) {
#pragma unroll
                for (int k = 0; k < 6; ++k)
                    if ((uint32_t)k >= b) x[k] *= inv;
            }
        }
    }
    // value j of level k, the same on every lane (j and k are)
    __device__ __forceinline__ double at(uint32_t k, uint32_t j) const {
        double y = x[0];
#pragma unroll
        for (int i = 1; i < 6; ++i)
            if (k == (uint32_t)i) y = x[i];
        const uint32_t r = j >> 5;
        if (k == 6) y = r ? v6[1] : v6[0];
        if (k == 7) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (r == (uint32_t)i) y = v7[i];
        }
        if (k == 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (r == (uint32_t)i) y = v8[i];
        }
        return __shfl_sync(0xffffffffu, y, (int)(j & 31u));
    }
};

// One warp per shot. mode 0: the measure_all order of the reference — qubit
// q measured with uniform u[shot*n + q] as `u < P0`, where P0 is the
// conditional probability given the earlier outcomes; a branch with
// probability <= 1e-12 zeroes the state, which normalize() then resets to
// |0..0>, so every later outcome is 0 (quantum_state.rs:424-455, 888-907).
// mode 1: inverse CDF with one uniform per shot, walking the same tree.
template <typename T>
__global__ void __launch_bounds__(128) k_shots(const T* a, uint32_t n, const double* norm2,
                                               const double* tree, const SampleLevels L,
                                               const double* __restrict__ u, uint64_t shots, int mode,
                                               unsigned long long* __restrict__ out) {
    grid_go();
    grid_wait();
    const AmpSrc<T> src = amp_src(a, norm2);
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < shots; s += nw) {
        double ua = 0.0, ub = 0.0;  // this shot's uniforms: mode 0 lane q (and q - 32), mode 1 all lanes
        if (mode == 0) {
            if (lane < n) ua = u[s * n + lane];
            if (lane + 32 < n) ub = u[s * n + 32 + lane];
        } else {
            ua = u[s];
        }
        uint64_t pre = 0;
        uint32_t q = 0;
        bool dead = false;
        double t = 0.0;
        for (int st = 0; st <= (int)L.count && !dead; ++st) {
            const uint32_t to = st < (int)L.count ? L.bits[L.count - 1 - st] : n;
            const uint32_t b = to - q;
            const bool leaf = to == n;
            const double* lv = leaf ? nullptr : tree + L.off[L.count - 1 - st];
            WarpTree w;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint32_t j = lane + 32u * r;
                w.v8[r] = 0.0;
                if (j < (1u << b)) {
                    const uint64_t i = pre | ((uint64_t)j << q);
                    w.v8[r] = leaf ? src.raw(i) : lv[i];
                }
            }
            w.build(b, leaf, src.inv);
            if (st == 0 && mode != 0) t = ua * w.at(0, 0);
            uint32_t loc = 0;
            for (uint32_t k = 0; k < b; ++k) {
                const double left = w.at(k + 1, loc);
                uint32_t bit;
                if (mode == 0) {
                    const uint32_t qq = q + k;
                    const double x = qq < 32 ? ua : ub;
                    const double uq = __shfl_sync(0xffffffffu, x, (int)(qq & 31u));
                    const double tot = w.at(k, loc);
                    const double p0 = left / tot;
                    bit = (uq < p0) ? 0u : 1u;
                    const double pb = bit ? w.at(k + 1, loc | (1u << k)) / tot : p0;
                    loc |= bit << k;
                    if (!(pb > 1e-12)) {
                        dead = true;
                        break;
                    }
                } else {
                    bit = (t < left) ? 0u : 1u;
                    if (bit) t -= left;
                    loc |= bit << k;
                }
            }
            pre |= (uint64_t)loc << q;
            q = to;
        }
        if (lane == 0) out[s] = pre;
    }
}

int fold_grid(uint32_t lo) {
    const uint64_t b = ((1ull << lo) + 127) / 128;
    return (int)(b < 148 * 16 ? b : 148 * 16);
}

}  // namespace

// The stored levels of an n-qubit state's tree, the largest first: n - 8
// bits split evenly into steps, the root step takes 8. Steps of at most 4 bits
// (16 loads a thread) up to 22 qubits, where 6-bit steps leave too few threads
// (20 qubits: 26 + 10 us in two launches), of 6 above, where fewer launches
// and 1/64 of the state of scratch count.
SampleLevels sample_levels(uint32_t n) {
    SampleLevels L{};
    const uint32_t step = n <= 22 ? 4 : 6;
    uint32_t rest = n > ROOT_BITS ? n - ROOT_BITS : 0, at = n;
    uint64_t off = 0;
    for (uint32_t steps = (rest + step - 1) / step; steps; --steps) {
        const uint32_t b = (rest + steps - 1) / steps;
        rest -= b;
        at -= b;
        L.bits[L.count] = at;
        L.off[L.count++] = off;
        off += 1ull << at;
    }
    L.total = off;
    return L;
}

template <typename T>
static cudaError_t fold_amps(const T* a, const double* norm2, uint32_t b, uint32_t lo, double* out, cudaStream_t st) {
    const int g = fold_grid(lo);
    switch (b) {
        case 1: return launch_overlapped(k_fold_amps<1, T>, g, 128, 0, st, a, norm2, lo, out);
        case 2: return launch_overlapped(k_fold_amps<2, T>, g, 128, 0, st, a, norm2, lo, out);
        case 3: return launch_overlapped(k_fold_amps<3, T>, g, 128, 0, st, a, norm2, lo, out);
        case 4: return launch_overlapped(k_fold_amps<4, T>, g, 128, 0, st, a, norm2, lo, out);
        case 5: return launch_overlapped(k_fold_amps<5, T>, g, 128, 0, st, a, norm2, lo, out);
        default: return launch_overlapped(k_fold_amps<6, T>, g, 128, 0, st, a, norm2, lo, out);
    }
}

cudaError_t launch_sample_tree(const void* a, bool f32, uint32_t n, const double* norm2, const SampleLevels& L, double* tree,
                               cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (uint32_t k = 0; k < L.count; ++k) {
        const uint32_t lo = L.bits[k];
        double* out = tree + L.off[k];
        if (k == 0) {
            e = f32 ? fold_amps((const float2*)a, norm2, n - lo, lo, out, st)
                    : fold_amps((const double2*)a, norm2, n - lo, lo, out, st);
            if (e != cudaSuccess) return e;
            continue;
        }
        const double* in = tree + L.off[k - 1];
        const int g = fold_grid(lo);
        switch (L.bits[k - 1] - lo) {
            case 1: e = launch_overlapped(k_fold_level<1>, g, 128, 0, st, in, lo, out); break;
            case 2: e = launch_overlapped(k_fold_level<2>, g, 128, 0, st, in, lo, out); break;
            case 3: e = launch_overlapped(k_fold_level<3>, g, 128, 0, st, in, lo, out); break;
            case 4: e = launch_overlapped(k_fold_level<4>, g, 128, 0, st, in, lo, out); break;
            case 5: e = launch_overlapped(k_fold_level<5>, g, 128, 0, st, in, lo, out); break;
            default: e = launch_overlapped(k_fold_level<6>, g, 128, 0, st, in, lo, out); break;
        }
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_shots(const void* a, bool f32, uint32_t n, const double* norm2, const double* tree, const SampleLevels& L,
                         const double* u, uint64_t shots, int mode, unsigned long long* out, cudaStream_t st) {
    const uint64_t blocks = (shots + 3) / 4;
    const int g = (int)(blocks < 148 * 16 ? blocks : 148 * 16);
    if (f32) return launch_overlapped(k_shots<float2>, g, 128, 0, st, (const float2*)a, n, norm2, tree, L, u, shots, mode, out);
    return launch_overlapped(k_shots<double2>, g, 128, 0, st, (const double2*)a, n, norm2, tree, L, u, shots, mode, out);
}

}  // namespace qoa
