// qoa_sample.cu — shots of a state: a radix marginal tree and one warp per shot.
//
// h_k[p] = sum over i with i mod 2^k == p of |a_i|^2 (the marginal of qubits
// 0..k-1) is what a shot walks from k = 0 to k = n. Only a few levels are
// stored (sample_levels): the state is read once into level K_1 = n - b_1,
// level K_2 = K_1 - b_2 comes from it, and so on down to at most 8 bits. A
// shot is one warp: at each stored level it gathers the up to 2^8 values
// below its prefix, folds them into the levels in between and walks those.
// Every sum pairs the top bit of its index first, at every level, whichever
// levels are stored, so a shot does not depend on the split. Where shots are
// many (sample_all_levels) the same folds store every level they pass, and a
// thread walks a shot.
//
// What bounds it: reading the state once (the fold of the amplitudes), and
// for small states the launches: up to 22 qubits 1 + ceil((n - 8) / 4) of them
// (steps of at most 4 bits), above 1 + ceil((n - 8) / 6), where a
// level-by-level tree takes n. The stored levels take 8 bytes for every 2^step
// amplitudes and a little more: 1/128 of a complex128 state with steps of 6
// bits, 1/32 with steps of 4. Measured on B200, a whole circuit with its shots,
// against level-by-level trees in scratch mapped on each call: 20 qubits 3.3 ->
// 1.5 ms, 27 qubits 39.8 -> 24.1 ms, 29 qubits (complex64 QFT) 78.5 -> 19.9 ms.
#include <cuda_runtime.h>

#include <algorithm>
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

// Offset of level k (1 <= k < n) in a tree of all levels.
__host__ __device__ __forceinline__ uint64_t level_at(uint32_t k) { return (1ull << k) - 2; }

// Sum over j < 2^B of the values p + (j << lo), top bit of j paired first.
// From amplitudes, 1/norm2 is applied to the sums of two (level n - 1). ALL:
// every sum on the way is a value of a level in between and goes to the tree
// of all levels at `out`; else the sum goes to out[p].
template <int B, int K, bool AMPS, bool ALL, typename S>
__device__ __forceinline__ double fold(const S& s, uint64_t p, uint32_t lo, uint32_t j, double* out) {
    if constexpr (K == B) {
        const uint64_t i = p + ((uint64_t)j << lo);
        if constexpr (AMPS) return s.raw(i);
        else return s[i];
    } else {
        double x = fold<B, K + 1, AMPS, ALL>(s, p, lo, j, out) + fold<B, K + 1, AMPS, ALL>(s, p, lo, j + (1u << K), out);
        if constexpr (AMPS && K == B - 1) x = x * s.inv;
        if constexpr (ALL) out[level_at(lo + K) + p + ((uint64_t)j << lo)] = x;
        else if constexpr (K == 0) out[p] = x;
        return x;
    }
}

template <int B, bool ALL, typename T>
__global__ void __launch_bounds__(128) k_fold_amps(const T* a, const double* norm2, uint32_t lo, double* out) {
    grid_go();
    grid_wait();
    const AmpSrc<T> s = amp_src(a, norm2);
    const uint64_t cnt = 1ull << lo;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < cnt; p += (uint64_t)gridDim.x * blockDim.x)
        fold<B, 0, true, ALL>(s, p, lo, 0, out);
}

template <int B, bool ALL>
__global__ void __launch_bounds__(128) k_fold_level(const double* in, uint32_t lo, double* out) {
    grid_go();
    grid_wait();
    const uint64_t cnt = 1ull << lo;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < cnt; p += (uint64_t)gridDim.x * blockDim.x)
        fold<B, 0, false, ALL>(in, p, lo, 0, out);
}

// The lowest levels of a tree of all levels: from level ROOT_BITS (n above
// it), or from the amplitudes, down to level 1.
template <typename T>
__global__ void __launch_bounds__(128) k_tree_root(const T* a, uint32_t n, const double* norm2, double* tree) {
    grid_go();
    grid_wait();
    __shared__ double s[1 << ROOT_BITS];
    uint32_t k;
    if (n > ROOT_BITS) {
        k = ROOT_BITS;
        for (uint32_t p = threadIdx.x; p < (1u << k); p += blockDim.x) s[p] = tree[level_at(k) + p];
    } else {
        const AmpSrc<T> src = amp_src(a, norm2);
        k = n - 1;
        for (uint32_t p = threadIdx.x; p < (1u << k); p += blockDim.x)
            tree[level_at(k) + p] = s[p] = (src.raw(p) + src.raw(p + (1u << k))) * src.inv;
    }
    while (--k >= 1) {
        __syncthreads();
        const uint32_t p = threadIdx.x, h = 1u << k;
        if (p < h) tree[level_at(k) + p] = s[p] = s[p] + s[p + h];
    }
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

// One thread per shot on a tree of all levels: n dependent loads, and shots
// beside one another hide them. The same sums and the same walk as k_shots.
template <typename T>
__global__ void __launch_bounds__(128) k_shots_tree(const T* a, uint32_t n, const double* norm2, const double* tree,
                                                    const double* __restrict__ u, uint64_t shots, int mode,
                                                    unsigned long long* __restrict__ out) {
    grid_go();
    grid_wait();
    const AmpSrc<T> src = amp_src(a, norm2);
    auto h = [&](uint32_t k, uint64_t p) -> double {
        if (k == n) return src.raw(p) * src.inv;
        if (k == 0) return n == 1 ? (src.raw(0) + src.raw(1)) * src.inv : tree[0] + tree[1];
        return tree[level_at(k) + p];
    };
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < shots; s += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t pre = 0;
        if (mode == 0) {
            double tot = h(0, 0);
            for (uint32_t q = 0; q < n; ++q) {
                const double left = h(q + 1, pre), p0 = left / tot;
                double kept = left, pb = p0;
                if (!(u[s * n + q] < p0)) {
                    pre |= 1ull << q;
                    kept = h(q + 1, pre);
                    pb = kept / tot;
                }
                if (!(pb > 1e-12)) break;
                tot = kept;
            }
        } else {
            double t = u[s] * h(0, 0);
            for (uint32_t q = 0; q < n; ++q) {
                const double left = h(q + 1, pre);
                if (t < left) continue;
                t -= left;
                pre |= 1ull << q;
            }
        }
        out[s] = pre;
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

// Shots from which a tree of all levels and a thread per shot beat the stored
// levels and a warp per shot (2.5 ns a shot at 20 qubits, against 0.1 ns and
// the tree's writes and launches). Whole calls in us, inverse CDF, warp against
// all levels: 20 qubits 2^14 shots 91 / 48, 2^20 4075 / 936; 24 qubits 2^14 150
// / 161, 2^16 398 / 210; 26 qubits (a tree too large to keep is mapped per
// call) 2^18 1501 / 1610, 2^20 5407 / 2391; 28 qubits 2^18 2219 / 3779, 2^20
// 6566 / 4532. Below 2^14 shots they differ by less than 20 % up to 22 qubits.
bool sample_all_levels(uint32_t n, uint64_t shots) {
    return shots >= std::max<uint64_t>(1ull << 14, (1ull << n) >> 8);
}
uint64_t sample_all_doubles(uint32_t n) { return n >= 2 ? level_at(n) : 1; }

template <bool ALL, typename T>
static cudaError_t fold_amps(const T* a, const double* norm2, uint32_t b, uint32_t lo, double* out, cudaStream_t st) {
    const int g = fold_grid(lo);
    switch (b) {
        case 1: return launch_overlapped(k_fold_amps<1, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
        case 2: return launch_overlapped(k_fold_amps<2, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
        case 3: return launch_overlapped(k_fold_amps<3, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
        case 4: return launch_overlapped(k_fold_amps<4, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
        case 5: return launch_overlapped(k_fold_amps<5, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
        default: return launch_overlapped(k_fold_amps<6, ALL, T>, g, 128, 0, st, a, norm2, lo, out);
    }
}
template <bool ALL>
static cudaError_t fold_level(const double* in, uint32_t b, uint32_t lo, double* out, cudaStream_t st) {
    const int g = fold_grid(lo);
    switch (b) {
        case 1: return launch_overlapped(k_fold_level<1, ALL>, g, 128, 0, st, in, lo, out);
        case 2: return launch_overlapped(k_fold_level<2, ALL>, g, 128, 0, st, in, lo, out);
        case 3: return launch_overlapped(k_fold_level<3, ALL>, g, 128, 0, st, in, lo, out);
        case 4: return launch_overlapped(k_fold_level<4, ALL>, g, 128, 0, st, in, lo, out);
        case 5: return launch_overlapped(k_fold_level<5, ALL>, g, 128, 0, st, in, lo, out);
        default: return launch_overlapped(k_fold_level<6, ALL>, g, 128, 0, st, in, lo, out);
    }
}

// tree: L.total doubles (the stored levels at L.off), or with ALL
// sample_all_doubles(n) (level k at 2^k - 2).
template <bool ALL, typename T>
static cudaError_t sample_tree(const T* a, uint32_t n, const double* norm2, const SampleLevels& L, double* tree,
                               cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (uint32_t k = 0; k < L.count && e == cudaSuccess; ++k) {
        const uint32_t lo = L.bits[k];
        double* out = ALL ? tree : tree + L.off[k];
        if (k == 0) {
            e = fold_amps<ALL>(a, norm2, n - lo, lo, out, st);
            continue;
        }
        const double* in = ALL ? tree + level_at(L.bits[k - 1]) : tree + L.off[k - 1];
        e = fold_level<ALL>(in, L.bits[k - 1] - lo, lo, out, st);
    }
    if (ALL && e == cudaSuccess && n >= 2) e = launch_overlapped(k_tree_root<T>, 1, 128, 0, st, a, n, norm2, tree);
    return e;
}

cudaError_t launch_sample_tree(const void* a, bool f32, uint32_t n, const double* norm2, const SampleLevels& L, bool all,
                               double* tree, cudaStream_t st) {
    if (f32) return all ? sample_tree<true>((const float2*)a, n, norm2, L, tree, st)
                        : sample_tree<false>((const float2*)a, n, norm2, L, tree, st);
    return all ? sample_tree<true>((const double2*)a, n, norm2, L, tree, st)
               : sample_tree<false>((const double2*)a, n, norm2, L, tree, st);
}

template <typename T>
static cudaError_t shots_on(const T* a, uint32_t n, const double* norm2, const double* tree, const SampleLevels& L, bool all,
                            const double* u, uint64_t shots, int mode, unsigned long long* out, cudaStream_t st) {
    const uint64_t blocks = all ? (shots + 127) / 128 : (shots + 3) / 4;
    const int g = (int)(blocks < 148 * 16 ? blocks : 148 * 16);
    if (all) return launch_overlapped(k_shots_tree<T>, g, 128, 0, st, a, n, norm2, tree, u, shots, mode, out);
    return launch_overlapped(k_shots<T>, g, 128, 0, st, a, n, norm2, tree, L, u, shots, mode, out);
}
cudaError_t launch_shots(const void* a, bool f32, uint32_t n, const double* norm2, const double* tree, const SampleLevels& L,
                         bool all, const double* u, uint64_t shots, int mode, unsigned long long* out, cudaStream_t st) {
    return f32 ? shots_on((const float2*)a, n, norm2, tree, L, all, u, shots, mode, out, st)
               : shots_on((const double2*)a, n, norm2, tree, L, all, u, shots, mode, out, st);
}

}  // namespace qoa
