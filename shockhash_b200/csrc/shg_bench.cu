// Measurement utilities (not part of the reference's interface):
//  * the seeded key generators the benchmark configurations name (std::mt19937_64), shared by the
//    CPU and GPU runs so both build from the same keys;
//  * the integer-pipe peaks of the searches: each search kernel's dominant inner loop (split: the
//    counting loops over staged keys; original leaf: remix, two fastrange32 cells, half masks;
//    bipartite leaf: remix, fastrange64, mask), two seeds per lane, on operands in registers and
//    shared memory. Their evaluations per second are the
//    denominators of the search kernels' roofline fractions.
#include <algorithm>
#include <cstdint>
#include <random>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#include "shg.h"
#include "shg_common.cuh"
#include "shg_internal.h"
#include "shg_sh1.cuh"
#include "shg_split.cuh"

namespace {

constexpr int kPeakThreads = 256;

// The split kernel's own counting loops (shg_split.cuh) alone: 256 staged keys in shared memory,
// lanes on consecutive seeds, two seeds per lane; the quarter split (NT = 4) or compare-and-count against
// NT thresholds, under remix or SIMDShockHash's split hash. `iters` key reads per thread, rounded up to
// whole rounds (the caller counts the rounded number).
constexpr uint32_t kPeakKeys = 256;
template <int NT, bool SIMD>
__global__ void __launch_bounds__(kPeakThreads) k_int_peak_split(uint64_t iters, uint32_t T0, uint32_t T1, uint32_t T2,
                                                                 unsigned long long *sink) {
    __shared__ shg::SplitKey<SIMD> keys[kPeakKeys];
    // low 30 bits zero: every seed of the run is within the keys' room
    for (uint32_t i = threadIdx.x; i < kPeakKeys; i += blockDim.x)
        keys[i] = shg::SplitKey<SIMD>::make(shg::remix(0x9E3779B97F4A7C15ULL * (i + 1) + blockIdx.x) & ~(uint64_t)(shg::kSeedSpan - 1));
    __syncthreads();
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    uint32_t seed = (threadIdx.x >> 5) * 64 + (threadIdx.x & 31), out = 0;
    for (uint64_t done = 0; done < iters; done += kPeakKeys, seed = (seed + 512) & (shg::kSeedSpan / 2 - 1)) {
        uint32_t c[2][3] = {};
        if constexpr (NT == 4) shg::quarter_range<2, SIMD>(keys, 0, kPeakKeys, seed, c);
        else shg::count_range<NT, 2, SIMD>(keys, 0, kPeakKeys, seed, T0, T1, T2, c);
        for (int s = 0; s < 2; s++) out ^= c[s][0] ^ c[s][1] ^ c[s][2];
    }
    sink[tid] = out;  // every thread's result is stored: no loop can fold
}
template <bool SIMD> void launch_peak_split(int nt, int blocks, uint64_t iters, unsigned long long *sink) {
    switch (nt) {
        case 1: k_int_peak_split<1, SIMD><<<blocks, kPeakThreads>>>(iters, 50331, 65536, 65536, sink); break;
        case 2: k_int_peak_split<2, SIMD><<<blocks, kPeakThreads>>>(iters, 21846, 43691, 65536, sink); break;
        case 3: k_int_peak_split<3, SIMD><<<blocks, kPeakThreads>>>(iters, 16384, 32768, 49152, sink); break;
        default: k_int_peak_split<4, SIMD><<<blocks, kPeakThreads>>>(iters, 16384, 32768, 49152, sink); break;
    }
}

// The original leaf search's first sieve as the leaf kernel runs it, alone: a leaf of h1 + h2 staged keys
// in shared memory, two pairs of consecutive seeds per lane, the masks compared after each round; no later
// sieves. `iters` pairs of evaluations per thread, rounded up to whole rounds (the caller counts the rounded
// number).
__global__ void __launch_bounds__(kPeakThreads) k_int_peak_sh1(uint64_t iters, uint32_t h1, uint32_t h2,
                                                               unsigned long long *sink) {
    __shared__ shg::SeedKey keys[64];
    __shared__ uint2 delta[64];
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {  // every key even
        keys[i] = shg::seed_key(shg::remix(0x9E3779B97F4A7C15ULL * (i + 1) + blockIdx.x) & ~(uint64_t)(shg::kSeedSpan - 1));
        const uint64_t d = keys[i].fold & 1 ? 0ull - shg::kRemixM1 : shg::kRemixM1;
        delta[i] = make_uint2((uint32_t)d, (uint32_t)(d >> 32));
    }
    __syncthreads();
    const uint32_t m = h1 + h2, all2 = (1u << h2) - 1;
    uint32_t at = (threadIdx.x >> 5) * 128, hits = 0;
    for (uint64_t done = 0; done < iters; done += 2 * m, at = (at + 1024) & (shg::kSeedSpan / 2 - 1)) {
        uint32_t mask[4], low[4];
        shg::sh1_half_pairs<2>(keys, delta, m, m, h2, at, mask, low);
#pragma unroll
        for (int t = 0; t < 4; t++) hits += shg::sh1_half_passes(mask[t], low[t], all2, h2);
    }
    sink[blockIdx.x * (uint64_t)blockDim.x + threadIdx.x] = hits;
}

// The bipartite leaf search's raw-seed hashing alone: 64 staged keys, two seeds per lane, the same arithmetic
// as the original leaves' first sieve (high product word, range reduction, one bit into a 32-bit mask).
__global__ void __launch_bounds__(kPeakThreads) k_int_peak_sh2(uint64_t iters, uint32_t half, unsigned long long *sink) {
    __shared__ shg::SeedKey keys[64];
    for (int i = threadIdx.x; i < 64; i += blockDim.x)
        keys[i] = shg::seed_key(shg::remix(0x9E3779B97F4A7C15ULL * (i + 1) + blockIdx.x) & ~(uint64_t)(shg::kSeedSpan - 1));
    __syncthreads();
    uint32_t at = (threadIdx.x >> 5) * 64 + (threadIdx.x & 31), out = 0;
    for (uint64_t done = 0; done < iters; done += 64, at = (at + 512) & (shg::kSeedSpan / 2 - 1)) {
        uint32_t mask[2] = {0, 0}, low[2] = {~0u, ~0u};
        shg::sh1_half_masks<2>(keys, 64, half, at, mask, low);
        out ^= mask[0] ^ mask[1] ^ low[0] ^ low[1];
    }
    sink[blockIdx.x * (uint64_t)blockDim.x + threadIdx.x] = out;
}

} // namespace

extern "C" {

// n keys from std::mt19937_64(seed), duplicates removed by drawing replacements (the reference
// loops forever on duplicate keys), in draw order.
void shg_keys_mt19937_64(uint64_t seed, uint64_t n, uint64_t *out) {
    std::mt19937_64 rng(seed);
    for (uint64_t i = 0; i < n; i++) out[i] = rng();
    std::vector<uint64_t> sorted(out, out + n);
    std::sort(sorted.begin(), sorted.end());
    if (std::adjacent_find(sorted.begin(), sorted.end()) == sorted.end()) return;
    std::vector<uint64_t> seen;
    seen.reserve(n);
    std::vector<uint64_t> tmp(out, out + n);
    std::sort(tmp.begin(), tmp.end());
    // replace later occurrences of a duplicate by fresh draws that are not present
    std::vector<uint64_t> uniq;
    uniq.reserve(n);
    std::vector<char> keep(n, 1);
    {
        std::vector<std::pair<uint64_t, uint64_t>> vi(n);
        for (uint64_t i = 0; i < n; i++) vi[i] = {out[i], i};
        std::sort(vi.begin(), vi.end());
        for (uint64_t i = 1; i < n; i++)
            if (vi[i].first == vi[i - 1].first) keep[vi[i].second] = 0;
    }
    for (uint64_t i = 0; i < n; i++) {
        while (!keep[i]) {
            const uint64_t v = rng();
            if (!std::binary_search(tmp.begin(), tmp.end(), v)) {
                out[i] = v;
                keep[i] = 1;
                tmp.insert(std::upper_bound(tmp.begin(), tmp.end(), v), v);
            }
        }
    }
}

// Request keys of the serving stream: out[j] = remix(seed ^ (j * 0x9E3779B97F4A7C15)), j < n. Each
// step is a bijection of 64-bit words, so the n keys are distinct with no check; host threads each
// fill a contiguous range.
void shg_keys_mix(uint64_t seed, uint64_t n, uint64_t *out, int threads) {
    const uint64_t T = (uint64_t)std::max(1, std::min(threads, 64));
    const uint64_t chunk = (n + T - 1) / T;
    auto fill = [&](uint64_t a, uint64_t b) {
        for (uint64_t j = a; j < b; j++) out[j] = shg::remix(seed ^ (j * 0x9E3779B97F4A7C15ULL));
    };
    if (T == 1 || n < (1u << 16)) {
        fill(0, n);
        return;
    }
    std::vector<std::thread> pool;
    for (uint64_t t = 0; t < T; t++) {
        const uint64_t a = std::min(n, t * chunk), b = std::min(n, a + chunk);
        if (a < b) pool.emplace_back(fill, a, b);
    }
    for (auto &th : pool) th.join();
}

// Integer-pipe peak of one search's inner loop (0 = quarter split, 1 = original leaf,
// 2 = bipartite leaf hashing, 3..5 = split compare-and-count with 1..3 thresholds, 6..8 = bipartite
// candidate scan, pair filter and pseudoforest edges, 9..12 = the loops of kinds 0 and 3..5 again
// (split_arith 1 runs the same ones), 13..15 = kinds 6..8 for leaves of more than 64 keys, 16..19 =
// kinds 0 and 3..5 under SIMDShockHash's split hash, 20 = kind 13 with the other form of the mask test).
int shg_int_peak_kind(int device, int kind, uint64_t iters, double *evals_per_s, double *ms_out) {
    if (kind < 0 || kind > 20) return SHG_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return SHG_ERR_CUDA;
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, device);
    const int blocks = prop.multiProcessorCount * 8;
    unsigned long long *sink;
    if (cudaMalloc(&sink, (size_t)blocks * kPeakThreads * 8) != cudaSuccess) return SHG_ERR_OOM;  // one result per thread
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    for (int rep = 0; rep < 2; rep++) {  // warm-up, then the timed run
        const uint64_t it = rep ? iters : iters / 16 + 1;
        if (rep) cudaEventRecord(a);
        if (kind == 1)
            k_int_peak_sh1<<<blocks, kPeakThreads>>>(it, 20, 20, sink);
        else if (kind == 2)
            k_int_peak_sh2<<<blocks, kPeakThreads>>>(it, 32, sink);
        else if (kind == 0 || kind == 9)
            launch_peak_split<false>(4, blocks, it, sink);
        else if (kind <= 5)
            launch_peak_split<false>(kind - 2, blocks, it, sink);
        else if (kind <= 8)  // the bipartite leaf's scan, pair filter and pseudoforest loops (64 edges per iteration)
            shg::launch_sh2_op_peak(kind - 6, blocks, kind == 8 ? it / 64 + 1 : it, sink);
        else if (kind <= 12)
            launch_peak_split<false>(kind - 9, blocks, it, sink);
        else if (kind >= 16 && kind <= 19)
            launch_peak_split<true>(kind == 16 ? 4 : kind - 16, blocks, it, sink);
        else if (kind == 20)
            shg::launch_sh2_op_peak(6, blocks, it, sink);
        else  // 13..15: kinds 6..8 for leaves of more than 64 keys (100 edges per iteration)
            shg::launch_sh2_op_peak(kind - 10, blocks, kind == 15 ? it / 100 + 1 : it, sink);
        if (rep) cudaEventRecord(b);
    }
    cudaEventSynchronize(b);
    float ms = 0;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(sink);
    if (cudaGetLastError() != cudaSuccess) return SHG_ERR_CUDA;
    double per_iter = 2.0;
    uint64_t timed_iters = iters;
    if (kind >= 6 && kind <= 8) {
        per_iter = shg::sh2_op_peak_per_iter(kind - 6);
        if (kind == 8) timed_iters = iters / 64 + 1;
    } else if (kind >= 13 && kind <= 15) {
        per_iter = shg::sh2_op_peak_per_iter(kind - 10);
        if (kind == 15) timed_iters = iters / 100 + 1;
    } else if (kind == 20) {
        per_iter = shg::sh2_op_peak_per_iter(6);
    } else if (kind == 1) {
        timed_iters = (iters + 79) / 80 * 80;  // whole rounds of the 40-key leaf, two pairs of seeds each
    } else if (kind == 2) {
        timed_iters = (iters + 63) / 64 * 64;  // whole rounds of the 64-key leaf
    } else {
        timed_iters = (iters + kPeakKeys - 1) / kPeakKeys * kPeakKeys;  // whole rounds of the split loops' keys
    }
    *evals_per_s = per_iter * (double)timed_iters * blocks * kPeakThreads / (ms * 1e-3);
    if (ms_out) *ms_out = ms;
    return SHG_OK;
}

int shg_int_peak(int device, uint64_t iters, double *evals_per_s, double *ms_out) {
    return shg_int_peak_kind(device, 0, iters, evals_per_s, ms_out);
}

} // extern "C"
