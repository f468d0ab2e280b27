// The first sieve of the original ShockHash leaf search (shg_leaves.cu), shared with its microbenchmark.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "shg_common.cuh"

namespace shg {

// Per seed offset at + 32 * t (t < SPL): the second-half cells of all m staged keys as a mask (cells
// below h2), taken from the high product word without remix's last xor-shift, and the smallest low word
// of (word + 1) * h2 over the keys. The cells are exact unless that is below 2 * h2 (sh1_half_passes).
template <int SPL>
__device__ __forceinline__ void sh1_half_masks(const SeedKey *__restrict__ staged, uint32_t m, uint32_t h2, uint32_t at,
                                               uint32_t (&mask)[SPL], uint32_t (&low)[SPL]) {
    const uint64_t range = h2;
#pragma unroll 4
    for (uint32_t k = 0; k < m; k++) {
        const SeedKey key = staged[k];
#pragma unroll
        for (int t = 0; t < SPL; t++) {
            const uint64_t p = seed_hi_product(key, at + 32 * t) * range + range;
            mask[t] |= 1u << (uint32_t)(p >> 32);
            low[t] = min(low[t], (uint32_t)p);
        }
    }
}
// The same for pairs of consecutive seeds that share remix's first product: with z = key + t even, the first
// xor-shift of z + 1 differs from that of z in its lowest bit only, so its product is that of z plus or minus
// M1 (delta; minus if the key's fold is odd). The lane's seeds are at + 64 p + 2 lane and the one after it,
// p < PAIRS, `at` even; keys [0, evens) are even under even seeds, the others, [evens, m), odd: their pairs are
// the seeds 2 lane - 1 and 2 lane, so that a seed 2 lane + 1 takes its odd keys' part from the next lane, and the
// last of the 64 * PAIRS seeds lacks it. Bound by the integer pipes; first sieve alone on leaves of 40 keys, two seeds
// per lane / two pairs: 1,354 / 1,588 G evaluations/s (four keys per turn of the loop; three 1,499, two 1,475, one 1,428).
constexpr uint32_t sh1_pair_seeds(int pairs) { return 64 * pairs - 2; }  // complete ones, an even number
template <int PAIRS>
__device__ __forceinline__ void sh1_half_pairs(const SeedKey *__restrict__ staged, const uint2 *__restrict__ delta, uint32_t evens,
                                               uint32_t m, uint32_t h2, uint32_t at, uint32_t (&mask)[2 * PAIRS],
                                               uint32_t (&low)[2 * PAIRS]) {
    const uint64_t range = h2;
    const int lane = threadIdx.x & 31;
    auto side = [&](uint32_t k0, uint32_t k1, uint32_t t0, uint32_t (&bits)[2 * PAIRS], uint32_t (&least)[2 * PAIRS]) {
        auto cell = [&](uint32_t l, uint32_t h, int i) {
            const uint32_t l2 = l ^ funnel_r(l, h, 27), h2_ = h ^ (h >> 27);
            const uint64_t p = (uint64_t)(mulhi32(l2, kM2Lo) + l2 * kM2Hi + h2_ * kM2Lo) * range + range;
            bits[i] |= 1u << (uint32_t)(p >> 32);
            least[i] = min(least[i], (uint32_t)p);
        };
#pragma unroll 4
        for (uint32_t k = k0; k < k1; k++) {
            const SeedKey key = staged[k];
            const uint2 d = delta[k];
#pragma unroll
            for (int p = 0; p < PAIRS; p++) {
                const uint32_t lo = (key.lo + (t0 + 64 * p)) ^ key.fold;
                const uint64_t first = (uint64_t)lo * kM1Lo + key.hc;
                const uint32_t l = (uint32_t)first, h = (uint32_t)(first >> 32) + lo * kM1Hi;
                cell(l, h, 2 * p);
                const uint64_t second = ((uint64_t)h << 32 | l) + ((uint64_t)d.y << 32 | d.x);
                cell((uint32_t)second, (uint32_t)(second >> 32), 2 * p + 1);
            }
        }
    };
    uint32_t odd_bits[2 * PAIRS], odd_least[2 * PAIRS];
#pragma unroll
    for (int i = 0; i < 2 * PAIRS; i++) mask[i] = odd_bits[i] = 0, low[i] = odd_least[i] = ~0u;
    side(0, evens, at + 2 * lane, mask, low);
    side(evens, m, at + 2 * lane - 1, odd_bits, odd_least);
#pragma unroll
    for (int p = 0; p < PAIRS; p++) {
        uint32_t nb = __shfl_down_sync(0xffffffffu, odd_bits[2 * p], 1), nl = __shfl_down_sync(0xffffffffu, odd_least[2 * p], 1);
        if (p + 1 < PAIRS) {
            const uint32_t wb = __shfl_sync(0xffffffffu, odd_bits[(2 * p + 2) % (2 * PAIRS)], 0),
                           wl = __shfl_sync(0xffffffffu, odd_least[(2 * p + 2) % (2 * PAIRS)], 0);
            if (lane == 31) nb = wb, nl = wl;
        }
        mask[2 * p] |= odd_bits[2 * p + 1];
        low[2 * p] = min(low[2 * p], odd_least[2 * p + 1]);
        mask[2 * p + 1] |= nb;
        low[2 * p + 1] = min(low[2 * p + 1], nl);
    }
}
// Whether a seed may cover the second half: never false for one that does.
__device__ __forceinline__ bool sh1_half_passes(uint32_t mask, uint32_t low, uint32_t all2, uint32_t h2) {
    return (mask & all2) == all2 || low < 2 * h2;
}

} // namespace shg
