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
// Whether a seed may cover the second half: never false for one that does.
__device__ __forceinline__ bool sh1_half_passes(uint32_t mask, uint32_t low, uint32_t all2, uint32_t h2) {
    return (mask & all2) == all2 || low < 2 * h2;
}

} // namespace shg
