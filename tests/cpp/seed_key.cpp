// Host check of the staged key form (SeedKey, shg_common.cuh): for every seed offset within a key's
// room it gives the low 16 bits of remix, and the top two of them at every bit position, and z back.
#include <cstdio>
#include <random>
#include "shg_common.cuh"
using namespace shg;

template <int P> int check(const SeedKey &k, uint64_t z, uint32_t t) {
    uint32_t a, b;
    seed_quarter_at<P>(k, t, a, b);
    const uint32_t want = remix(z + t) & 0xFFFF, v = seed_low16_at30(k, t);
    if ((((a ^ b) >> (P - 1)) & 3) != want >> 14 || v >> 15 != want) {
        printf("P %d z %llx t %u\n", P, (unsigned long long)z, t);
        return 1;
    }
    if constexpr (P < 31) return check<P + 1>(k, z, t);
    else return 0;
}

int main() {
    std::mt19937_64 rng(5);
    for (int i = 0; i < 200000; i++) {
        uint64_t z = rng();
        if (i % 3 == 0) z |= 0x3fffffffull - rng() % 100;  // little room
        if (i % 7 == 0) z |= ~0ull << (rng() % 64);
        const SeedKey k = seed_key(z);
        const uint32_t room = seed_room(z);
        if (seed_key_z(k) != z || room == 0 || room > kSeedSpan) return printf("z %llx\n", (unsigned long long)z), 1;
        const uint32_t ts[4] = {0, room - 1, (uint32_t)(rng() % room), (uint32_t)(rng() % (room < 5000 ? room : 5000))};
        for (uint32_t t : ts)
            if (check<17>(k, z, t)) return 1;
    }
    // the original leaves' first sieve (shg_sh1.cuh): a cell taken without remix's last xor-shift is the
    // exact one, or the low word says that it may not be
    for (uint32_t h2 = 1; h2 <= 30; h2++) {
        for (uint64_t j = 0; j <= h2; j++)
            for (int d = -70; d <= 70; d++) {
                const uint32_t t = (uint32_t)((j << 32) / h2 + d);
                const uint64_t p = (uint64_t)t * h2 + h2;
                const uint32_t cell = fastrange32(t ^ (t >> 31), h2);
                if ((uint32_t)p >= 2 * h2 && (uint32_t)(p >> 32) != cell) return printf("h2 %u t %u\n", h2, t), 1;
            }
    }
    for (int i = 0; i < 200000; i++) {  // the high word of the second product
        const uint64_t z = rng();
        const uint32_t t = (uint32_t)(rng() % seed_room(z)), hi = seed_hi_product(seed_key(z), t);
        if ((hi ^ (hi >> 31)) != (uint32_t)(remix(z + t) >> 32) || seed_lo(seed_key(z), t) != (uint32_t)remix(z + t))
            return printf("words z %llx\n", (unsigned long long)z), 1;
    }
    printf("ok\n");
    return 0;
}
