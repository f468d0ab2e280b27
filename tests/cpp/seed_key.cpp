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
    printf("ok\n");
    return 0;
}
