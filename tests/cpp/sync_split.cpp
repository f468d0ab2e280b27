// The split search by several blocks per node (shg_split.cuh) under many thread orders: the threads of a block
// stay together, and the seed and the partition are those of a sequential search.
#include "cuda_emu.h"
#include "shg_split.cuh"
using namespace shg;

template <int SPL, int THREADS, bool SIMD> int check(uint32_t m, uint32_t unit, int fanout, uint32_t stripes, uint64_t seed) {
    std::mt19937_64 rng(seed);
    std::vector<uint64_t> keys(m), in;
    for (auto &k : keys) k = rng();
    if (seed % 2) {  // low 30 bits about to run over: plain rounds and staging again
        for (auto &k : keys) k = ((k | 0x3fffffff) - start_seed(0)) - rng() % 4000;
    }
    in = keys;
    Node nd{};
    nd.m = (uint16_t)m, nd.unit = (uint16_t)unit, nd.fanout = (uint8_t)fanout, nd.g = 20;
    nd.kind = fanout == 2 ? kSplit2 : kSplitK;
    // sequential search
    auto part_of = [&](uint64_t z) {
        const uint32_t h = ((SIMD ? simd_split_low16(z) : remix_low16(z)) * m) >> 16;
        return fanout == 2 ? (uint32_t)(h >= unit) : h / unit;
    };
    uint64_t want = 0;
    const int parts = fanout == 2 ? 2 : (m + unit - 1) / unit;
    for (;; want++) {
        std::vector<uint32_t> c(parts);
        for (uint64_t k : in) c[part_of(k + start_seed(0) + want)]++;
        bool ok = true;
        for (int p = 0; p + 1 < parts; p++) ok = ok && c[p] == unit;
        if (ok) break;
    }
    std::vector<uint64_t> sorted = in;
    std::stable_sort(sorted.begin(), sorted.end(), [&](uint64_t a, uint64_t b) {
        return part_of(a + start_seed(0) + want) < part_of(b + start_seed(0) + want);
    });
    using S = SplitSmem<SPL, THREADS, SIMD>;
    uint64_t code = ~0ull;
    uint32_t err = 0;
    unsigned long long work = 0, kind_work[4] = {};
    SplitBest best{};
    const char *e = emu::run(stripes, THREADS, sizeof(S), seed, [&]() {
        S &sm = *reinterpret_cast<S *>(emu::shared + blockIdx.x * emu::shared_bytes);
        split_node<SPL, THREADS, SIMD, false, true>(sm, nd, 0, keys.data(), &code, 0, &err, &work, kind_work, 8,
                                                    SplitStripe{blockIdx.x, stripes, &best});
    });
    if (e || err || code != want || keys != sorted) {
        printf("m %u unit %u fanout %d stripes %u seed %llu: %s, err %u, code %llu want %llu\n", m, unit, fanout, stripes,
               (unsigned long long)seed, e ? e : "wrong products", err, (unsigned long long)code, (unsigned long long)want);
        return 1;
    }
    return 0;
}

int main() {
    int bad = 0;
    for (uint64_t seed = 0; seed < 24; seed++) {
        bad += check<1, 128, false>(96, 24, 4, 5, seed);   // quarter split
        bad += check<1, 64, false>(90, 40, 3, 4, seed);    // two thresholds
        bad += check<1, 64, true>(100, 30, 4, 3, seed);    // three thresholds, SIMDShockHash's split hash
        bad += check<2, 64, false>(2000, 960, 2, 2, seed); // two parts: few trials, one stripe takes part
    }
    printf(bad ? "failed\n" : "ok\n");
    return bad != 0;
}
