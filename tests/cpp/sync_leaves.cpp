// The leaf searches (shg_leaves.cu, shg_leaves_sh2.cu; their kernels without the launching functions, in
// leaves_sh1.inc and leaves_sh2.inc) under many thread orders: the threads of a block stay together, and seed and
// retrieval bits are the oracle's. The cases come from the file argv[1]: kind (1 original, 2 bipartite), number of leaves, then per leaf its size, seed, keys, and the keys' bits.
#include "cuda_emu.h"
#include "leaves_sh1.inc"
#include "leaves_sh2.inc"
#include <cinttypes>
using namespace shg;

struct Leaf {
    std::vector<uint64_t> keys;
    std::vector<uint32_t> bits;
    uint64_t seed;
};
int bad = 0;

template <class Kernel>
void check(const char *name, const std::vector<Leaf> &leaves, uint64_t order, unsigned threads, size_t smem, const Kernel &kernel) {
    std::vector<Node> nodes;
    std::vector<uint32_t> ids;
    std::vector<uint64_t> keys;
    for (size_t i = 0; i < leaves.size(); i++) {
        Node nd{};
        nd.start = (uint32_t)keys.size(), nd.m = (uint16_t)leaves[i].keys.size(), nd.g = 20;
        nodes.push_back(nd), ids.push_back((uint32_t)i);
        keys.insert(keys.end(), leaves[i].keys.begin(), leaves[i].keys.end());
    }
    std::vector<uint64_t> codes(leaves.size(), ~0ull), rib_keys(keys.size(), 0);
    std::vector<uint8_t> bits(keys.size(), 9);
    uint32_t err = 0;
    unsigned int next = 0;
    unsigned long long work[8] = {};
    const char *e = emu::run(1, threads, smem, order, [&]() {
        kernel(nodes.data(), ids.data(), (uint32_t)leaves.size(), keys.data(), codes.data(), rib_keys.data(), bits.data(), &err,
               work, &next);
    });
    bool ok = !e && !err;
    for (size_t i = 0; ok && i < leaves.size(); i++) {
        ok = codes[i] == leaves[i].seed;
        for (size_t k = 0; ok && k < leaves[i].keys.size(); k++) {
            const size_t at = nodes[i].start + k;
            uint64_t key = rib_keys[at] ? rib_keys[at] : keys[at];  // original leaves list them in cell order
            const size_t j = std::find(leaves[i].keys.begin(), leaves[i].keys.end(), key) - leaves[i].keys.begin();
            ok = j < leaves[i].keys.size() && bits[at] == leaves[i].bits[j];
        }
    }
    if (!ok) {
        bad++;
        printf("%s, %zu leaves of %zu.. keys, order %" PRIu64 ": %s, err %u\n", name, leaves.size(), leaves[0].keys.size(), order,
               e ? e : "wrong products", err);
    }
}

template <int M> void bipartite(const std::vector<Leaf> &leaves, uint64_t order) {
    const uint32_t smax = M > 64 ? 16384 : 4096, cmax = M > 64 ? 16384 : 2048;
    Sh2Global<M> g;
    g.carve(nullptr, smax, cmax);
    const size_t slice = ((size_t)(g.raw + (uint64_t)g.rawcap * (M / 8)) + 255) & ~(size_t)255;
    std::vector<uint64_t> scratch(4 * slice / 8 + 2);
    uint8_t *const base = (uint8_t *)(((uintptr_t)scratch.data() + 15) & ~(uintptr_t)15);
    check("bipartite, warp", leaves, order, 128, 4 * sizeof(Sh2Smem<M>),
          [=](const Node *nodes, const uint32_t *ids, uint32_t n, const uint64_t *keys, uint64_t *codes, uint64_t *, uint8_t *bits,
              uint32_t *err, unsigned long long *work, unsigned *next) {
              k_leaves_sh2_v2<M, NodeLeaves, 4>(NodeLeaves{nodes, ids, codes}, n, keys, bits, base, slice, smax, cmax, err, work,
                                                next, kQuadMinRecSplit);
          });
    check("bipartite, block", leaves, order, 32 * kBlockLeafWarps<M>, sizeof(Sh2BlockSmem<M>),
          [=](const Node *nodes, const uint32_t *ids, uint32_t n, const uint64_t *keys, uint64_t *codes, uint64_t *, uint8_t *bits,
              uint32_t *err, unsigned long long *work, unsigned *next) {
              k_leaves_sh2_block<M, NodeLeaves>(NodeLeaves{nodes, ids, codes}, n, keys, bits, base, slice, smax, cmax, err, work,
                                                next, kQuadMinRecSplit);
          });
}

// Candidate capacities at which a leaf's round no longer fits: both forms list the same prefix of the candidates, so they
// find the seed, or report that the capacity is exceeded, at the same capacities.
template <int M> void capacities(const Leaf &leaf, uint64_t order) {
    int found = 0, full = 0;
    for (uint32_t cmax = 2; cmax <= 512; cmax += cmax < 32 ? 2 : 32) {
        const uint32_t smax = 4096;
        Sh2Global<M> g;
        g.carve(nullptr, smax, cmax);
        const size_t slice = ((size_t)(g.raw + (uint64_t)g.rawcap * (M / 8)) + 255) & ~(size_t)255;
        std::vector<uint64_t> scratch(4 * slice / 8 + 2);
        uint8_t *const base = (uint8_t *)(((uintptr_t)scratch.data() + 15) & ~(uintptr_t)15);
        Node nd{};
        nd.m = (uint16_t)leaf.keys.size();
        const uint32_t id = 0;
        uint64_t code[2] = {~0ull, ~0ull};
        uint32_t err[2] = {};
        const char *e[2];
        for (int form = 0; form < 2; form++) {
            std::vector<uint8_t> bits(leaf.keys.size());
            unsigned long long work[8] = {};
            unsigned next = 0;
            const NodeLeaves src{&nd, &id, &code[form]};
            if (form == 0)
                e[0] = emu::run(1, 32, 4 * sizeof(Sh2Smem<M>), order, [&]() {
                    k_leaves_sh2_v2<M, NodeLeaves, 4>(src, 1, leaf.keys.data(), bits.data(), base, slice, smax, cmax, &err[0], work,
                                                      &next, kQuadMinRecSplit);
                });
            else
                e[1] = emu::run(1, 32 * kBlockLeafWarps<M>, sizeof(Sh2BlockSmem<M>), order, [&]() {
                    k_leaves_sh2_block<M, NodeLeaves>(src, 1, leaf.keys.data(), bits.data(), base, slice, smax, cmax, &err[1], work,
                                                      &next, kQuadMinRecSplit);
                });
        }
        const bool ok = code[0] == leaf.seed ? err[0] == 0 : code[0] == ~0ull && err[0] == kErrScratch;
        if (e[0] || e[1] || !ok || code[0] != code[1] || err[0] != err[1]) {
            bad++;
            printf("capacity %u, %zu keys: %s %s, err %u %u, seed %" PRIu64 " %" PRIu64 " want %" PRIu64 "\n", cmax, leaf.keys.size(),
                   e[0] ? e[0] : "", e[1] ? e[1] : "", err[0], err[1], code[0], code[1], leaf.seed);
        }
        (code[1] == leaf.seed ? found : full)++;
    }
    if (!found || !full) bad++, printf("capacities of %zu keys: found %d, exceeded %d\n", leaf.keys.size(), found, full);
}

int main(int, char **argv) {
    FILE *f = fopen(argv[1], "r");
    int kind = 0;
    size_t count = 0;
    for (uint64_t set = 0; f && fscanf(f, "%d %zu", &kind, &count) == 2; set++) {
        std::vector<Leaf> leaves(count);
        for (Leaf &l : leaves) {
            size_t m = 0;
            if (fscanf(f, "%zu %" SCNu64, &m, &l.seed) != 2) return 2;
            l.keys.resize(m), l.bits.resize(m);
            for (auto &k : l.keys)
                if (fscanf(f, "%" SCNu64, &k) != 1) return 2;
            for (auto &b : l.bits)
                if (fscanf(f, "%u", &b) != 1) return 2;
        }
        for (uint64_t order = 10 * set; order < 10 * set + 10; order++) {
            if (kind == 1) {
                auto sh1 = [&](auto kernel) {
                    return [kernel](const Node *nodes, const uint32_t *ids, uint32_t n, const uint64_t *keys, uint64_t *codes,
                                    uint64_t *rib_keys, uint8_t *bits, uint32_t *err, unsigned long long *work, unsigned *next) {
                        kernel(nodes, ids, n, keys, codes, rib_keys, bits, 0, err, work, next, 0);
                    };
                };
                const unsigned th = 32 * kLeafWarps;
                check("original, block", leaves, order, th, 0, sh1(k_leaves_sh1<1, true, false>));
                check("original, block, pairs", leaves, order, th, 0, sh1(k_leaves_sh1<2, true, true>));
                check("original, warp", leaves, order, th, 0, sh1(k_leaves_sh1<2, false, false>));
                check("original, warp, pairs", leaves, order, th, 0, sh1(k_leaves_sh1<1, false, true>));
            } else {
                if (leaves.size() == 1 && leaves[0].keys.size() == 64 && order == 10 * set) capacities<64>(leaves[0], order);
                if (leaves[0].keys.size() <= 64) bipartite<64>(leaves, order);
                else bipartite<128>(leaves, order);
            }
        }
    }
    printf(bad ? "failed\n" : "ok\n");
    return bad != 0;
}
