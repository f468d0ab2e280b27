// ShockHash leaf searches, one warp per leaf, leaves pulled from a device counter.
//
// Original ShockHash (ShockHash.h:404-434): lanes take consecutive seeds x, or pairs of them; a lane's seed
// passes when the two candidate cells of all m keys cover all m cells and the cuckoo graph
// (cells = vertices, keys = edges) is a pseudoforest. Seeds go through three sieves in seed order:
// the second-half cells of all keys cover their half (one key in 8 to 20 does, for leaves of 30 to 40
// keys), both halves are covered, pseudoforest. The pseudoforest test peels the graph (group_peel); the
// reference inserts into a cuckoo table instead, and
// ordered cuckoo insertion succeeds exactly when the graph is a pseudoforest, so both accept the
// same seeds. The coverage mask is kept as two 32-bit halves (first-half and second-half cells).
// The smallest accepted seed is kept (ballot + find-first-set), then lane 0 replays
// the reference's ordered cuckoo insertion to obtain the cell of every key (the retrieval bits).
//
// The bipartite leaf search is in shg_leaves_sh2.cu.
#include <cstdint>
#include <cuda_runtime.h>
#include "shg_common.cuh"
#include "shg_internal.h"
#include "shg_sh1.cuh"

namespace shg {

constexpr int kLeafWarps = 4;  // warps per block

// Ordered cuckoo insertion with cycle detection (TinyBinaryCuckooHashTable.h:169-198), run by one
// thread. cell[c] = key index or -1; xr[e] = c1 ^ c2 of key e. Returns false when the walk returns
// to its start (insertion impossible) or exceeds `limit` steps.
__device__ bool cuckoo_insert(int16_t *cell, uint8_t *xr, int e, uint32_t c1, uint32_t c2, int limit) {
    xr[e] = (uint8_t)(c1 ^ c2);
    if (cell[c1] < 0) { cell[c1] = (int16_t)e; return true; }
    if (cell[c2] < 0) { cell[c2] = (int16_t)e; return true; }
    uint32_t cur = c1;
    const uint32_t orig_cell = cur;
    int entry = e;
    for (int step = 0; step < limit; step++) {
        const uint32_t alt = xr[entry] ^ cur;
        const int displaced = cell[alt];
        cell[alt] = (int16_t)entry;
        entry = displaced;
        if (entry < 0) return true;
        cur = alt;
        if (cur == orig_cell && entry == e) return false;
    }
    return false;
}

// ------------------------------------------------------------------ original ShockHash leaves
// Seeds that pass a sieve queue up in seed order for the next one, so that each runs with its lanes
// filled: the first sieve's survivors are tested for the other half's coverage 32 at a time (one per lane;
// leaves of up to kSh1SmallLeaf keys, which expect fewer seeds than a round has, after every round),
// and the full coverage's for the pseudoforest property four at a time, straight after that (waiting for two /
// three / four of them: ShockHash<30>, 4M keys 9.0 -> 9.3 / 9.4 / 9.6 ms, ShockHash<40>, 1M 36.1 -> 36.4 / 37.2 / 38.0).
//
// What bounds it: the integer pipes, in the first sieve, which sees every seed. It therefore works on
// staged keys (SeedKey, shg_common.cuh), looks at one half of the cells only (one range reduction, shift
// and or per key instead of two), and takes the high word of remix without its last xor-shift: that
// can change the lowest bit alone, so the cell is the same unless the product with the half's size
// lies within one size of a multiple of 2^32. The smallest low word over the keys says whether one
// does; such a seed (about 1 in 10^6) counts as passing, and the second sieve decides.
constexpr uint32_t kSh1SmallLeaf = 16;
constexpr uint64_t kSh1Unsure = 1ull << 63;  // on a waiting seed offset (below 2^41): the second half is to be checked
constexpr uint32_t kSh1Half = 31 + 128;       // waiting for the full coverage: at most 31, plus one round's (at most 128)

struct Sh1WarpSmem {
    SeedKey staged[64];     // the keys under the first seed of the current span (PAIRS: even ones first)
    uint64_t half[kSh1Half];  // seed offsets that cover the second half, ascending
    uint64_t q[32];         // coverage-passing seed offsets of a batch, ascending
    uint64_t keys[64];
    union {
        uint64_t fkeys[64];  // rotation fitting: even keys in order, odd keys from the back
        uint2 delta[64];     // PAIRS: what a key's first product changes by from an even seed to the next
    };
    int16_t cell[64];
    uint8_t xr[64];
};

// Whether the cuckoo graph of m keys over m cells, all of them covered, is a pseudoforest; a group of 8 lanes
// tests one graph, the warp four (`live` false: no graph, and false for it). cells(k, c1, c2): the two cells of key
// k of the group's graph. As there are as many edges as vertices, the graph is a pseudoforest exactly if no
// component is a tree. So the vertices of degree one are taken off with their edges, all at a time, until there
// are none: a tree ends in an edge between two of them or in a vertex whose edges all went. They are the
// vertices seen once, but not twice, in the union of the lanes' edges.
//
// Against one lane per graph with a union-find in shared memory, of which few graphs at a time filled few lanes:
// hashing takes an eighth of the steps, and a turn of the peeling (about five) has no dependent memory access.
// Leaf stage: ShockHash<16>, 2M keys 0.70 -> 0.49 ms; ShockHash<30>, 4M 10.9 -> 9.0; ShockHash<40>, 1M 39.1 -> 35.4.
// M: a word with more bits than cells (the top bit carries the lanes' verdicts). E: keys per lane.
template <class M, int E, class Cells>
__device__ __forceinline__ bool group_peel(uint32_t m, bool live, const Cells &cells) {
    constexpr M kTree = (M)1 << (8 * sizeof(M) - 1);
    M v[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const uint32_t k = 8 * e + (threadIdx.x & 7);
        v[e] = 0;
        if (live && k < m) {
            uint32_t c1, c2;
            cells(k, c1, c2);
            v[e] = (M)1 << c1 | (M)1 << c2;
        }
    }
    M left = ((M)1 << m) - 1, ones = 0;  // vertices not taken off; those of degree one
    bool tree = !live;
    for (;;) {
        M once = 0, twice = 0;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const M x = v[e] & ones;
            if (x) {
                if (x == v[e]) once |= kTree;
                v[e] = 0;
            }
            twice |= once & v[e];
            once |= v[e];
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const M xo = __shfl_xor_sync(0xffffffffu, once, o), xt = __shfl_xor_sync(0xffffffffu, twice, o);
            twice |= xt | (once & xo);
            once |= xo;
        }
        left &= ~ones;
        tree = tree || (once & kTree) || (left & ~once);
        ones = tree ? 0 : once & ~twice;
        if (!__any_sync(0xffffffffu, ones != 0)) return !tree;
    }
}
// Words and keys per lane by the number of cells: 32 bits hold up to 31 of them, and five keys for each of the eight
// lanes are enough up to 40. Leaf stage at 1M keys, five keys / eight: ShockHash<32> 4.86 / 4.96 ms, <40> 34.9 / 35.0, rotation
// fitting <40> 5.82 / 5.96. (Six keys up to 48 against eight: ShockHash<44>, 50,000 keys 11.6-11.9 / 12.0-12.2 ms, <48>, 20,000 30.4-31.0 /
// 29.7-30.3: within what runs differ by.)
template <class Cells> __device__ __forceinline__ bool group_pseudoforest(uint32_t m, bool live, const Cells &cells) {
    if (m == 1) return live;  // its two cells are one
    if (m < 32) return group_peel<uint32_t, 4>(m, live, cells);
    if (m <= 40) return group_peel<uint64_t, 5>(m, live, cells);
    return group_peel<uint64_t, 8>(m, live, cells);
}

// Rotation of the low l bits of v by r < l (ShockHash.h:299-301).
template <class M> __device__ __forceinline__ M rot_bits(M v, uint32_t r, uint32_t l, M all) {
    return r ? ((v << r) | (v >> (l - r))) & all : v;
}

// The cells of a staged key under seed offset t (sh1_cells).
__device__ __forceinline__ void sh1_staged_cells(const SeedKey &k, uint32_t t, uint32_t m, uint32_t &c1, uint32_t &c2) {
    uint32_t l2, h2;
    seed_mid(k, t, l2, h2);
    const uint64_t p = (uint64_t)l2 * kM2Lo;
    const uint32_t lo = (uint32_t)p, hi = (uint32_t)(p >> 32) + l2 * kM2Hi + h2 * kM2Lo;
    c1 = fastrange32(lo ^ funnel_r(lo, hi, 31), m / 2);
    c2 = fastrange32(hi ^ (hi >> 31), (m + 1) / 2) + m / 2;
}

// ShockHash<L, true>: a leaf of exactly L keys with rotation fitting (ShockHash.h:316-399). Keys
// are split into set A (even keys, in order) and set B (odd keys, from the back); for seed x, set A
// hashes with x & ~mask (mask 7 when L > 32, so eight seeds share set A's cells) and set B with x.
// For r = 0..L-1 the candidate is set B's cells rotated by r: it passes when A's cells and B's
// rotated cells cover all L cells and the cuckoo graph is a pseudoforest. The answer is the
// smallest x, then the smallest r; the stored code is (x - start_seed) * L + r.
//
// Lanes take consecutive x. What bounds a round is the pseudoforest tests: about a third of the seeds
// have a rotation that covers, and one in thirty of those rotations passes. So the covering pairs (x, r) of
// a round are put in order first and then tested side by side, instead of each lane
// testing its own while the others wait (ShockHash<30, true>, 2M keys: leaf stage 4.8 -> 1.6 ms), four graphs
// peeled by groups of lanes (0.86 ms). M: 32-bit
// masks for L <= 32.
template <class M>
__device__ bool rotation_leaf(Sh1WarpSmem &sm, uint16_t *cells, int lane, uint32_t m, uint64_t seed0,
                              uint64_t cap_x, uint64_t &code) {
    const unsigned below = (1u << lane) - 1;
    uint32_t nA = 0, nB = 0;
    for (uint32_t k0 = 0; k0 < m; k0 += 32) {
        const uint32_t k = k0 + lane;
        const uint64_t key = k < m ? sm.keys[k] : 0;
        const bool even = (key & 1) == 0;
        const unsigned be = __ballot_sync(0xffffffffu, k < m && even), bo = __ballot_sync(0xffffffffu, k < m && !even);
        if (k < m) sm.fkeys[even ? nA + __popc(be & below) : m - 1 - (nB + __popc(bo & below))] = key;
        nA += __popc(be);
        nB += __popc(bo);
    }
    __syncwarp();
    const uint32_t gmask = m > 32 ? 7 : 0;
    const M all = (M)~(M)0 >> (8 * sizeof(M) - m);
    // Rounds of 32 seeds start at a multiple of 8 (seeds below seed0 in the first round take no
    // part), so with gmask = 7 each aligned group of 8 lanes shares set A's seed: its lanes hash
    // every eighth set-A key and OR their masks together.
    const uint64_t x_lo = seed0 & ~7ull, end = cap_x + (seed0 - x_lo);
    auto stage = [&](uint64_t at) {  // the keys for seeds x_lo + at, + at + 1, ...; how many they are good for
        uint32_t room = kSeedSpan;
        for (uint32_t k = lane; k < m; k += 32) {
            const uint64_t z = sm.fkeys[k] + x_lo + at;
            sm.staged[k] = seed_key(z);
            room = min(room, seed_room(z));
        }
        room = __reduce_min_sync(0xffffffffu, room);
        __syncwarp();
        return room;
    };
    uint64_t base0 = 0;
    uint32_t room = stage(0);
    uint16_t *const win = reinterpret_cast<uint16_t *>(sm.q);  // 32 covering pairs: lane << 8 | r
    for (uint64_t off = 0; off < end; off += 32) {
        const bool plain = off - base0 + 32 > room;  // some key's low bits run over in this round
        const uint32_t t = (uint32_t)(off - base0) + lane;
        const uint64_t x = x_lo + off + lane;
        const bool live = x >= seed0 && x - seed0 < cap_x;
        // cells[k * 32 + lane] = c1 | c2 << 8 of key k under the lane's seed; with gmask a set-A key's cells sit
        // in the slot of the group lane that hashed it
        auto hash = [&](uint32_t k, uint32_t mask) -> M {
            uint32_t c1, c2;
            if (plain) sh1_cells(sm.fkeys[k], x & ~(uint64_t)mask, m, c1, c2);
            else sh1_staged_cells(sm.staged[k], t & ~mask, m, c1, c2);
            cells[k * 32 + lane] = (uint16_t)(c1 | c2 << 8);
            return (M)1 << c1 | (M)1 << c2;
        };
        M a = 0, b = 0;
        if (gmask) {
            for (uint32_t k = lane & 7; k < nA; k += 8) a |= hash(k, gmask);
            a |= __shfl_xor_sync(0xffffffffu, a, 1);
            a |= __shfl_xor_sync(0xffffffffu, a, 2);
            a |= __shfl_xor_sync(0xffffffffu, a, 4);
        } else {
            for (uint32_t k = 0; k < nA; k++) a |= hash(k, 0);
        }
        for (uint32_t k = nA; k < m; k++) b |= hash(k, 0);
        M fits = 0;  // rotations with which the lane's seed covers all cells
        if (live)
            for (uint32_t r = 0; r < m; r++)
                if ((a | rot_bits(b, r, m, all)) == all) fits |= (M)1 << r;
        const uint32_t mine = sizeof(M) == 8 ? __popcll(fits) : __popc((uint32_t)fits);
        uint32_t incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t pos = incl - mine;  // of the lane's first pair still to be tested
        int src = -1, fr = 0;
        for (uint32_t q0 = 0; q0 < total && src < 0; q0 += 32) {
            for (; fits && pos < q0 + 32; pos++) {
                const uint32_t r = sizeof(M) == 8 ? __ffsll((long long)fits) - 1 : __ffs((int)fits) - 1;
                fits &= fits - 1;
                win[pos - q0] = (uint16_t)(lane << 8 | r);
            }
            __syncwarp();
            for (uint32_t q1 = 0; q1 < 32 && q0 + q1 < total && src < 0; q1 += 4) {
                const bool live = q0 + q1 + lane / 8 < total;
                const uint32_t w = live ? win[q1 + lane / 8] : 0, from = w >> 8, r = w & 0xFF;
                const bool ok = group_pseudoforest(m, live, [&](uint32_t k, uint32_t &c1, uint32_t &c2) {
                    const uint32_t c = cells[k * 32 + (k < nA && gmask ? (from & ~7u) | (k & 7) : from)];
                    c1 = c & 0xFF;
                    c2 = c >> 8;
                    if (k >= nA) {
                        c1 += r;
                        c2 += r;
                        if (c1 >= m) c1 -= m;
                        if (c2 >= m) c2 -= m;
                    }
                });
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                if (bal) {
                    src = __shfl_sync(0xffffffffu, from, __ffs(bal) - 1);
                    fr = __shfl_sync(0xffffffffu, r, __ffs(bal) - 1);
                }
            }
            __syncwarp();  // the window is read before it is written again
        }
        __syncwarp();  // the cells are read before the next round's are written
        if (src >= 0) {
            const uint64_t fx = x_lo + off + src - seed0;
            if (fx >= cap_x) return false;
            code = fx * m + (uint64_t)fr;
            // orientation: the reference's ordered insertion in set order, then cell order
            if (lane == 0) {
                const uint64_t xf = seed0 + fx;
                for (uint32_t c = 0; c < m; c++) sm.cell[c] = -1;
                bool okc = true;
                for (uint32_t k = 0; k < m && okc; k++) {
                    uint32_t c1, c2;
                    if (k < nA) {
                        sh1_cells(sm.fkeys[k], xf & ~(uint64_t)gmask, m, c1, c2);
                    } else {
                        sh1_cells(sm.fkeys[k], xf, m, c1, c2);
                        c1 = (c1 + fr) % m;
                        c2 = (c2 + fr) % m;
                    }
                    okc = cuckoo_insert(sm.cell, sm.xr, (int)k, c1, c2, 8 * (int)m + 16);
                }
                if (!okc) code = ~0ull;
            }
            code = __shfl_sync(0xffffffffu, code, 0);
            return code != ~0ull;
        }
        if (plain) {
            base0 = off + 32;
            room = stage(base0);
        }
    }
    return false;
}

// SPL: seeds per lane and round, or pairs of them with PAIRS (1 or 2; a tuning parameter, the same seed is found
// either way).
// PAIRS (sh1_pairs, below): the first sieve takes a key under two consecutive seeds at a time (sh1_half_pairs).
// BLOCK: the block's warps search a leaf together (not with rotation fitting): warp w takes the rounds w,
// w + kLeafWarps, ..., on its own, and goes on until its next round begins past the smallest passing seed
// any of them has found, so every smaller seed has been tried. One leaf then takes a quarter of the time,
// and with it the launch's tail, in which the last leaves run alone.
// Eight blocks per SM: 64 registers (72 without the bound: ShockHash<16>, 2M keys 0.53 instead of 0.49 ms; ten
// blocks, 48 registers: ShockHash<30>, 4M 9.3 instead of 9.1).
template <int SPL, bool BLOCK, bool PAIRS>
__global__ void __launch_bounds__(kLeafWarps * 32, 8) k_leaves_sh1(const Node *__restrict__ nodes, const uint32_t *__restrict__ ids,
                                                                uint32_t count, const uint64_t *__restrict__ keys,
                                                                uint64_t *__restrict__ codes, uint64_t *__restrict__ rib_keys,
                                                                uint8_t *__restrict__ rib_bits, uint64_t max_trials,
                                                                uint32_t *__restrict__ err, unsigned long long *__restrict__ work,
                                                                unsigned int *__restrict__ next_leaf, uint32_t rot_leaf) {
    __shared__ Sh1WarpSmem wsm[kLeafWarps];
    extern __shared__ uint16_t rot_cells[];  // rotation fitting only: [warp][64 keys][32 lanes]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Sh1WarpSmem &sm = wsm[warp];
    unsigned long long evals = 0;
    __shared__ unsigned long long block_best;  // BLOCK: smallest passing seed offset of the leaf so far
    __shared__ uint32_t block_leaf;
    for (;;) {
        uint32_t li = 0;
        if constexpr (BLOCK) {
            __syncthreads();
            if (threadIdx.x == 0) {
                block_leaf = atomicAdd(next_leaf, 1u);
                block_best = ~0ull;
            }
            __syncthreads();
            li = block_leaf;
        } else {
            if (lane == 0) li = atomicAdd(next_leaf, 1u);
            li = __shfl_sync(0xffffffffu, li, 0);
        }
        if (li >= count) break;
        const uint32_t id = ids[li];
        const Node nd = nodes[id];
        const uint32_t m = nd.m;
        for (uint32_t k = lane; k < m; k += 32) sm.keys[k] = keys[nd.start + k];
        __syncwarp();
        const uint64_t seed0 = start_seed(nd.level);
        // Coverage in two 32-bit halves: c1 < m/2 and c2 - m/2 < (m+1)/2, both <= 30 for m <= 60.
        const uint32_t h1 = m / 2, h2 = (m + 1) / 2;
        // (m = 1: fastrange32(., 0) = 0 always sets bit 0 of the empty first half; that cell is the
        // second half's cell 0, which c2 = 0 covers, so bit 0 counts as covered.)
        const uint32_t all1 = h1 ? (1u << h1) - 1 : 1u, all2 = (1u << h2) - 1;
        // ~2^(g+1) trials are expected; 2^(g+10) is only reached by duplicate keys.
        uint64_t cap = 1ull << min(nd.g + 10, 40);
        if (max_trials && max_trials < cap) cap = max_trials;
        if (!BLOCK && rot_leaf && m == rot_leaf) {
            // ~2^(g+1) codes x * L + r are expected; the cap counts seeds x
            uint64_t cap_x = (1ull << min(nd.g + 10, 40)) / m + 1;
            if (max_trials && max_trials < cap_x) cap_x = max_trials;
            uint64_t code = 0;
            const bool ok = m <= 32 ? rotation_leaf<uint32_t>(sm, rot_cells + warp * 64 * 32, lane, m, seed0, cap_x, code)
                                    : rotation_leaf<uint64_t>(sm, rot_cells + warp * 64 * 32, lane, m, seed0, cap_x, code);
            if (!ok) {
                if (lane == 0) atomicOr(err, code == ~0ull ? kErrInternal : kErrTrialLimit);
                continue;
            }
            if (lane == 0) {
                codes[id] = code;
                evals += (code / m + 1) * m;
            }
            __syncwarp();
            // retrieval input in cell order; the bit is the unrotated cell's half (ShockHash.h:384-391)
            for (uint32_t c = lane; c < m; c += 32) {
                const int e = sm.cell[c];
                const uint64_t key = e >= 0 ? sm.fkeys[e] : 0;
                const uint32_t r = (uint32_t)(code % m);
                const uint32_t cell = (key & 1) ? (c + m - r) % m : c;
                rib_keys[nd.start + c] = key;
                rib_bits[nd.start + c] = cell < m / 2 ? 0 : 1;
            }
            __syncwarp();
            continue;
        }
        uint64_t found = ~0ull;
        // queued survivors, tested four at a time in queue (= seed) order: the first passing one is
        // the smallest passing seed, as every smaller seed failed coverage or an earlier test
        const unsigned below = (1u << lane) - 1;
        uint32_t nq = 0;
        auto drain = [&]() {
            for (uint32_t q0 = 0; q0 < nq && found == ~0ull; q0 += 4) {
                const bool live = q0 + lane / 8 < nq;
                const uint64_t off = live ? sm.q[q0 + lane / 8] : 0;
                const bool pass = group_pseudoforest(
                    m, live, [&](uint32_t k, uint32_t &c1, uint32_t &c2) { sh1_cells(sm.keys[k], seed0 + off, m, c1, c2); });
                const unsigned bal = __ballot_sync(0xffffffffu, pass);
                if (bal) found = __shfl_sync(0xffffffffu, off, __ffs(bal) - 1);
            }
            nq = 0;
            __syncwarp();  // the queue's slots are read before the next round refills them
        };
        // the second sieve: the first n <= 32 waiting seeds, one per lane, against the first half's cells (and,
        // where the first sieve was not sure, the second half's). Waiting seeds are within the staged keys'
        // span, but for those of a round hashed in plain form.
        uint32_t nhalf = 0;
        uint64_t base0 = 0;  // the keys are staged for seed0 + base0 and the seeds after it
        auto cover = [&](uint32_t n, bool plain) {
            const uint64_t entry = (uint32_t)lane < n ? sm.half[lane] : base0, off = entry & ~kSh1Unsure;
            uint32_t c1m = 0;
            if (!plain) {
                const uint32_t t = (uint32_t)(off - base0);
#pragma unroll 4
                for (uint32_t k = 0; k < m; k++) c1m |= 1u << fastrange32(seed_lo(sm.staged[k], t), h1);
            }
            bool ok = (uint32_t)lane < n && (plain || c1m == all1);
            if (ok && (plain || (entry & kSh1Unsure))) {
                uint32_t c2m = 0;
                c1m = 0;
                for (uint32_t k = 0; k < m; k++) {
                    const uint64_t r = remix(sm.keys[k] + seed0 + off);
                    c1m |= 1u << fastrange32((uint32_t)r, h1);
                    c2m |= 1u << fastrange32((uint32_t)(r >> 32), h2);
                }
                ok = c1m == all1 && c2m == all2;
            }
            __syncwarp();
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (ok) sm.q[nq + __popc(bal & below)] = off;
            nq += __popc(bal);
            __syncwarp();  // the queue is written before other lanes read it
            // the rest moves up
            const uint32_t rest = nhalf - n;
            for (uint32_t i = 0; i < rest; i += 32) {
                const uint64_t v = i + lane < rest ? sm.half[n + i + lane] : 0;
                __syncwarp();
                if (i + lane < rest) sm.half[i + lane] = v;
                __syncwarp();
            }
            nhalf = rest;
            if (nq) drain();
        };
        // the keys staged for seeds seed0 + at, + at + 1, ...; how many such seeds they are good for
        uint32_t evens = 0;
        auto stage = [&](uint64_t at) {
            uint32_t room = kSeedSpan, odds = 0;
            if constexpr (!PAIRS) {
                for (uint32_t k = lane; k < m; k += 32) {
                    const uint64_t z = sm.keys[k] + seed0 + at;
                    sm.staged[k] = seed_key(z);
                    room = min(room, seed_room(z));
                }
                room = __reduce_min_sync(0xffffffffu, room);
                __syncwarp();
                return room;
            }
            evens = 0;
            for (uint32_t k0 = 0; k0 < m; k0 += 32) {
                const uint32_t k = k0 + lane;
                const uint64_t z = k < m ? sm.keys[k] + seed0 + at : 0;
                const unsigned be = __ballot_sync(0xffffffffu, k < m && !(z & 1)), bo = __ballot_sync(0xffffffffu, k < m && (z & 1));
                if (k < m) {
                    const uint32_t slot = z & 1 ? m - 1 - (odds + __popc(bo & below)) : evens + __popc(be & below);
                    const SeedKey key = seed_key(z);
                    const uint64_t d = key.fold & 1 ? 0ull - kRemixM1 : kRemixM1;
                    sm.staged[slot] = key;
                    sm.delta[slot] = make_uint2((uint32_t)d, (uint32_t)(d >> 32));
                    room = min(room, seed_room(z));
                }
                evens += __popc(be);
                odds += __popc(bo);
            }
            room = __reduce_min_sync(0xffffffffu, room);
            __syncwarp();
            return room;
        };
        uint32_t room = stage(0);
        const uint32_t batch = m <= kSh1SmallLeaf ? 1 : 32;
        // one shared-memory key read feeds the evaluations of all the lane's seeds
        constexpr int kIn = PAIRS ? 2 : 1, kLane = SPL * kIn;
        constexpr uint32_t kSeeds = PAIRS ? sh1_pair_seeds(SPL) : 32 * SPL, kStep = kSeeds * (BLOCK ? kLeafWarps : 1);
        for (uint64_t base = BLOCK ? kSeeds * warp : 0; base < cap && found == ~0ull; base += kStep) {
            // other warps lower block_best meanwhile, so lanes may read different values: the warp leaves as one
            if (BLOCK && __any_sync(0xffffffffu, base > *(volatile unsigned long long *)&block_best)) break;
            uint32_t mask[kLane], low[kLane];
#pragma unroll
            for (int i = 0; i < kLane; i++) mask[i] = 0, low[i] = ~0u;
            const bool plain = base - base0 + 32 * kLane > room;
            if (!plain) {
                if constexpr (!PAIRS) sh1_half_masks<SPL>(sm.staged, m, h2, (uint32_t)(base - base0) + lane, mask, low);
                else sh1_half_pairs<SPL>(sm.staged, sm.delta, evens, m, h2, (uint32_t)(base - base0), mask, low);
            } else {  // some key's low bits run over in this round
                for (uint32_t k = 0; k < m; k++)
#pragma unroll
                    for (int i = 0; i < kLane; i++) {
                        const uint64_t x = seed0 + base + 32 * kIn * (i / kIn) + kIn * lane + i % kIn;
                        mask[i] |= 1u << fastrange32((uint32_t)(remix(sm.keys[k] + x) >> 32), h2);
                    }
            }
#pragma unroll
            for (int p = 0; p < SPL; p++) {  // seeds in order: all lanes' p-th seed or pair before the next
                const uint32_t first = kIn * (32 * p + lane);
                bool ok[kIn];
                uint32_t pos = nhalf;
#pragma unroll
                for (int i = 0; i < kIn; i++) {
                    ok[i] = first + i < kSeeds && sh1_half_passes(mask[kIn * p + i], low[kIn * p + i], all2, h2);
                    const unsigned bal = __ballot_sync(0xffffffffu, ok[i]);
                    pos += __popc(bal & below);
                    nhalf += __popc(bal);
                }
#pragma unroll
                for (int i = 0; i < kIn; i++)
                    if (ok[i]) {
                        const bool sure = (mask[kIn * p + i] & all2) == all2 && low[kIn * p + i] >= 2 * h2;
                        sm.half[pos++] = (base + first + i) | (sure ? 0 : kSh1Unsure);
                    }
            }
            __syncwarp();
            while (found == ~0ull && nhalf >= (plain ? 1 : batch)) cover(min(nhalf, 32u), plain);
            if (plain) {
                base0 = base + kStep;
                room = stage(base0);
            }
        }
        while (found == ~0ull && nhalf) cover(min(nhalf, 32u), false);  // what still waits (the trial limit, or BLOCK)
        if (found == ~0ull && nq) drain();
        if constexpr (BLOCK) {
            if (lane == 0 && found != ~0ull) atomicMin(&block_best, (unsigned long long)found);
            __syncthreads();
            found = block_best;
            if (warp) continue;  // one warp writes the leaf's products
        }
        if (found == ~0ull || found >= cap) {
            if (lane == 0) atomicOr(err, kErrTrialLimit);
            continue;
        }
        // Orientation: the reference's ordered cuckoo insertion (construct, TinyBinaryCuckooHashTable.h:80-106).
        if (lane == 0) {
            const uint64_t x = seed0 + found;
            for (uint32_t c = 0; c < m; c++) sm.cell[c] = -1;
            bool okc = true;
            for (uint32_t k = 0; k < m && okc; k++) {
                uint32_t c1, c2;
                sh1_cells(sm.keys[k], x, m, c1, c2);
                okc = cuckoo_insert(sm.cell, sm.xr, (int)k, c1, c2, 8 * (int)m + 16);
            }
            if (!okc) atomicOr(err, kErrInternal);
            codes[id] = found;
            evals += (found + 1) * m;
        }
        __syncwarp();
        // Retrieval input in cell order: key in cell i, bit (i >= m/2) (ShockHash.h:425-428).
        for (uint32_t c = lane; c < m; c += 32) {
            const int e = sm.cell[c];
            rib_keys[nd.start + c] = e >= 0 ? sm.keys[e] : 0;
            rib_bits[nd.start + c] = c >= m / 2 ? 1 : 0;
        }
        __syncwarp();
    }
    if (lane == 0 && evals) atomicAdd(&work[1], evals);
}

int leaves_sh1_warps_per_block() { return kLeafWarps; }

// Whether the first sieve works on pairs of seeds: a seed costs it less, but a round has twice the seeds, and
// a leaf's last round (last four with a block per leaf) is half wasted; staging costs more, too. It pays
// where a leaf takes many rounds. Leaf stage, single seeds / pairs: a warp per leaf, leaves of 24 keys (2M
// keys) 1.73 / 1.91 ms, 26 (4M) 4.76 / 4.92, 28 (4M) 7.04 / 7.02, 29 (4M) 8.81 / 8.65, 30 (1M) 3.23 / 3.14, 30 (4M)
// 11.15 / 10.88, 33 (8M) 45.3 / 43.7; a block per leaf, 32 (1M) 6.18 / 6.72, 33 (1M) 7.63 / 7.88, 34 (1M) 9.35 / 9.15,
// 35 (1M) 11.99 / 11.38, 40 (30,000 keys) 3.9 / 3.4, 40 (1M) 42.1 / 39.1, 48 (20,000) 30.4 / 26.5.
static bool sh1_pairs(int leaf, bool block) { return block ? leaf >= 34 : leaf >= 29; }

void launch_leaves_sh1_ctr(const Node *nodes, const uint32_t *ids, uint32_t count, const uint64_t *keys, uint64_t *codes,
                           uint64_t *rib_keys, uint8_t *rib_bits, uint64_t max_trials, uint32_t *err,
                           unsigned long long *work, unsigned int *ctr, int grid, cudaStream_t s, uint32_t rot_leaf,
                           int spl, bool block, int leaf) {
    if (!count) return;
    block = block && !rot_leaf;
    cudaMemsetAsync(ctr, 0, sizeof(unsigned int), s);
    const size_t dyn = rot_leaf ? (size_t)kLeafWarps * 64 * 32 * sizeof(uint16_t) : 0;  // 16 KB per block
    const bool pairs = !rot_leaf && sh1_pairs(leaf, block);
    auto kernel = block ? (pairs ? (spl == 1 ? k_leaves_sh1<1, true, true> : k_leaves_sh1<2, true, true>)
                                 : (spl == 1 ? k_leaves_sh1<1, true, false> : k_leaves_sh1<2, true, false>))
                        : (pairs ? (spl == 1 ? k_leaves_sh1<1, false, true> : k_leaves_sh1<2, false, true>)
                                 : (spl == 1 ? k_leaves_sh1<1, false, false> : k_leaves_sh1<2, false, false>));
    kernel<<<grid, kLeafWarps * 32, dyn, s>>>(nodes, ids, count, keys, codes, rib_keys, rib_bits, max_trials, err, work, ctr,
                                              rot_leaf);
}

} // namespace shg
