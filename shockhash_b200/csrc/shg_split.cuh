// RecSplit split-seed search and stable partition of one node (ShockHash.h:451-547,
// ShockHash2.h:290-386), shared by the per-level split kernel (shg_split.cu) and the work-queue
// kernel (shg_leaves_sh2.cu).
//
// One thread block per split node. The node's keys (<= 3000 x 8 B) sit in shared memory and are
// read as warp-wide broadcasts; each lane owns SPL consecutive-in-round seeds and keeps
// per-seed part counts in registers. A seed x is valid when every part but the last receives
// exactly its size under  part(k) = remap16(remix(k + x), m) / unit  (fanout 2: h >= split).
//
// The part test never multiplies: h = (r16 * m) >> 16 < K  <=>  r16 < ceil(K * 65536 / m) with
// r16 the low 16 bits of remix, so each part boundary becomes one 16-bit threshold and only the
// low 47 bits of remix's second product are needed.
//
// What bounds it: the integer pipes (ALU and multiply-add, each half a warp instruction per cycle and
// scheduler). So the loop is laid out for the fewest instructions on the busier of the two:
//   * keys are staged as SeedKey (shg_common.cuh), which takes remix's first xor-shift and the high
//     half of its first product out of the loop;
//   * counts are not added up per key: a key leaves one bit per threshold (or its two-bit quarter) in a
//     word, and the bits of 32 (16) keys are counted at once with popc.
// Per seed and key that is about 17 pipe slots (8 ALU, 9 multiply-add) where the plain 64-bit form took
// about 24 (14 ALU), measured on the quarter loop alone: 1026 -> 1671 G evaluations/s.
//
// Rounds: the block evaluates 32*SPL*G seeds per round (SPL seeds per lane, G warp groups; a
// group's warps split the node's keys and merge counts in shared memory). G is picked from the
// node's expected trial count 1/p (the same p the Golomb-Rice memo uses) so that a round stays near
// 1/round_div of it and the overshoot past the answer stays small. The smallest valid seed of the
// first round that has one is the answer, identical to the reference's sequential `for (;;) x++`
// search, for every choice of SPL, block size and round_div (the tuning parameters).
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>
#include "shg_common.cuh"
#include "shg_internal.h"

namespace shg {

// A node's key as the search loop reads it: ShockHash and ShockHash2 (SIMD = false) split by remix,
// SIMDShockHash by fmix32 of the xor of the halves of z = key + seed. z() is the staged z again,
// low16(z) the hash in its plain form, quarter(t) a word with the hash's two top bits under z + t as
// its own top bits (top(t): all 16 of them).
template <bool SIMD> struct SplitKey : SeedKey {
    __device__ __forceinline__ static SplitKey make(uint64_t z) { return SplitKey{seed_key(z)}; }
    __device__ __forceinline__ uint64_t z() const { return seed_key_z(*this); }
    __device__ __forceinline__ static uint32_t low16(uint64_t z) { return remix_low16(z); }
    __device__ __forceinline__ uint32_t quarter(uint32_t t) const {
        uint32_t a, b;
        seed_quarter_at<31>(*this, t, a, b);
        return a ^ b;
    }
};
template <> struct alignas(8) SplitKey<true> {
    uint32_t lo, hi;  // the halves of z: adding t leaves the high one alone while seed_room lasts
    __device__ __forceinline__ static SplitKey make(uint64_t z) { return SplitKey{(uint32_t)z, (uint32_t)(z >> 32)}; }
    __device__ __forceinline__ uint64_t z() const { return (uint64_t)hi << 32 | lo; }
    __device__ __forceinline__ static uint32_t low16(uint64_t z) { return simd_split_low16(z); }
    __device__ __forceinline__ uint32_t quarter(uint32_t t) const { return top(t); }
    __device__ __forceinline__ uint32_t top(uint32_t t) const {  // fmix32, its last xor-shift at bits 16..31
        uint32_t y = (lo + t) ^ hi;
        y ^= y >> 16;
        y *= 0x85ebca6bu;
        y ^= y >> 13;
        return (y * 0xc2b2ae35u) ^ (y * (0xc2b2ae35u << 16));
    }
};

template <int SPL, int THREADS, bool SIMD> struct SplitSmem {
    static constexpr int kWarps = THREADS / 32;
    uint32_t part_counts[kWarps][32 * SPL][3];
    uint64_t scan[kWarps];
    uint32_t best[2];   // smallest valid seed slot of a round, by the round's parity
    uint32_t stop[2];   // striped search: no smaller seed can come from this block's next rounds
    uint32_t last;      // striped search: this block is the last of the node's to be done (not `stop`, which a late
                        // warp may still have to read)
    uint64_t found;     // striped search, in the node's last block: the smallest seed of all its blocks
    uint32_t room;      // smallest seed_room of the staged keys
    SplitKey<SIMD> keys[kMaxBucket];  // last: a launch takes memory for the keys of its largest node only
};
template <int SPL, int THREADS, bool SIMD> inline size_t split_smem_bytes(uint32_t max_m) {
    using S = SplitSmem<SPL, THREADS, SIMD>;
    return sizeof(S) - (size_t)(kMaxBucket - (int)max_m) * sizeof(SplitKey<SIMD>);
}

// Counts of keys below each of NT thresholds, for SPL seeds t0, t0 + 32, ..., over keys [lo, hi).
template <int NT, int SPL, bool SIMD>
__device__ __forceinline__ void count_range(const SplitKey<SIMD> *__restrict__ sk, uint32_t lo, uint32_t hi, uint32_t t0,
                                            const uint32_t T0, const uint32_t T1, const uint32_t T2,
                                            uint32_t (&c)[SPL][3]) {
    const uint32_t T[3] = {T0, T1, T2};
    if constexpr (SIMD) {
#pragma unroll 4
        for (uint32_t i = lo; i < hi; i++) {
            const SplitKey<SIMD> k = sk[i];
#pragma unroll
            for (int s = 0; s < SPL; s++) {
                const uint32_t v = k.top(t0 + 32 * s);
#pragma unroll
                for (int t = 0; t < NT; t++) c[s][t] += v < T[t] << 16;
            }
        }
    } else {
        // the hash at bits 15..30 and bit 31 clear: hash < T is the sign bit of v - (T << 15), which a
        // funnel shift appends to a word of up to 32 keys' bits
        for (uint32_t i = lo; i < hi;) {
            const uint32_t end = min(hi, i + 32);
            uint32_t w[SPL][NT] = {};
#pragma unroll 4
            for (; i < end; i++) {
                const SplitKey<SIMD> k = sk[i];
#pragma unroll
                for (int s = 0; s < SPL; s++) {
                    const uint32_t v = seed_low16_at30(k, t0 + 32 * s);
#pragma unroll
                    for (int t = 0; t < NT; t++) w[s][t] = __funnelshift_l(v - (T[t] << 15), w[s][t], 1);
                }
            }
#pragma unroll
            for (int s = 0; s < SPL; s++)
#pragma unroll
                for (int t = 0; t < NT; t++) c[s][t] += __popc(w[s][t]);
        }
    }
}

// Quarter split (fanout 4 with m = 4 * unit, every full first-level node): the thresholds are
// k * 16384, so a key's part is the hash's two top bits b1 b0. The sums of b0, of b1 and of b0 & b1 over
// the keys fix the four part counts; they are (2u, 2u, u) exactly when every part gets u keys. Each
// stays at or below m <= 4 * 128, so one word holds the three, 10 bits each.
__device__ __forceinline__ uint32_t quarter_tally(uint32_t w) {  // w: up to 16 keys' (b1, b0), zeros elsewhere
    const uint32_t b0 = w & 0x55555555u, b1 = (w >> 1) & 0x55555555u;
    return __popc(b0) + (__popc(b1) << 10) + (__popc(b0 & b1) << 20);
}
__device__ __forceinline__ uint32_t quarter_need(uint32_t u) { return 2 * u | 2 * u << 10 | u << 20; }

template <int J, int SPL>  // keys J .. 7 of a group of eight: their bits to positions 16 + 2 J ... of w
__device__ __forceinline__ void quarter_eight(const SplitKey<false> *__restrict__ sk, uint32_t t0, uint32_t (&w)[SPL]) {
    if constexpr (J < 8) {
        const SplitKey<false> k = sk[J];
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            uint32_t a, b;
            seed_quarter_at<17 + 2 * J>(k, t0 + 32 * s, a, b);
            w[s] |= (a ^ b) & (3u << (16 + 2 * J));
        }
        quarter_eight<J + 1, SPL>(sk, t0, w);
    }
}

template <int SPL, bool SIMD>
__device__ __forceinline__ void quarter_range(const SplitKey<SIMD> *__restrict__ sk, uint32_t lo, uint32_t hi, uint32_t t0,
                                              uint32_t (&c)[SPL][3]) {
    uint32_t i = lo;
    if constexpr (!SIMD) {
        // sixteen keys per step, each key's bits multiplied straight to their place in the word: an
        // and-xor and half an or per key, where appending them with a funnel shift takes an xor and
        // a shift (1634 against 1671 G evaluations/s)
        for (; i + 16 <= hi; i += 16) {
            uint32_t w0[SPL] = {}, w1[SPL] = {};
            quarter_eight<0, SPL>(sk + i, t0, w0);
            quarter_eight<0, SPL>(sk + i + 8, t0, w1);
#pragma unroll
            for (int s = 0; s < SPL; s++) c[s][0] += quarter_tally(w0[s] >> 16 | w1[s]);
        }
    }
    while (i < hi) {
        const uint32_t end = min(hi, i + 16);
        uint32_t w[SPL] = {};
#pragma unroll 4
        for (; i < end; i++) {
            const SplitKey<SIMD> k = sk[i];
#pragma unroll
            for (int s = 0; s < SPL; s++) w[s] = __funnelshift_l(k.quarter(t0 + 32 * s), w[s], 2);
        }
#pragma unroll
        for (int s = 0; s < SPL; s++) c[s][0] += quarter_tally(w[s]);
    }
}

// The same counts in plain 64-bit arithmetic, for a round in which some key's low bits run over
// (t0 may then be beyond its seed_room). NT = 4: quarter split.
template <int NT, int SPL, bool SIMD>
__device__ __noinline__ void count_plain(const SplitKey<SIMD> *__restrict__ sk, uint32_t lo, uint32_t hi, uint64_t t0,
                                         const uint32_t T0, const uint32_t T1, const uint32_t T2, uint32_t (&c)[SPL][3]) {
    const uint32_t T[3] = {T0, T1, T2};
    for (uint32_t i = lo; i < hi; i++) {
        const uint64_t z = sk[i].z() + t0;
#pragma unroll
        for (int s = 0; s < SPL; s++) {
            const uint32_t r = SplitKey<SIMD>::low16(z + 32 * s);
            if constexpr (NT == 4) {
                c[s][0] += quarter_tally(r >> 14);
            } else {
#pragma unroll
                for (int t = 0; t < NT; t++) c[s][t] += r < T[t];
            }
        }
    }
}

// Sets sm.room from the keys in each thread's share (sm.room holds kSeedSpan before; all threads).
template <class Smem> __device__ __forceinline__ void merge_room(Smem &sm, uint32_t room) {
    room = __reduce_min_sync(0xffffffffu, room);
    if ((threadIdx.x & 31) == 0 && room < kSeedSpan) atomicMin(&sm.room, room);
}

// A node searched by several blocks (its stripes): block `index` of `count` takes every count-th round and
// stops once its next round begins past the smallest valid seed that any of them has found. So every
// smaller seed has been tried when the last of them is done, and that block (nobody waits for another)
// partitions the node.
struct SplitStripe {
    uint32_t index, count;
    SplitBest *node;  // zero before the launch
};

// Smallest valid trial index (seed - seed0), or ~0 when `cap` trials were exhausted. The keys are
// staged for seeds seed0 + base0, base0 + 1, ... (base0: 0 on entry, moved on when a key's low bits run
// over). NT = number of part thresholds compared (1..3); NT = 4 selects the quarter split. STRIPED: the
// smallest among this block's rounds, or ~0 when another block's seed makes the search end.
template <int NT, bool STRIPED, int SPL, int THREADS, bool SIMD>
__device__ __forceinline__ uint64_t search_seeds(SplitSmem<SPL, THREADS, SIMD> &sm, uint32_t m, const uint32_t T0, const uint32_t T1,
                                 const uint32_t T2, const uint32_t N0, const uint32_t N1, const uint32_t N2, int G,
                                 uint64_t cap, uint64_t &base0, const SplitStripe &stripe) {
    constexpr int kWarps = THREADS / 32, kSeedsPerWarp = 32 * SPL;
    constexpr int NC = NT == 4 ? 1 : NT;  // counters per seed
    const uint32_t need[3] = {N0, N1, N2};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpg = kWarps / G;  // warps per group
    const int group = warp / wpg, sub = warp % wpg;
    const uint32_t lo = (uint32_t)((uint64_t)m * sub / wpg), hi = (uint32_t)((uint64_t)m * (sub + 1) / wpg);
    const uint32_t per_round = (uint32_t)(kSeedsPerWarp * G);
    const uint32_t slot0 = (uint32_t)group * kSeedsPerWarp + lane;  // seed slot s is slot0 + 32 s
    uint32_t room = sm.room, parity = 0;
    const uint64_t step = STRIPED ? (uint64_t)per_round * stripe.count : per_round;
    for (uint64_t base = STRIPED ? (uint64_t)per_round * stripe.index : 0; base < cap; base += step) {
        uint32_t c[SPL][3] = {};
        const uint64_t at = base - base0;
        const bool plain = at + per_round > room;
        if (plain) count_plain<NT, SPL, SIMD>(sm.keys, lo, hi, at + slot0, T0, T1, T2, c);
        else if constexpr (NT == 4) quarter_range<SPL, SIMD>(sm.keys, lo, hi, (uint32_t)at + slot0, c);
        else count_range<NT, SPL, SIMD>(sm.keys, lo, hi, (uint32_t)at + slot0, T0, T1, T2, c);
        if (wpg > 1) {
#pragma unroll
            for (int s = 0; s < SPL; s++)
#pragma unroll
                for (int t = 0; t < NC; t++) sm.part_counts[warp][s * 32 + lane][t] = c[s][t];
            __syncthreads();
            if (sub == 0) {
#pragma unroll
                for (int s = 0; s < SPL; s++)
#pragma unroll
                    for (int t = 0; t < NC; t++) {
                        uint32_t tot = 0;
                        for (int w = 0; w < wpg; w++) tot += sm.part_counts[warp + w][s * 32 + lane][t];
                        c[s][t] = tot;
                    }
            }
        }
        if (sub == 0) {
#pragma unroll
            for (int s = 0; s < SPL; s++) {
                bool ok = true;
#pragma unroll
                for (int t = 0; t < NC; t++) ok &= c[s][t] == need[t];
                if (ok) atomicMin(&sm.best[parity], slot0 + 32u * s);
            }
        }
        if (STRIPED && threadIdx.x == 0)
            sm.stop[parity] = ~*(volatile unsigned long long *)&stripe.node->inv_best <= base + step;
        __syncthreads();
        const uint32_t b = sm.best[parity];
        if (b != 0xffffffffu) return base + b < cap ? base + b : ~0ull;  // at most `cap` seeds count
        if (STRIPED && sm.stop[parity]) return ~0ull;
        parity ^= 1;  // a warp that is ahead writes the other word while this one is still read
        if (plain) {  // stage the keys again from the next round's first seed on
            if (threadIdx.x == 0) sm.room = kSeedSpan;
            __syncthreads();
            uint32_t mine = kSeedSpan;
            for (uint32_t i = threadIdx.x; i < m; i += THREADS) {
                const uint64_t z = sm.keys[i].z() + at + step;
                sm.keys[i] = SplitKey<SIMD>::make(z);
                mine = min(mine, seed_room(z));
            }
            merge_room(sm, mine);
            __syncthreads();
            room = sm.room;
            base0 = base + step;
        }
    }
    return ~0ull;
}

// One split node searched and partitioned by the whole block (THREADS threads): the smallest valid
// seed from start_seed[level] on, its code x - start_seed to codes[id], the node's keys permuted in
// place into its parts. Returns (block-uniformly) after the partition's writes are issued; a node
// whose search reaches its trial cap sets kErrTrialLimit and leaves its keys as they were.
// L2: load the node's keys past L1 (needed when another SM may have rewritten them since this SM
// last read those lines, as in the work-queue kernel; the per-level launches start with clean L1s).
// STRIPED: the calling block is one stripe of the node's search.
template <int SPL, int THREADS, bool SIMD, bool L2 = false, bool STRIPED = false>
__device__ __forceinline__ void split_node(SplitSmem<SPL, THREADS, SIMD> &sm, const Node nd, const uint32_t id,
                                           uint64_t *__restrict__ keys, uint64_t *__restrict__ codes,
                                           const uint64_t max_trials, uint32_t *__restrict__ err,
                                           unsigned long long *__restrict__ work,
                                           unsigned long long *__restrict__ kind_work, const int round_div,
                                           SplitStripe stripe = SplitStripe{0, 1, nullptr}) {
    constexpr int kWarps = THREADS / 32, kSeedsPerWarp = 32 * SPL;
    const uint32_t m = nd.m;
    const uint64_t seed0 = start_seed(nd.level);
    auto stage = [&]() {
        if (threadIdx.x == 0) {
            sm.best[0] = sm.best[1] = 0xffffffffu;
            sm.room = kSeedSpan;
        }
        __syncthreads();
        uint32_t room = kSeedSpan;
        for (uint32_t i = threadIdx.x; i < m; i += THREADS) {
            const uint64_t z = (L2 ? __ldcg(&keys[nd.start + i]) : keys[nd.start + i]) + seed0;
            sm.keys[i] = SplitKey<SIMD>::make(z);
            room = min(room, seed_room(z));
        }
        merge_room(sm, room);
    };
    if constexpr (!STRIPED) stage();  // a stripe first finds out whether it takes part

    // Part boundaries as thresholds on the low 16 bits of remix (see header).
    uint32_t T[3] = {65536u, 65536u, 65536u}, need[3] = {m, m, m};
    int NT;
    double p;
    if (nd.kind == kSplit2) {
        NT = 1;
        T[0] = (uint32_t)(((uint64_t)nd.unit * 65536u + m - 1) / m);
        need[0] = nd.unit;
        const double k0 = nd.unit, k1 = m - nd.unit;
        p = sqrt((double)m) / (sqrt(2 * M_PI) * sqrt(k0) * sqrt(k1));
    } else {
        NT = nd.fanout - 1;
        double sp = 1;
        for (int t = 0; t < NT; t++) {
            const uint64_t K = (uint64_t)(t + 1) * nd.unit;
            T[t] = (uint32_t)((K * 65536u + m - 1) / m);
            need[t] = (uint32_t)K;
            sp *= sqrt((double)nd.unit);
        }
        sp *= sqrt((double)(m - (uint32_t)NT * nd.unit));
        p = sqrt((double)m) / (pow(2 * M_PI, NT / 2.0) * sp);
    }
    // Warp groups: aim for a round (of all stripes together) of ~1/round_div of the expected trials. A stripe
    // for which fewer than two rounds of the smallest size are expected takes no part.
    double expect = 1.0 / p;
    if constexpr (STRIPED) {
        stripe.count = min(stripe.count, max(1u, (uint32_t)(expect / (2 * kSeedsPerWarp))));
        if (stripe.index >= stripe.count) return;
        expect /= stripe.count;
    }
    if constexpr (STRIPED) stage();
    int G = 1;
    while (G < kWarps && (double)(kSeedsPerWarp * G * 2) * (double)round_div <= expect) G <<= 1;
    __syncthreads();

    // Trial cap: 2^(g+12) is ~2000 expected searches (g ~ log2(0.48 / p)), so only duplicate keys
    // or a caller-set max_trials can reach it.
    uint64_t cap = 1ull << min(nd.g + 12, 40);
    if (max_trials && max_trials < cap) cap = max_trials;
    uint64_t trial, base0 = 0;
    const bool quarter = nd.kind == kSplitK && nd.fanout == 4 && m == 4u * nd.unit;
    if (quarter) {
        NT = 4;
        need[0] = quarter_need(nd.unit);
    }
    switch (NT) {
        case 1: trial = search_seeds<1, STRIPED>(sm, m, T[0], T[1], T[2], need[0], need[1], need[2], G, cap, base0, stripe); break;
        case 2: trial = search_seeds<2, STRIPED>(sm, m, T[0], T[1], T[2], need[0], need[1], need[2], G, cap, base0, stripe); break;
        case 3: trial = search_seeds<3, STRIPED>(sm, m, T[0], T[1], T[2], need[0], need[1], need[2], G, cap, base0, stripe); break;
        default: trial = search_seeds<4, STRIPED>(sm, m, T[0], T[1], T[2], need[0], need[1], need[2], G, cap, base0, stripe); break;
    }
    if constexpr (STRIPED) {
        if (threadIdx.x == 0) {
            if (trial != ~0ull) atomicMax(&stripe.node->inv_best, ~trial);
            __threadfence();  // the seed before the count of finished blocks
            const bool last = atomicAdd(&stripe.node->done, 1u) == stripe.count - 1;
            __threadfence();
            sm.last = last;
            if (last) sm.found = ~atomicMax(&stripe.node->inv_best, 0ull);
        }
        __syncthreads();
        if (!sm.last) return;
        trial = sm.found;
    }
    if (trial == ~0ull) {
        if (threadIdx.x == 0) atomicOr(err, kErrTrialLimit);
        return;
    }
    // from here on z + off is a key under its node's seed, and z - back the key itself
    const uint64_t off = trial - base0, back = seed0 + base0;

    // Stable partition (counting sort by part, original order inside a part). Each thread owns a
    // contiguous chunk; per-part counts are packed 16 bits per part into one 64-bit word and
    // exclusive-scanned across the block.
    const uint32_t chunk = (m + THREADS - 1) / THREADS;
    const uint32_t lo = min(m, threadIdx.x * chunk), hi = min(m, lo + chunk);
    uint64_t mine = 0;
    for (uint32_t i = lo; i < hi; i++) {
        const uint32_t r = SplitKey<SIMD>::low16(sm.keys[i].z() + off);
        const uint32_t part = (r >= T[0]) + (r >= T[1]) + (r >= T[2]);
        mine += 1ull << (16 * part);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();  // sm.scan reuse
    if (lane == 31) sm.scan[warp] = incl;
    __syncthreads();
    uint64_t before = 0;
    for (int w = 0; w < warp; w++) before += sm.scan[w];
    uint64_t run = before + incl - mine;  // exclusive prefix, packed
    const uint32_t unit = nd.unit;
    for (uint32_t i = lo; i < hi; i++) {
        const uint64_t z = sm.keys[i].z();
        const uint32_t r = SplitKey<SIMD>::low16(z + off);
        const uint32_t part = (r >= T[0]) + (r >= T[1]) + (r >= T[2]);
        const uint32_t dest = part * unit + (uint32_t)((run >> (16 * part)) & 0xFFFF);
        run += 1ull << (16 * part);
        if (dest < m) keys[nd.start + dest] = z - back;
        else atomicOr(err, kErrInternal);  // unreachable for a valid seed; never write outside the node
    }
    if (threadIdx.x == 0) {
        codes[id] = trial;  // x - start_seed[level]
        atomicAdd(work, (unsigned long long)(trial + 1) * m);
        // useful evaluations by inner loop: 1, 2 or 3 compared thresholds, or the quarter split
        atomicAdd(&kind_work[quarter ? 3 : NT - 1], (unsigned long long)(trial + 1) * m);
    }
}

} // namespace shg
