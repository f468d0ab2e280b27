// RecSplit split-seed search and stable partition, one launch per tree level (one block per node);
// the node's search is split_node in shg_split.cuh.
#include "shg_split.cuh"

namespace shg {

template <int SPL, int THREADS, bool SIMD, bool STRIPED>
__global__ void __launch_bounds__(THREADS) k_split(const Node *__restrict__ nodes, const uint32_t *__restrict__ ids,
                                                   uint64_t *__restrict__ keys, uint64_t *__restrict__ codes,
                                                   uint64_t max_trials, uint32_t *__restrict__ err,
                                                   unsigned long long *__restrict__ work,
                                                   unsigned long long *__restrict__ kind_work, int round_div,
                                                   uint32_t stripes, SplitBest *best) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    SplitSmem<SPL, THREADS, SIMD> &sm = *reinterpret_cast<SplitSmem<SPL, THREADS, SIMD> *>(smem_raw);
    const uint32_t i = STRIPED ? blockIdx.x / stripes : blockIdx.x;
    const uint32_t id = ids[i];
    split_node<SPL, THREADS, SIMD, false, STRIPED>(sm, nodes[id], id, keys, codes, max_trials, err, work, kind_work, round_div,
                                                   SplitStripe{blockIdx.x - i * stripes, stripes, best + i});
}

template <int SPL, int THREADS, bool SIMD>
static void launch_split_t(const Node *nodes, const uint32_t *ids, uint32_t count, uint64_t *keys, uint64_t *codes,
                           uint64_t max_trials, uint32_t *err, unsigned long long *work, unsigned long long *kind_work,
                           uint32_t max_m, int round_div, uint32_t stripes, SplitBest *best, cudaStream_t s) {
    // A launch takes memory for its largest node. The limit, though, is an attribute of the kernel on the device,
    // and engines in other threads launch the same kernel: every launch sets the same value, room for any node.
    const size_t smem = split_smem_bytes<SPL, THREADS, SIMD>(max_m);
    auto kernel = stripes > 1 ? k_split<SPL, THREADS, SIMD, true> : k_split<SPL, THREADS, SIMD, false>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SplitSmem<SPL, THREADS, SIMD>));
    kernel<<<count * stripes, THREADS, smem, s>>>(nodes, ids, keys, codes, max_trials, err, work, kind_work, round_div, stripes,
                                                  best);
}

// Parameters a tuning table may set (the SIMDShockHash form is chosen by the engine, not the table).
bool split_tuning_valid(int spl, int threads, int round_div, int arith) {
    return (spl == 1 || spl == 2 || spl == 4) && (threads == 128 || threads == 256 || threads == 512) && round_div >= 1 &&
           round_div <= 64 && (arith == 0 || arith == 1);
}

void launch_split_level(const Node *nodes, const uint32_t *ids, uint32_t count, uint64_t *keys, uint64_t *codes,
                        uint64_t max_trials, uint32_t *err, unsigned long long *work, unsigned long long *kind_work,
                        uint32_t max_m, const SplitTuning &t, uint32_t stripes, SplitBest *best, cudaStream_t s) {
    if (!count) return;
    const bool simd = t.arith == kSplitArithSimd;
    // Nodes of at most 128 keys: half the threads (unless the table asks for another number), at least one for each
    // key. Their blocks spend their time on the prologue, two or three rounds and the partition, so what counts is how many
    // nodes an SM holds. Splits stage, 256 / 128 threads: ShockHash<2>, b = 200, 1M keys 3.24 / 1.95 ms, ShockHash<8>, b = 1000, 1M 1.21 / 0.88,
    // ShockHash<16>, b = 400, 1M 0.66 / 0.56, ShockHash2<64>, 4M 14.3 / 14.2. Up to 256 keys: ShockHash2<64>, 1M 4.85 instead of
    // 4.67; up to 512: ShockHash2<16>, 30,000 keys 0.18 instead of 0.15.
    if (t.threads == SplitTuning().threads && max_m <= 128)
        return launch_split_level(nodes, ids, count, keys, codes, max_trials, err, work, kind_work, max_m,
                                  SplitTuning{t.spl, 128, t.round_div, t.arith}, stripes, best, s);
#define SHG_SPLIT_CASE(SPL, TH)                                                                                      \
    if (t.spl == SPL && t.threads == TH)                                                                            \
        return simd ? launch_split_t<SPL, TH, true>(nodes, ids, count, keys, codes, max_trials, err, work, kind_work, \
                                                    max_m, t.round_div, stripes, best, s)                                          \
                    : launch_split_t<SPL, TH, false>(nodes, ids, count, keys, codes, max_trials, err, work, kind_work, \
                                                     max_m, t.round_div, stripes, best, s);
    SHG_SPLIT_CASE(1, 128) SHG_SPLIT_CASE(1, 256) SHG_SPLIT_CASE(1, 512)
    SHG_SPLIT_CASE(2, 128) SHG_SPLIT_CASE(2, 256) SHG_SPLIT_CASE(2, 512)
    SHG_SPLIT_CASE(4, 128) SHG_SPLIT_CASE(4, 256) SHG_SPLIT_CASE(4, 512)
#undef SHG_SPLIT_CASE
    launch_split_level(nodes, ids, count, keys, codes, max_trials, err, work, kind_work, max_m,
                       SplitTuning{2, 256, t.round_div, t.arith}, stripes, best, s);  // other values: the default shape
}

} // namespace shg
