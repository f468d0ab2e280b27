// Device code on the host, for tests of its synchronisation: every CUDA thread is a fiber that runs until
// its next barrier or warp operation, and a seeded scheduler picks which one runs next. So any order that the
// language allows between two barriers can occur, the threads of a warp one by one included. A run ends with
// an error when the lanes of a warp, or the threads of a block, do not arrive at the same barrier or warp
// operation (told apart by source line), when some never arrive, or when the step limit is reached.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <ucontext.h>
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

namespace emu {

enum State { kReady, kWarp, kBlock, kDone };
struct Fiber {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack;
    unsigned thread = 0, block = 0;
    State state = kReady;
    int line = 0;
    uint64_t value = 0, lanes[32];  // what it brings to a warp operation, and what all lanes brought
};
inline std::vector<Fiber> fibers;
inline Fiber *current = nullptr;
inline ucontext_t main_ctx;
inline std::function<void()> body;
inline unsigned threads = 0, blocks = 0;
inline uint8_t *shared = nullptr;  // dynamic shared memory, one area per block
inline size_t shared_bytes = 0;

inline void wait(State s, int line, uint64_t value = 0) {
    current->state = s;
    current->line = line;
    current->value = value;
    swapcontext(&current->ctx, &main_ctx);
}
inline void entry() {
    body();
    current->state = kDone;
    swapcontext(&current->ctx, &main_ctx);
}
// The group [first, first + count) is released when all of it waits at one line.
inline const char *release(size_t first, size_t count, State s) {
    size_t waiting = 0, done = 0;
    for (size_t i = first; i < first + count; i++) {
        waiting += fibers[i].state == s;
        done += fibers[i].state == kDone;
    }
    if (!waiting) return nullptr;
    if (done) return "some threads have left, others wait for them";
    if (waiting < count) return nullptr;
    for (size_t i = first; i < first + count; i++)
        if (fibers[i].line != fibers[first].line) return "threads wait at different places for one another";
    if (s == kWarp)
        for (size_t i = first; i < first + count; i++)
            for (size_t j = 0; j < 32; j++) fibers[i].lanes[j] = fibers[first + j].value;
    for (size_t i = first; i < first + count; i++) fibers[i].state = kReady;
    return nullptr;
}
// Runs fn on nblocks blocks of nthreads threads, all resident; null, or what went wrong.
inline const char *run(unsigned nblocks, unsigned nthreads, size_t smem, uint64_t seed, std::function<void()> fn) {
    static std::vector<uint64_t> area;
    area.assign((nblocks * smem + 7) / 8 + 2, 0xABABABABABABABABull);
    shared = (uint8_t *)(((uintptr_t)area.data() + 15) & ~(uintptr_t)15);
    shared_bytes = smem;
    blocks = nblocks, threads = nthreads, body = std::move(fn);
    const size_t total = (size_t)nblocks * nthreads, stack = 256 << 10;
    std::vector<Fiber>(total).swap(fibers);
    for (size_t i = 0; i < total; i++) {
        Fiber &f = fibers[i];
        f.thread = i % nthreads, f.block = (unsigned)(i / nthreads);
        f.stack.reset(new char[stack]);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.get();
        f.ctx.uc_stack.ss_size = stack;
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, entry, 0);
    }
    std::mt19937_64 rng(seed);
    std::vector<size_t> ready;
    for (uint64_t steps = 0; steps < 200000000ull;) {
        ready.clear();
        for (size_t i = 0; i < total; i++)
            if (fibers[i].state == kReady) ready.push_back(i);
        if (ready.empty()) {
            bool done = true;
            for (auto &f : fibers) done = done && f.state == kDone;
            return done ? nullptr : "threads wait for one another for ever";
        }
        std::shuffle(ready.begin(), ready.end(), rng);
        // a part of the ready threads only, so that some fall behind
        const size_t take = 1 + rng() % ready.size();
        for (size_t r = 0; r < take; r++, steps++) {
            current = &fibers[ready[r]];
            swapcontext(&main_ctx, &current->ctx);
            if (current->state == kReady) return "a thread stopped without waiting";
            const size_t i = ready[r];
            if (const char *e = release(i / 32 * 32, 32, kWarp)) return e;
            if (const char *e = release(i / nthreads * nthreads, nthreads, kBlock)) return e;
        }
    }
    return "step limit";
}

template <class T> uint64_t to_word(T v) {
    uint64_t w = 0;
    memcpy(&w, &v, sizeof v);
    return w;
}
template <class T> T from_word(uint64_t w) {
    T v;
    memcpy(&v, &w, sizeof v);
    return v;
}
inline unsigned lane() { return current->thread & 31; }
template <class T> T shfl(int line, T v, unsigned src) {
    wait(kWarp, line, to_word(v));
    return from_word<T>(current->lanes[src & 31]);
}
template <class T> T shfl_up(int line, T v, unsigned d) {
    wait(kWarp, line, to_word(v));
    return lane() >= d ? from_word<T>(current->lanes[lane() - d]) : v;
}
template <class T> T shfl_down(int line, T v, unsigned d) {
    wait(kWarp, line, to_word(v));
    return lane() + d < 32 ? from_word<T>(current->lanes[lane() + d]) : v;
}
template <class T> T shfl_xor(int line, T v, unsigned m) {
    wait(kWarp, line, to_word(v));
    return from_word<T>(current->lanes[lane() ^ m]);
}
inline unsigned ballot(int line, bool p) {
    wait(kWarp, line, p);
    unsigned r = 0;
    for (int i = 0; i < 32; i++) r |= (unsigned)(current->lanes[i] & 1) << i;
    return r;
}
inline unsigned reduce_min(int line, unsigned v) {
    wait(kWarp, line, v);
    uint64_t r = ~0ull;
    for (uint64_t w : current->lanes) r = std::min(r, w);
    return (unsigned)r;
}
struct Index {
    unsigned y = 0, z = 0;
    int kind;
    struct X {
        int kind;
        operator unsigned() const {
            return kind == 0 ? current->thread : kind == 1 ? current->block : kind == 2 ? threads : blocks;
        }
    } x;
    explicit Index(int k) : kind(k), x{k} {}
};

} // namespace emu

#ifndef __noinline__
#define __noinline__
#endif
static emu::Index threadIdx(0), blockIdx(1), blockDim(2), gridDim(3);
#define __syncthreads() emu::wait(emu::kBlock, __LINE__)
#define __syncwarp() emu::wait(emu::kWarp, __LINE__)
#define __ballot_sync(m, p) emu::ballot(__LINE__, (p) != 0)
#define __any_sync(m, p) (emu::ballot(__LINE__, (p) != 0) != 0)
#define __all_sync(m, p) (emu::ballot(__LINE__, (p) != 0) == 0xffffffffu)
#define __shfl_sync(m, v, s) emu::shfl(__LINE__, v, s)
#define __shfl_up_sync(m, v, d) emu::shfl_up(__LINE__, v, d)
#define __shfl_down_sync(m, v, d) emu::shfl_down(__LINE__, v, d)
#define __shfl_xor_sync(m, v, d) emu::shfl_xor(__LINE__, v, d)
#define __reduce_min_sync(m, v) emu::reduce_min(__LINE__, v)
#define __threadfence() ((void)0)

using std::max;
using std::min;
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __popcll(unsigned long long v) { return __builtin_popcountll(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __clzll(long long v) { return v ? __builtin_clzll((unsigned long long)v) : 64; }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline uint64_t __umul64hi(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t n) {
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << (n & 31)) >> 32);
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t n) { return (uint32_t)((((uint64_t)hi << 32) | lo) >> (n & 31)); }
template <class T> T __ldg(const T *p) { return *p; }
template <class T> T __ldcg(const T *p) { return *p; }
template <class T, class V> T atomicAdd(T *p, V v) { T o = *p; *p = o + (T)v; return o; }
template <class T, class V> T atomicMin(T *p, V v) { T o = *p; *p = std::min(o, (T)v); return o; }
template <class T, class V> T atomicMax(T *p, V v) { T o = *p; *p = std::max(o, (T)v); return o; }
template <class T, class V> T atomicOr(T *p, V v) { T o = *p; *p = o | (T)v; return o; }
inline size_t __cvta_generic_to_shared(const void *p) { return (size_t)p; }
// Static shared memory: one area per kernel instance, so a run of such a kernel has one block.
#undef __shared__
#define __shared__ static
#undef __launch_bounds__
#define __launch_bounds__(...)
