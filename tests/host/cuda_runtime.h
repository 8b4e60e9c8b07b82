// A thread block on the CPU, for the kernels' device code compiled as plain
// C++ (tests/test_rows_on_host.py).  Every lane is a fiber that runs alone until
// its next warp-wide operation; who runs next is drawn at random.  So lanes of
// a warp are as far apart as the language lets them be: code that counts on
// them staying together without saying so reads values that are not there yet.
#pragma once

#include <setjmp.h>
#include <ucontext.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#define __device__
#define __host__
#define __global__ static
#define __forceinline__ inline
#define __restrict__ __restrict
#define __launch_bounds__(...)
#define __align__(n) alignas(n)

using cudaError_t = int;
using cudaStream_t = void *;

struct uint4 {
    uint32_t x, y, z, w;
};
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }

namespace host {

struct Index {
    unsigned x, y, z;
};
inline Index thread_index{}, block_index{}, block_size{}, grid_size{1, 1, 1};

struct Barrier {  // of a warp's lanes, or the block's
    int waiting = 0;
    unsigned long turn = 0;
};

struct Fiber {
    ucontext_t start;
    jmp_buf at;
    bool begun = false, done = false;
    std::vector<char> stack;
    const Barrier *until = nullptr;  // runnable once this has turned past `turn`
    unsigned long turn = 0;
    unsigned long ops = 0;
    uint64_t value[2];  // what the lane brought to its latest two operations
};

inline std::vector<Fiber> fibers;
inline std::vector<Barrier> warps;
inline Barrier block;
inline int current;
inline jmp_buf scheduler;
inline ucontext_t scheduler_start;
inline void (*body)(void *);
inline void *body_arg;
alignas(256) inline uint8_t shared[232448];

// The first warp that leaves (adds to `leaving`) runs `on_leave`.
inline const void *leaving;
inline void (*on_leave)();

inline void pause() {
    Fiber &f = fibers[current];
    if (!_setjmp(f.at)) _longjmp(scheduler, 1);
}

inline void meet(Barrier &b, int of) {
    Fiber &f = fibers[current];
    f.turn = b.turn;
    if (++b.waiting == of) {
        b.waiting = 0;
        ++b.turn;
    }
    f.until = &b;
    pause();
}

inline void entry() {
    body(body_arg);
    fibers[current].done = true;
    _longjmp(scheduler, 1);
}

// Run `threads` lanes of one block.
inline void launch(int threads, unsigned seed, void (*fn)(void *), void *arg) {
    std::mt19937 rng(seed);
    fibers.assign(threads, {});
    warps.assign(threads / 32, {});
    block = {};
    block_size = {unsigned(threads), 1, 1};
    body = fn;
    body_arg = arg;
    std::memset(shared, 0xAB, sizeof shared);
    std::vector<int> ready;
    for (;;) {
        ready.clear();
        bool all = true;
        for (int t = 0; t < threads; ++t) {
            const Fiber &f = fibers[t];
            if (f.done) continue;
            all = false;
            if (!f.until || f.until->turn != f.turn) ready.push_back(t);
        }
        if (all) return;
        if (ready.empty()) {
            std::fprintf(stderr, "lanes of a warp wait for lanes that left or wait elsewhere\n");
            std::abort();
        }
        // A random warp's lanes, in random order: each until it waits.
        const int warp = ready[rng() % ready.size()] / 32;
        std::vector<int> lanes;
        for (int t : ready)
            if (t / 32 == warp) lanes.push_back(t);
        for (size_t k = lanes.size(); k > 1; --k) std::swap(lanes[k - 1], lanes[rng() % k]);
        for (int t : lanes) {
            Fiber &f = fibers[t];
            current = t;
            thread_index = {unsigned(t), 0, 0};
            f.until = nullptr;
            if (_setjmp(scheduler)) continue;
            if (f.begun) _longjmp(f.at, 1);
            f.begun = true;
            f.stack.resize(1 << 18);
            getcontext(&f.start);
            f.start.uc_stack.ss_sp = f.stack.data();
            f.start.uc_stack.ss_size = f.stack.size();
            f.start.uc_link = nullptr;
            makecontext(&f.start, entry, 0);
            swapcontext(&scheduler_start, &f.start);
        }
    }
}

// All lanes of the warp bring a value; the reader sees everyone's.
struct Exchange {
    const Fiber *first;
    int lane, slot;
    explicit Exchange(uint64_t v) {
        Fiber &f = fibers[current];
        first = &fibers[current / 32 * 32];
        lane = current % 32;
        slot = f.ops++ & 1;
        f.value[slot] = v;
        meet(warps[current / 32], 32);
    }
    uint64_t of(int l) const { return first[l & 31].value[slot]; }
};

template <class T>
uint64_t pack(T v) {
    static_assert(sizeof(T) <= 8);
    uint64_t r = 0;
    std::memcpy(&r, &v, sizeof v);
    return r;
}
template <class T>
T unpack(uint64_t r) {
    T v;
    std::memcpy(&v, &r, sizeof v);
    return v;
}

}  // namespace host

#define threadIdx (host::thread_index)
#define blockIdx (host::block_index)
#define blockDim (host::block_size)
#define gridDim (host::grid_size)

inline void __syncwarp(unsigned = ~0u) { host::Exchange e(0); }
inline void __syncthreads() { host::meet(host::block, int(host::fibers.size())); }
inline unsigned __ballot_sync(unsigned, bool p) {
    const host::Exchange e(p);
    unsigned m = 0;
    for (int l = 0; l < 32; ++l) m |= unsigned(e.of(l)) << l;
    return m;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline bool __all_sync(unsigned m, bool p) { return __ballot_sync(m, p) == ~0u; }
template <class T>
T __shfl_sync(unsigned, T v, int from) {
    return host::unpack<T>(host::Exchange(host::pack(v)).of(from));
}
template <class T>
T __shfl_down_sync(unsigned, T v, int by) {
    const host::Exchange e(host::pack(v));
    return host::unpack<T>(e.of(e.lane + by < 32 ? e.lane + by : e.lane));
}
inline unsigned __reduce_min_sync(unsigned, unsigned v) {
    const host::Exchange e(v);
    unsigned r = ~0u;
    for (int l = 0; l < 32; ++l) r = unsigned(e.of(l)) < r ? unsigned(e.of(l)) : r;
    return r;
}
inline unsigned __reduce_or_sync(unsigned, unsigned v) {
    const host::Exchange e(v);
    unsigned r = 0;
    for (int l = 0; l < 32; ++l) r |= unsigned(e.of(l));
    return r;
}

template <class T>
T atomicAdd(T *p, T v) {
    if (p == host::leaving && host::on_leave) {
        host::on_leave();
        host::on_leave = nullptr;
    }
    const T old = *p;
    *p = old + v;
    return old;
}
template <class T>
T atomicCAS(T *p, T expect, T v) {
    const T old = *p;
    if (old == expect) *p = v;
    return old;
}
template <class T>
T atomicExch(T *p, T v) {
    const T old = *p;
    *p = v;
    return old;
}
template <class T>
T __ldg(const T *p) { return *p; }
template <class T>
T __ldcg(const T *p) { return *p; }
template <class T>
void __stcg(T *p, T v) { *p = v; }
inline void __threadfence() {}
inline void __nanosleep(unsigned) {}

inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __popcll(unsigned long long x) { return __builtin_popcountll(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __ffsll(long long x) { return __builtin_ffsll(x); }
inline int __clz(int x) { return x ? __builtin_clz(unsigned(x)) : 32; }
