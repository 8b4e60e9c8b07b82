// wide_kernels.cu -- the sym_fold search on boards over 64 cells (9x9).
//
// experiments/9x9/sym_fold9.cpp runs sym_fold's recursion with 128-bit masks
// (sym_fold9.cpp:34, 261-312) so that cells past 63 can be counted.  This is
// the same search as the 64-bit batched kernel -- lockstep rounds, a persistent
// grid fed by a warp-cooperative split ring, lanes sharing within the warp, the
// last row counted on masks -- with 128-bit position masks, 96-cell successor lists and
// 128-byte split records.  Cases arrive as the 64-byte records of the 64-bit
// path (the host expands them to at most 64 cells); the list bytes past the
// record start as zeros and are written by insertions before they are read.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "dfs_core.cuh"
#include "engine.hpp"
#include "tail.cuh"

namespace mf {
namespace {

struct Mask128 {
    uint64_t lo, hi;
};

__device__ __forceinline__ bool w_zero(const Mask128 &m) { return (m.lo | m.hi) == 0; }
__device__ __forceinline__ int w_low(const Mask128 &m) {
    return m.lo ? __ffsll(static_cast<long long>(m.lo)) - 1
                : 63 + __ffsll(static_cast<long long>(m.hi));
}
__device__ __forceinline__ Mask128 w_drop_low(Mask128 m) {
    if (m.lo) m.lo &= m.lo - 1;
    else m.hi &= m.hi - 1;
    return m;
}
__device__ __forceinline__ int w_popc(const Mask128 &m) { return __popcll(m.lo) + __popcll(m.hi); }
__device__ __forceinline__ Mask128 w_low_bits(int k) {
    return Mask128{low_bits(k), k <= 64 ? 0ULL : low_bits(k - 64)};
}
__device__ __forceinline__ void w_set(Mask128 &m, int x) {
    const uint64_t b = 1ULL << (x & 63);
    m.lo |= x < 64 ? b : 0ULL;
    m.hi |= x < 64 ? 0ULL : b;
}

// Shared tables: 4 edge pages of kWideCells, then per cell the packed list of
// pages whose neighbour has a smaller number (9 bits each: page << 7 |
// neighbour) and its length.
constexpr size_t kWidePages = 4 * kWideCells;
constexpr size_t kWideTables = 1280;
static_assert(kWidePages + 8 * kWideCells + kWideCells <= kWideTables, "wide table layout");
constexpr int kWideWords = kWideCells / 4;  // list words per lane
constexpr int kWideRecordWords = 32;        // 128-byte split records
static_assert(kWideWords + 4 + 3 <= kWideRecordWords, "wide record layout");

template <int TPB>
__device__ __forceinline__ void stage_wide_tables(uint8_t *smem, const uint8_t *__restrict__ edges) {
    for (int k = threadIdx.x; k < int(kWidePages / 4); k += TPB)
        reinterpret_cast<uint32_t *>(smem)[k] = __ldg(reinterpret_cast<const uint32_t *>(edges) + k);
    for (int k = threadIdx.x; k < kWideCells; k += TPB) {
        uint64_t q = 0;
        int c = 0;
        for (int p = 0; p < 4; ++p) {
            const int nb = __ldg(edges + p * kWideCells + k);
            if (nb < k) q |= uint64_t(nb | (p << 7)) << (9 * c++);
        }
        reinterpret_cast<uint64_t *>(smem + kWidePages)[k] = q;
        smem[kWidePages + 8 * kWideCells + k] = uint8_t(c);
    }
}

// get_good with 128-bit masks (sym_fold9.cpp:286-312), in the two-chain form
// of SymRules::gaps: the (at most two) placed-neighbour pages of cell i are
// walked side by side, a chain that is back at its start retracing itself
// until the other is done.
struct SymRulesW {
    const uint8_t *edge;
    const uint64_t *pages;
    const uint8_t *count;
    template <int TPB>
    __device__ __forceinline__ Mask128 gaps(const List<TPB> &L, int i,
                                            unsigned long long &nodes) const {
        ++nodes;
        Mask128 good = w_low_bits(i);
        uint64_t q = pages[i];
        for (int left = count[i]; left > 0 && !w_zero(good); left -= 2, q >>= 18) {
            const uint64_t qb = left > 1 ? (q >> 9) : q;
            const int oA = int(q & 127), oB = int(qb & 127);
            const uint8_t *eA = edge + int((q >> 7) & 3) * kWideCells;
            const uint8_t *eB = edge + int((qb >> 7) & 3) * kWideCells;
            Mask128 aA{0, 0}, aB{0, 0};
            w_set(aA, oA);
            w_set(aB, oB);
            int jA = L.get(oA), jB = L.get(oB);
            bool dA = jA == oA, dB = jB == oB;
            while (!(dA && dB)) {
                const int pA = eA[jA];
                const int pB = eB[jB];
                const int xA = pA < i ? pA : jA;
                const int xB = pB < i ? pB : jB;
                w_set(aA, xA);
                w_set(aB, xB);
                jA = L.get(xA);
                jB = L.get(xB);
                dA |= jA == oA;
                dB |= jB == oB;
            }
            good.lo &= aA.lo & aB.lo;
            good.hi &= aA.hi & aB.hi;
        }
        return good;
    }
};

__device__ __forceinline__ SymRulesW wide_rules(const uint8_t *smem) {
    return SymRulesW{smem, reinterpret_cast<const uint64_t *>(smem + kWidePages),
                     smem + kWidePages + 8 * kWideCells};
}

// 128-bit mask stack.  The mask of level lvl holds positions below lvl, so
// its high word can be non-zero only for lvl > 64: low words get one row per
// level (level k at lo[k*TPB]), high words rows only for levels 65 ..
// 64 + kWideHiRows (after the low rows), and the other levels read zero.
// The chosen positions are interleaved bytes.
constexpr int kWideHiRows = 16;  // levels 65..80: enough below 82 cells

template <int TPB, int LEVELS>
struct StackW {
    uint64_t *lo;
    List<TPB> chosen;
    int base;
    __device__ __forceinline__ Mask128 get(int lvl) const {
        const uint64_t hi = lvl > 64 ? lo[(LEVELS + lvl - 65) * TPB] : 0ULL;
        return Mask128{lo[(lvl - base) * TPB], hi};
    }
    __device__ __forceinline__ void set(int lvl, const Mask128 &v) const {
        lo[(lvl - base) * TPB] = v.lo;
        if (lvl > 64) lo[(LEVELS + lvl - 65) * TPB] = v.hi;
    }
    __device__ __forceinline__ int pick(int lvl) const { return chosen.get(lvl - base); }
    __device__ __forceinline__ void set_pick(int lvl, int j) const { chosen.put(lvl - base, j); }
};

// The same in local memory, for the kernel that counts the last row by itself:
// it needs the shared memory for that, and its list search is a few nodes in a
// hundred.
template <int LEVELS>
struct LocalStackW {
    uint64_t lo[LEVELS], hi[kWideHiRows];
    uint8_t chosen[LEVELS];
    int base;
    __device__ __forceinline__ Mask128 get(int lvl) const {
        return Mask128{lo[lvl - base], lvl > 64 ? hi[lvl - 65] : 0ULL};
    }
    __device__ __forceinline__ void set(int lvl, const Mask128 &v) {
        lo[lvl - base] = v.lo;
        if (lvl > 64) hi[lvl - 65] = v.hi;
    }
    __device__ __forceinline__ int pick(int lvl) const { return chosen[lvl - base]; }
    __device__ __forceinline__ void set_pick(int lvl, int j) { chosen[lvl - base] = uint8_t(j); }
};

// Row counting on the 9x9 board.  A level is full at eight frames: three CTAs
// fit on an SM then, two with the 64-bit kernels' sixteen.  (Counting only the
// last eight cells, whose roots are a fifth the size: 582 ms for 2,000 cases at
// 48 cells, and 636 ms by list alone.)
constexpr int kWideRow = 9;
constexpr int kWideTailCells = 79;
using WideTail = Tail<true, kWideRow, kWideTailCells, 8, 6>;

template <int TPB, int LEVELS, bool kRow>
struct WideStack {
    using type = StackW<TPB, LEVELS>;
};
template <int TPB, int LEVELS>
struct WideStack<TPB, LEVELS, true> {
    using type = LocalStackW<LEVELS>;
};

template <int TPB, int LEVELS>
struct CarveW {
    static constexpr size_t kList = size_t(kWideWords) * 4 * TPB;
    static constexpr size_t kMask = size_t(LEVELS + kWideHiRows) * 8 * TPB;
    static constexpr size_t kPick = size_t((LEVELS + 3) / 4) * 4 * TPB;
    static constexpr size_t kBytes = kWideTables + kList + kMask + kPick;
    static constexpr size_t kRowBytes = kWideTables + kList + TPB / 32 * WideTail::Y::kBytes;
};

// advance of dfs_core.cuh with 128-bit masks (a taken split item starts here).
template <class List, class Stk>
__device__ __forceinline__ int advance_w(const List &L, Stk &S, int &lvl, int root) {
    for (;;) {
        const Mask128 cur = S.get(lvl);
        if (w_zero(cur)) {
            if (lvl == root) return -1;
            --lvl;
            L.put(S.pick(lvl), L.get(lvl));  // detach item lvl
            continue;
        }
        const int j = w_low(cur);
        S.set(lvl, w_drop_low(cur));
        L.put(lvl, L.get(j));  // insert item lvl after j
        L.put(j, lvl);
        S.set_pick(lvl, j);
        return lvl + 1;
    }
}

// apply_advance of dfs_core.cuh with 128-bit masks: consume level eval's
// mask g (handed over in registers) and move to the next node; -1 when the
// unit's subtree is exhausted.
template <class List, class Stk>
__device__ __forceinline__ int apply_advance_w(const List &L, Stk &S, int &lvl, int eval, int root,
                                               int last, bool fresh, const Mask128 &g,
                                               unsigned long long &leaves) {
    Mask128 cur;
    if (eval == last) {
        leaves += w_popc(g);
        if (fresh) return -1;
        L.put(S.pick(lvl), L.get(lvl));  // detach item lvl (= eval - 1)
        cur = S.get(lvl);
    } else {
        lvl = eval;
        cur = g;
    }
    for (;;) {
        if (w_zero(cur)) {
            if (lvl == root) return -1;
            --lvl;
            L.put(S.pick(lvl), L.get(lvl));  // detach item lvl
            cur = S.get(lvl);
            continue;
        }
        const int j = w_low(cur);
        S.set(lvl, w_drop_low(cur));
        L.put(lvl, L.get(j));  // insert item lvl after j
        L.put(j, lvl);
        S.set_pick(lvl, j);
        return lvl + 1;
    }
}

__device__ __forceinline__ void wide_take(const uint4 *slots, const Queue &Q, unsigned long long t,
                                          uint32_t (&w)[kWideRecordWords]) {
    const unsigned long long cell = t & (Q.capacity - 1);
    __threadfence();
    const uint4 *src = slots + cell * (kWideRecordWords / 4);
#pragma unroll
    for (int q = 0; q < kWideRecordWords / 4; ++q) {
        const uint4 x = __ldcg(src + q);
        w[4 * q] = x.x;
        w[4 * q + 1] = x.y;
        w[4 * q + 2] = x.z;
        w[4 * q + 3] = x.w;
    }
    __threadfence();
    atomicExch(Q.seq + cell, t + Q.capacity);
}

__device__ __forceinline__ void wide_put(uint4 *slots, const Queue &Q, unsigned long long t,
                                         const uint32_t (&w)[kWideRecordWords]) {
    const unsigned long long cell = t & (Q.capacity - 1);
    uint4 *dst = slots + cell * (kWideRecordWords / 4);
#pragma unroll
    for (int q = 0; q < kWideRecordWords / 4; ++q)
        __stcg(dst + q, make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]));
    __threadfence();
    atomicExch(Q.seq + cell, t + 1);
}

// The persistent loop of the 64-bit batched kernel (dfs_kernels.cu), for
// 128-bit masks: initial units by a warp-aggregated atomicAdd, lockstep
// rounds, bookkeeping every `period` rounds (idle-lane report, donation of
// the shallowest untried siblings while lanes wait), split items taken by
// idle lanes, and the same leaving rule; lanes of a warp share as there.  With
// kRow the 9x9 board's last row is counted on masks (tail.cuh).  Split record: list
// words 0..kWideWords-1, owner, untried mask (4 words), level, whether the row may
// be counted on masks.
template <int TPB, int LEVELS, bool kRow>
__global__ void __launch_bounds__(TPB)
    sym_wide_kernel(const uint8_t *__restrict__ edges, int start_i, int last,
                    const uint8_t *__restrict__ cycles, uint32_t record_bytes, unsigned long long num,
                    unsigned long long *counts, unsigned long long *nodes_out, Queue Q,
                    uint4 *slots, uint32_t period, uint32_t wait_limit, uint32_t spread) {
    extern __shared__ __align__(16) uint8_t smem[];
    stage_wide_tables<TPB>(smem, edges);
    __syncthreads();
    using C = CarveW<TPB, LEVELS>;
    const SymRulesW R = wide_rules(smem);
    const List<TPB> L = List<TPB>::at(smem + kWideTables, kWideCells);
    typename WideStack<TPB, LEVELS, kRow>::type S;
    if constexpr (!kRow) {
        S.lo = reinterpret_cast<uint64_t *>(smem + kWideTables + C::kList) + threadIdx.x;
        S.chosen = List<TPB>::at(smem + kWideTables + C::kList + C::kMask, (LEVELS + 3) / 4 * 4);
    }
    S.base = start_i;

    const int lane = threadIdx.x & 31;
    WideTail tail;
    tail.area = smem + kWideTables + C::kList + threadIdx.x / 32 * WideTail::Y::kBytes;
    tail.lane = lane;
    TailPages pages{};
    if constexpr (kRow) pages = sym_row_pages(smem, last, kWideCells);
    const int row_first = last + 1 - kWideRow;  // first level of the counted row
    int row_level = kNoRow;                     // ... of the unit at hand
    bool by_walk = false, share_miss = false;
    const unsigned lt_mask = (1u << lane) - 1u;
    constexpr int kOwner = kWideWords, kMaskW = kWideWords + 1, kRoot = kWideWords + 5,
                  kRowOk = kWideWords + 6;
    // Fewer units than lanes are spread over `spread` warps.
    const unsigned long long warps = (unsigned long long)gridDim.x * (TPB / 32);
    bool busy = false, fresh = false;
    bool init_left = (unsigned long long)lane * spread < num;
    int lvl = start_i, root = start_i, eval = start_i;
    uint32_t owner = 0;
    unsigned long long leaves = 0, nodes = 0, started = 0;
    long long finished = 0;  // items done less pieces taken, not reported yet
    uint32_t idle_rounds = 0, round = 0, nap = 256;
    int reported_idle = 0;
    bool ring_hint = false;

    auto flush = [&]() {
        if (leaves) atomicAdd(counts + owner, leaves);
        leaves = 0;
        ++finished;
    };

    auto take_splits = [&](unsigned need) -> bool {
        const int want = __popc(need);
        unsigned long long first = 0;
        const int got = ring_claim(Q, &Q.hdr->spawn_head, want, true, first);
        const int rank = __popc(need & lt_mask);
        if (((need >> lane) & 1u) && rank < got) {
            uint32_t w[kWideRecordWords];
            wide_take(slots, Q, first + rank, w);
            ++started;
#pragma unroll
            for (int k = 0; k < kWideWords; ++k) L.set_word(k, w[k]);
            owner = w[kOwner];
            root = int(w[kRoot]);
            lvl = root;
            S.set(root, Mask128{uint64_t(w[kMaskW]) | (uint64_t(w[kMaskW + 1]) << 32),
                                uint64_t(w[kMaskW + 2]) | (uint64_t(w[kMaskW + 3]) << 32)});
            eval = advance_w(L, S, lvl, root);  // an item's mask is never empty
            fresh = false;
            by_walk = false;
            if (kRow) row_level = w[kRowOk] ? row_first : kNoRow;
            busy = eval >= 0;
            if (!busy) ++finished;
        }
        return got < want;
    };

    // The shallowest level with untried siblings, and those.
    auto shallowest = [&](int &s) -> Mask128 {
        s = root;
        if (!busy || fresh) return Mask128{0, 0};
        while (s < lvl && w_zero(S.get(s))) ++s;
        return S.get(s);
    };

    auto donate = [&](int quota) {
        int s = root;
        const Mask128 m = shallowest(s);
        const bool can = !w_zero(m) && (row_level != kNoRow ? row_level - s >= kRowSplit
                                                            : last - s >= kMinRingHeight);
        const unsigned donors = shallowest_lanes(can, s, quota);
        if (!donors) return;
        unsigned long long first = 0;
        const int got = ring_claim(Q, &Q.hdr->spawn_tail, __popc(donors), false, first);
        const int rank = __popc(donors & lt_mask);
        if (!((donors >> lane) & 1u) || rank >= got) return;
        for (int l = lvl; l >= s; --l) L.put(S.pick(l), L.get(l));
        uint32_t w[kWideRecordWords];
#pragma unroll
        for (int k = 0; k < kWideRecordWords; ++k) w[k] = 0;
#pragma unroll
        for (int k = 0; k < kWideWords; ++k) w[k] = L.word(k);
        w[kOwner] = owner;
        w[kMaskW] = uint32_t(m.lo);
        w[kMaskW + 1] = uint32_t(m.lo >> 32);
        w[kMaskW + 2] = uint32_t(m.hi);
        w[kMaskW + 3] = uint32_t(m.hi >> 32);
        w[kRoot] = uint32_t(s);
        w[kRowOk] = row_level != kNoRow;
        for (int l = s; l <= lvl; ++l) {
            const int j = S.pick(l);
            L.put(l, L.get(j));
            L.put(j, l);
        }
        S.set(s, Mask128{0, 0});
        wide_put(slots, Q, first + rank, w);
    };

    // share_in_warp of dfs_core.cuh with 128-bit masks and separate picks.
    auto share = [&](unsigned idle) -> bool {
        int s = root;
        const Mask128 m = shallowest(s);
        const int floor = row_level != kNoRow ? row_level - kRowShare : last - kMinShareHeight;
        const unsigned donors = shallowest_lanes(!w_zero(m) && s <= floor, s, __popc(idle));
        const int n = __popc(donors);
        if (n == 0) return false;
        const bool give = (donors >> lane) & 1u;
        const int rank = __popc(idle & lt_mask);
        const bool take = ((idle >> lane) & 1u) && rank < n;
        const int from = take ? nth_bit(donors, rank) : lane;
        if (give)
            for (int l = lvl; l >= s; --l) L.put(S.pick(l), L.get(l));
        __syncwarp();
        const int level = __shfl_sync(kFull, s, from);
        const Mask128 mask{__shfl_sync(kFull, m.lo, from), __shfl_sync(kFull, m.hi, from)};
        const uint32_t whose = __shfl_sync(kFull, owner, from);
        const int its_row = __shfl_sync(kFull, row_level, from);
        if (take) {
            const List<TPB> theirs{L.base + 4 * (from - lane)};
            for (int j = 0; j < level; ++j) L.put(j, theirs.get(j));
            owner = whose;
            row_level = its_row;
            root = level;
            lvl = level;
            S.set(root, mask);
            eval = advance_w(L, S, lvl, root);
            --finished;  // see report_finished
            fresh = false;
            by_walk = false;
            busy = true;
        }
        __syncwarp();
        if (give) {
            for (int l = s; l <= lvl; ++l) {
                const int j = S.pick(l);
                L.put(l, L.get(j));
                L.put(j, l);
            }
            S.set(s, Mask128{0, 0});
        }
        return true;
    };

    for (;;) {
        // Initial units for lanes without work, one warp-aggregated claim.
        const unsigned want_init = __ballot_sync(kFull, !busy && init_left);
        if (want_init) {
            const int leader = __ffs(want_init) - 1;
            unsigned long long base = 0;
            if (lane == leader)
                base = atomicAdd(&Q.hdr->init_next, (unsigned long long)__popc(want_init));
            base = __shfl_sync(kFull, base, leader);
            if (!busy && init_left) {
                const unsigned long long k = base + __popc(want_init & lt_mask);
                if (k < num) {
                    // 64-byte records (cases of at most 64 cells) or 96-byte
                    // ones (deeper 9x9 expansions); list words past the
                    // record start as zeros.
                    const uint4 *src = reinterpret_cast<const uint4 *>(cycles + k * record_bytes);
                    const int vecs = int(record_bytes / 16);
#pragma unroll
                    for (int q = 0; q < kWideWords / 4; ++q) {
                        const uint4 x = q < vecs ? __ldg(src + q) : make_uint4(0, 0, 0, 0);
                        L.set_word(4 * q, x.x);
                        L.set_word(4 * q + 1, x.y);
                        L.set_word(4 * q + 2, x.z);
                        L.set_word(4 * q + 3, x.w);
                    }
                    owner = uint32_t(k);
                    root = start_i;
                    ++started;
                    by_walk = false;
                    const bool ok = list_valid(L, start_i);
                    if (kRow)
                        row_level = ok && pages_planar(L, smem, kWideCells, start_i) ? row_first
                                                                                     : kNoRow;
                    if (!ok) {
                        atomicExch(&Q.hdr->error, kErrMalformed);
                        ++finished;
                    } else if (start_i > last) {
                        leaves = 1;
                        flush();
                    } else {
                        busy = true;
                        fresh = true;
                        lvl = start_i;
                        eval = start_i;
                    }
                } else {
                    init_left = false;
                }
            }
        }
        const unsigned unfed = __ballot_sync(kFull, !busy && !init_left);
        if (__popc(unfed) >= kShareLanes && unfed != kFull && !share_miss) share_miss = !share(unfed);
        if (ring_hint) {
            const unsigned need = __ballot_sync(kFull, !busy && !init_left);
            if (need && (__popc(need) >= kTakeLanes || round + 1 >= period) && take_splits(need))
                ring_hint = false;
        }
        const bool bookkeeping = ++round >= period;
        if (!__any_sync(kFull, busy)) {
            report_finished(Q.hdr, finished);
            if (lane == 0) {
                if (reported_idle != kWarpTake) {
                    atomicAdd(reinterpret_cast<unsigned long long *>(&Q.hdr->idle_lanes),
                              (unsigned long long)(long long)(kWarpTake - reported_idle));
                    reported_idle = kWarpTake;
                }
            }
            const unsigned need = __ballot_sync(kFull, !init_left && lane < kWarpTake);
            const HeaderView now(Q.hdr);
            if (need && now.spawn_tail() != now.spawn_head()) take_splits(need);
            if (__any_sync(kFull, busy) || __any_sync(kFull, init_left)) {
                idle_rounds = 0;
                nap = 256;
                continue;
            }
            const bool stop = (now.init_next() >= num && now.completed() >= num + now.spawn_tail()) ||
                              now.error() != 0u || ++idle_rounds > wait_limit;
            if (stop) break;
            __nanosleep(nap);
            if (nap < 8192) nap <<= 1;
            continue;
        }
        idle_rounds = 0;
        nap = 256;
        auto at_row = [&]() { return kRow && busy && eval >= row_level && eval < last && !by_walk; };
        if (busy && !at_row()) {
            const Mask128 g = R.gaps(L, eval, nodes);
            by_walk = false;
            eval = apply_advance_w(L, S, lvl, eval, root, last, fresh, g, leaves);
            fresh = false;
            if (eval < 0) {
                flush();
                busy = false;
            }
        }
        if constexpr (kRow) {
            const bool here = at_row();
            const unsigned at = __ballot_sync(kFull, here);
            if (at && (__popc(at) >= kTailRoots || !__any_sync(kFull, busy && !here))) {
                uint32_t W[WideTail::kRow] = {};
                uint32_t c = 0, counted = 0;
                WideTail::Hist r = 0, h = 0;
                bool ok = false;
                tail.prepare_setup();
                if (here) {
                    auto w = [&](int e) -> int { return pages.b[last - e]; };
                    ok = tail.setup(L, eval, last - eval, pages, w, eval > row_first ? eval - 1 : -1, c, W,
                                    r, h);
                    if (ok) counted = __popc(c) + 1;
                    else by_walk = true;
                }
                tail.enqueue_roots(ok, last - eval, c, W, r, h);
                tail.drain(counted, leaves, nodes);
                if (ok) {
                    eval = apply_advance_w(L, S, lvl, eval, root, last, fresh, Mask128{0, 0}, leaves);
                    fresh = false;
                    if (eval < 0) {
                        flush();
                        busy = false;
                    }
                }
                __syncwarp();
                round += kTailRounds;
            }
        }
        if (!bookkeeping) continue;
        round = 0;
        const unsigned idle_mask = __ballot_sync(kFull, !busy);
        report_finished(Q.hdr, finished);
        if (lane == 0) {
            const int idle_now = __popc(idle_mask);
            if (idle_now != reported_idle) {
                atomicAdd(reinterpret_cast<unsigned long long *>(&Q.hdr->idle_lanes),
                          (unsigned long long)(long long)(idle_now - reported_idle));
                reported_idle = idle_now;
            }
        }
        const HeaderView now(Q.hdr);
        long long queued = 0;
        const int quota = split_quota(now, num, warps, queued);
        ring_hint = queued > 0;
        share_miss = false;
        if (quota > 0) donate(quota);
    }

    if (lane == 0 && reported_idle)
        atomicAdd(reinterpret_cast<unsigned long long *>(&Q.hdr->idle_lanes),
                  (unsigned long long)(-(long long)reported_idle));
    const unsigned long long ns = warp_sum(nodes);
    const unsigned long long st = warp_sum(started);
    if (lane == 0) {
        if (nodes_out && ns) atomicAdd(nodes_out, ns);
        if (st) atomicAdd(&Q.hdr->tasks_run, st);
        leave_and_check(Q.hdr, num);
    }
}

__global__ void wide_ring_init(unsigned long long *seq, unsigned long long capacity) {
    for (unsigned long long k = blockIdx.x * blockDim.x + threadIdx.x; k < capacity;
         k += gridDim.x * blockDim.x)
        seq[k] = k;
}

template <int kWideTPB, int LEVELS, bool kRow>
cudaError_t launch_wide_levels(const uint8_t *d_edges, int start_i, int last, const uint8_t *d_cycles,
                               uint32_t record_bytes, uint64_t num, uint64_t *d_counts, uint64_t *d_nodes, const Queue &Q,
                               uint4 *slots, const BatchKnobs &knobs, cudaStream_t stream) {
    static std::mutex mu;
    static bool raised[16] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    constexpr size_t smem =
        kRow ? CarveW<kWideTPB, LEVELS>::kRowBytes : CarveW<kWideTPB, LEVELS>::kBytes;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 16) return cudaErrorInvalidDevice;
        if (!raised[dev]) {
            e = cudaFuncSetAttribute(sym_wide_kernel<kWideTPB, LEVELS, kRow>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
            if (e != cudaSuccess) return e;
            raised[dev] = true;
        }
    }
    int fit = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, sym_wide_kernel<kWideTPB, LEVELS, kRow>,
                                                      kWideTPB, smem);
    if (e != cudaSuccess) return e;
    if (fit < 1) return cudaErrorInvalidConfiguration;
    if (knobs.blocks_per_sm > 0 && int(knobs.blocks_per_sm) < fit) fit = int(knobs.blocks_per_sm);
    const int sms = device_sm_count();
    uint32_t spread = uint32_t(sms * fit * (kWideTPB / 32));
    // Shallow units as in the 64-bit kernel; those of six levels or less are done
    // sooner than many warps have fetched theirs (3,000 of five / three levels with
    // the first warps full, over ten warps an SM and over one: 34 / 30, 36 / 34 and
    // 30 / 26 us; of six 36, 40 and over four 36; 30,000 of six 46, 42 and 51).
    const uint64_t levels = last + 1 - start_i, sm = uint64_t(sms);
    if (!kRow && levels <= kShallow) {
        const uint64_t few = levels <= 5 ? sm : levels == 6 ? std::max(4 * sm, num / 16) : kShallowWarps * sm;
        spread = uint32_t(std::min({uint64_t(spread), kShallowWarps * sm, few}));
    }
    sym_wide_kernel<kWideTPB, LEVELS, kRow><<<unsigned(sms * fit), kWideTPB, smem, stream>>>(
        d_edges, start_i, last, d_cycles, record_bytes, num,
        reinterpret_cast<unsigned long long *>(d_counts),
        reinterpret_cast<unsigned long long *>(d_nodes), Q, slots, knobs.node_budget,
        knobs.wait_limit, spread);
    return cudaGetLastError();
}

}  // namespace

uint64_t wide_workspace_bytes(uint64_t capacity) {
    return 256 + capacity * (4 * kWideRecordWords) + capacity * sizeof(unsigned long long);
}

cudaError_t launch_sym_wide(const uint8_t *d_wide_edges, int start_i, int stop_i,
                            const uint8_t *d_cycles, uint32_t record_bytes, uint64_t num,
                            uint64_t *d_counts,
                            uint64_t *d_nodes, void *d_workspace, const BatchKnobs &knobs,
                            cudaStream_t stream) {
    const uint64_t cap = knobs.queue_capacity;
    uint8_t *p = static_cast<uint8_t *>(d_workspace);
    Queue Q{};
    Q.hdr = reinterpret_cast<QueueHeader *>(p);
    Q.slots = nullptr;  // wide records live in `slots` below
    Q.seq = reinterpret_cast<unsigned long long *>(p + 256 + cap * (4 * kWideRecordWords));
    Q.capacity = cap;
    auto *slots = reinterpret_cast<uint4 *>(p + 256);
    cudaError_t e = cudaMemsetAsync(Q.hdr, 0, 256, stream);
    if (e != cudaSuccess) return e;
    wide_ring_init<<<64, 256, 0, stream>>>(Q.seq, cap);
    e = cudaGetLastError();
    if (e != cudaSuccess || num == 0) return e;
    e = cudaMemsetAsync(d_counts, 0, num * sizeof(uint64_t), stream);
    if (e != cudaSuccess) return e;
    const int levels = stop_i - 1 - start_i;
    // Stored levels run up to stop_i - 2; their high words need rows up to
    // stop_i - 2 - 65 < kWideHiRows.
    if ((record_bytes != kSymCells && record_bytes != kWideCells) || start_i > int(record_bytes) ||
        stop_i > 66 + kWideHiRows || stop_i > kWideCells)
        return cudaErrorInvalidValue;
    // The whole 9x9 row is nearly all of the search; near its end there is
    // nothing above it to search by list.
    if (stop_i == 81 && start_i <= stop_i - kWideRow && levels <= 56)
        return launch_wide_levels<128, 56, true>(d_wide_edges, start_i, stop_i - 1, d_cycles,
                                                 record_bytes, num, d_counts, d_nodes, Q, slots,
                                                 knobs, stream);
    if (levels <= 40)
        return launch_wide_levels<64, 40, false>(d_wide_edges, start_i, stop_i - 1, d_cycles, record_bytes, num,
                                      d_counts,
                                      d_nodes, Q, slots, knobs, stream);
    if (levels <= 56)
        return launch_wide_levels<64, 56, false>(d_wide_edges, start_i, stop_i - 1, d_cycles, record_bytes, num,
                                      d_counts,
                                      d_nodes, Q, slots, knobs, stream);
    return cudaErrorInvalidValue;  // deeper searches need a deeper expansion first
}

}  // namespace mf
