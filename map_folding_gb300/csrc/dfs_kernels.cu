// dfs_kernels.cu -- sm_103a counting kernels.
//
// Both hot paths of the reference are the same search shape: a circular
// successor list (Lunnon: b[] over leaves, mf.c:128-142; sym_fold: cycle[]
// over spiral cells, sym_fold.cpp:206-217), grown one item per level by
// inserting item `lvl` after a chosen position, with the set of admissible
// positions recomputed at every level by walking the list.  The engine below
// keeps that list per thread in shared memory (byte per item, in 128-byte
// rows shared by four warps so a warp never has a bank conflict), keeps the
// per-level choices as a 64-bit mask stack whose lowest bit is the current
// pick (in shared memory when the search is at most 48 levels deep, else in
// local memory) instead of the reference's gap[] array, walks a node's two
// constraint chains side by side, and counts the last level with a popcount.
// Gap rules:
//   LunnonRules  -- mf.c:88-124 as a bitwise AND of per-dimension walk masks
//   SymRules     -- sym_fold.cpp:179-204 (get_good)
// Kernels:
//   *_plain_kernel    one unit (prefix state / case) per lane, lanes of a warp
//                     sharing what is left, one launch
//   *_batched_kernel  persistent grid, device work queue, subtree splitting;
//                     the last row counted on masks (tail.cuh)
//
// Every unit's list is checked to be a permutation of its placed items before
// its search starts, which bounds every walk (see list_valid); the device
// queue is non-blocking (no thread ever waits on another), so malformed input
// cannot hang a kernel: a unit whose list is malformed reports UINT64_MAX
// (plain) or raises the queue error flag (batched).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "dfs_core.cuh"
#include "engine.hpp"
#include "tail.cuh"

namespace mf {
namespace {

// ------------------------------------------------------- plain kernels ---

// The plain kernels: each warp takes `per_warp` consecutive units, one a lane
// (32, or fewer where there are too few units to give every resident warp 32),
// and its lanes share what is left when theirs are done (run_units).  8,191
// states of the 5x5 map at depth 15, one lane each to the end, took 7.9 ms.

// d_counts[k] = completions of case k (UINT64_MAX if its cycle is malformed).
// Shared memory: sym tables and hop rows, the carve, the warps' counters.
template <int TPB, int LEVELS>
__global__ void __launch_bounds__(TPB)
    sym_plain_kernel(const uint8_t *__restrict__ edges, int start_i, int stop_i,
                     const uint8_t *__restrict__ cycles, uint64_t num, int per_warp,
                     unsigned long long *__restrict__ counts,
                     unsigned long long *__restrict__ nodes_out) {
    extern __shared__ __align__(16) uint8_t smem[];
    using C = Carve<TPB, 16, LEVELS>;
    const SymHopRules R = stage_sym_hop_rules<TPB>(smem, edges, start_i, stop_i - start_i);
    const size_t tables = sym_tables_bytes(stop_i - start_i);
    const List<TPB> L = C::list(smem, tables);
    typename StackOf<TPB, LEVELS>::type S;
    init_stack<TPB, 16, LEVELS>(S, smem, tables);
    const int lane = threadIdx.x & 31;
    const uint64_t unit = (uint64_t(blockIdx.x) * (TPB / 32) + threadIdx.x / 32) * per_warp + lane;
    const bool active = lane < per_warp && unit < num;
    if (active) load_list<TPB, 16>(L, cycles + unit * kSymCells, kSymCells);

    unsigned long long nodes = 0;
    const bool bad = active && !list_valid(L, start_i);
    S.base = start_i;
    auto *acc = reinterpret_cast<unsigned long long *>(smem + tables + C::kThreadBytes) +
                (threadIdx.x & ~31);
    const unsigned long long leaves =
        run_units(R, L, S, active && !bad, start_i, stop_i - 1, acc, nodes);
    if (active) counts[unit] = bad ? ~0ULL : leaves;
    if (nodes_out) {
        const unsigned long long s = warp_sum(nodes);
        if ((threadIdx.x & 31) == 0 && s) atomicAdd(nodes_out, s);
    }
}

// Shared memory: the map's neighbour table, the carve, the warps' counters.
template <int TPB, int LEVELS>
__global__ void __launch_bounds__(TPB)
    lunnon_plain_kernel(const uint8_t *__restrict__ table, int table_bytes, int n, int dim,
                        int start_leaf, const uint8_t *__restrict__ states, uint32_t stride,
                        uint64_t num, int per_warp, unsigned long long *__restrict__ per_state,
                        unsigned long long *__restrict__ total,
                        unsigned long long *__restrict__ nodes_out) {
    extern __shared__ __align__(16) uint8_t smem[];
    using C = Carve<TPB, 17, LEVELS>;
    for (int k = threadIdx.x; k < table_bytes / 4; k += TPB)
        reinterpret_cast<uint32_t *>(smem)[k] = __ldg(reinterpret_cast<const uint32_t *>(table) + k);
    const List<TPB> L = C::list(smem, table_bytes);
    typename StackOf<TPB, LEVELS>::type S;
    init_stack<TPB, 17, LEVELS>(S, smem, table_bytes);
    const int lane = threadIdx.x & 31;
    const uint64_t unit = (uint64_t(blockIdx.x) * (TPB / 32) + threadIdx.x / 32) * per_warp + lane;
    const bool active = lane < per_warp && unit < num;
    if (active) load_list<TPB, 17>(L, states + unit * stride, stride);
    __syncthreads();

    unsigned long long nodes = 0;
    const bool bad = active && !list_valid(L, start_leaf < n + 1 ? start_leaf : n + 1);
    S.base = start_leaf;
    auto *acc = reinterpret_cast<unsigned long long *>(smem + table_bytes + C::kThreadBytes) +
                (threadIdx.x & ~31);
    unsigned long long leaves = run_units(LunnonRules{smem, n, dim}, L, S, active && !bad,
                                          start_leaf, n, acc, nodes);
    leaves = bad ? 0 : leaves * static_cast<unsigned long long>(n);
    if (active && per_state) per_state[unit] = bad ? ~0ULL : leaves;
    if (total) {
        const unsigned long long s = warp_sum(leaves);
        if ((threadIdx.x & 31) == 0 && s) atomicAdd(total, s);
    }
    if (nodes_out) {
        const unsigned long long s = warp_sum(nodes);
        if ((threadIdx.x & 31) == 0 && s) atomicAdd(nodes_out, s);
    }
}

// ------------------------------------------------- persistent kernels ----

// Ready a launch: the ring's sequence numbers, the run header and `words`
// counters, in one launch instead of one and two memsets (2-3 us each, a third
// of a small map's time on the device).
__global__ void launch_init_kernel(Queue Q, unsigned long long *counts, unsigned long long words) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    const unsigned long long at = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (unsigned long long k = at; k < Q.capacity; k += step) Q.seq[k] = k;
    for (unsigned long long k = at; k < words; k += step) counts[k] = 0;
    if (at < 32) reinterpret_cast<unsigned long long *>(Q.hdr)[at] = 0;  // its 256 bytes
}

// Lunnon: levels to go, of a map with rows, from which they pay (4x4 at depth 11,
// four levels: 154 us by list, 81 by rows; below that a prefix is a node or two).
constexpr int kRowLevels = 4;

// Most cells of a list that the row count takes: all but two of a square's;
// for Lunnon maps kRowLeaves' worth (what the frames' place holds as scratch).
template <bool kSym, int TMAX>
__host__ __device__ constexpr int tail_cells() {
    return kSym && TMAX > 2 ? TMAX * TMAX - 2 : kRowLeaves - 1;
}

template <bool kSym>
__host__ __device__ constexpr int tail_fill() {
    return kSym ? kTailFill : kLunnonTailFill;
}

template <bool kSym, int TMAX>
__host__ __device__ constexpr size_t tail_bytes(int tpb) {
    if constexpr (TMAX > 0) return size_t(tpb / 32) * TailLayout<TMAX, tail_cells<kSym, TMAX>(), tail_fill<kSym>(), 5>::kBytes;
    else return 0;
}

template <bool kSym, int TMAX>
__device__ __forceinline__ uint8_t *tail_of_warp(uint8_t *areas) {
    return areas + tail_bytes<kSym, TMAX>(int(threadIdx.x) & ~31);
}

struct SymSource {
    const uint8_t *cycles;
    int start_i;
    int last;
    int row;  // cells of the board's last row (0: counted to a partial depth)
};

struct LunnonSource {
    const uint8_t *states;
    const uint32_t *state_owner;
    uint32_t stride;
};

// The persistent loop, in lockstep rounds.  Each round every busy lane
// evaluates one node, consumes it and advances to its next node; a lane whose
// unit is exhausted starts its next one at once: the next unit's index is
// taken with an atomicAdd when the previous unit starts, so only the record
// load is paid when the unit is needed (holding the record in registers
// ahead of time cost 16-20 registers per thread for the whole search, which
// the occupancy needs more).  Every `period` rounds
// a warp does its bookkeeping: it reports finished units and its idle-lane
// count, lets idle lanes take split items, and -- while fewer split items are
// queued than lanes wait for work -- lets a few busy lanes give away their
// shallowest untried siblings.  In between, lanes that run dry take pieces of
// their own warp's work (share_in_warp).  A warp leaves when it is idle and all work is
// accounted for, or when it has stayed idle for wait_limit rounds; leaving is
// always safe, because the warp that owns a split item's parent keeps looping
// until it has nothing left.  The last warp out checks that the work
// accounting closed (leave_and_check).
//
// With TMAX > 0 a lane that comes to the last row (of up to TMAX cells) stops
// there, and once enough lanes have (count_rows_now) the warp counts
// their rows together on masks (tail.cuh).
template <int TPB, int WORDS, bool kSym, int TMAX, class Stk>
__device__ __forceinline__ void persistent_loop(const uint8_t *s_tables,
                                                const LunnonInstanceDev *s_inst,
                                                const SymSource &sym, const LunnonSource &lun,
                                                unsigned long long num,
                                                unsigned long long *counts,
                                                unsigned long long *nodes_out, const Queue &Q,
                                                uint32_t period, uint32_t wait_limit, uint32_t spread,
                                                const List<TPB> &L, Stk &S, uint8_t *tail_area) {
    constexpr int kVecs = (WORDS + 3) / 4;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    bool busy = false, fresh = false;
    bool walking = false;  // a resumable walk is under way
    SymHopRules::Walk swalk{};
    LunnonRules::Walk lwalk{};
    int lvl = 0, root = 0, last = 0, eval = 0;
    uint32_t owner = 0;
    unsigned long long leaves = 0, nodes = 0, started = 0;
    long long finished = 0;  // items done less pieces taken, not reported yet
    uint32_t idle_rounds = 0, round = 0;
    int reported_idle = 0;  // lane 0: idle lanes this warp last reported
    bool ring_hint = false;  // warp-uniform: the split ring probably has items
    const SymHopRules srules{s_tables + 9 * kSymCells,
                             reinterpret_cast<const uint32_t *>(s_tables + 4 * kSymCells),
                             s_tables + 8 * kSymCells, sym.start_i};
    LunnonRules lrules{s_tables, 0, 0};
    using RowTail =
        Tail<kSym, (TMAX > 0 ? TMAX : 2), tail_cells<kSym, TMAX>(), tail_fill<kSym>()>;
    RowTail tail;
    tail.area = tail_area;
    tail.lane = lane;
    TailPages pages{};
    int row_level = kNoRow;  // first level of the last row
    bool by_walk = false;    // the node at hand has too many gaps for the row count
    if constexpr (TMAX > 0 && kSym) {
        if (sym.row > 0) {
            row_level = sym.last + 1 - sym.row;
            pages = sym_row_pages(s_tables, sym.last, kSymCells);
        }
    }

    // Prefetch state: 0 = no initial unit left for this lane, 1 = index
    // taken.  The first indices come from one warp-aggregated atomicAdd; fewer
    // units than lanes are spread over `spread` warps.
    const unsigned long long warps = (unsigned long long)gridDim.x * (TPB / 32);
    const unsigned long long even = (num + spread - 1) / spread;
    const int own = even < 32 ? int(even) : 32;
    unsigned long long pre_k = 0;
    {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&Q.hdr->init_next, (unsigned long long)own);
        pre_k = __shfl_sync(kFull, base, 0) + lane;
    }
    int pre_stage = lane < own ? 1 : 0;
    uint4 pre[kVecs];
    uint32_t pre_owner = 0;

#define MF_FETCH_RECORD()                                                                   \
    do {                                                                                   \
        const uint4 *src_ = kSym                                                           \
            ? reinterpret_cast<const uint4 *>(sym.cycles + pre_k * kSymCells)              \
            : reinterpret_cast<const uint4 *>(lun.states + pre_k * lun.stride);            \
        _Pragma("unroll") for (int q_ = 0; q_ < kVecs; ++q_) pre[q_] = __ldg(src_ + q_);   \
        if (!kSym) pre_owner = __ldg(lun.state_owner + pre_k);                             \
    } while (0)

    auto flush = [&]() {
        if (leaves) {
            const unsigned long long weight = kSym ? 1ULL : static_cast<unsigned long long>(lrules.n);
            atomicAdd(counts + owner, leaves * weight);
        }
        leaves = 0;
        ++finished;
    };

    int row_len = 0;  // Lunnon: leaves of a row of the map
    auto set_instance = [&](uint32_t inst) -> int {
        const LunnonInstanceDev I = s_inst[inst];
        lrules = LunnonRules{s_tables + I.table_offset, I.n, I.dim};
        last = I.n;
        S.base = I.start_leaf;
        if constexpr (TMAX > 0) {
            const int row = I.row < TMAX ? I.row : TMAX;
            row_level = row >= 2 ? I.n + 1 - row : kNoRow;
            // Partner tables: neighbour rows of the last two leaves, dimension
            // 0 along the row, dimension 1 across.
            const int w = I.n + 1;
            pages.a1 = lrules.table + I.n * w;
            pages.a0 = lrules.table + (I.n - 1) * w;
            pages.b = lrules.table + (w + I.n) * w;
            row_len = I.row;
        }
        return I.start_leaf;
    };

    // Warp-cooperative intake of split items by the lanes in `need` (all 32
    // lanes call): one claim on the ring's head, then each taking lane copies
    // its item.  Returns true if fewer items were available than asked for.
    auto take_splits = [&](unsigned need) -> bool {
        const int want = __popc(need);
        unsigned long long first = 0;
        const int got = ring_claim(Q, &Q.hdr->spawn_head, want, true, first);
        const bool mine = (need >> lane) & 1u;
        const int rank = __popc(need & lt_mask);
        if (mine && rank < got) {
            uint32_t w[24];
            ring_take(Q, first + rank, w);
            ++started;
#pragma unroll
            for (int k2 = 0; k2 < WORDS; ++k2) L.set_word(k2, w[k2]);
            owner = w[17];
            root = int(w[20]);
            if (kSym) {
                last = sym.last;
                S.base = sym.start_i;
                if constexpr (TMAX > 0) row_level = w[21] ? sym.last + 1 - sym.row : kNoRow;
            } else {
                set_instance(owner);
            }
            lvl = root;
            S.set(root, uint64_t(w[18]) | (uint64_t(w[19]) << 32));
            eval = advance(L, S, lvl, root);  // an item's mask is never empty
            walking = false;
            fresh = false;
            busy = eval >= 0;
        }
        return got < want;
    };

    // Warp-cooperative donation (all 32 lanes call): up to `quota` busy lanes
    // with an untried sibling set high enough above the counted level give the
    // shallowest such set away, those with the shallowest sets first.  One
    // claim on the ring's tail reserves cells for all donors; each donor rolls
    // its list back to that level, copies it out, replays, and publishes.
    auto donate = [&](int quota) {
        int s = root;
        const uint64_t m = busy && !fresh ? shallowest_siblings(S, root, lvl, s) : 0;
        const int low = TMAX > 0 && row_level != kNoRow ? row_level - s : last - s;
        const bool can = busy && !fresh && m != 0 &&
                         low >= (TMAX > 0 && row_level != kNoRow ? kRowSplit : kMinRingHeight);
        const unsigned donors = shallowest_lanes(can, s, quota);
        if (!donors) return;
        const bool give = (donors >> lane) & 1u;
        unsigned long long first = 0;
        const int got = ring_claim(Q, &Q.hdr->spawn_tail, __popc(donors), false, first);
        const int rank = __popc(donors & lt_mask);
        if (!give || rank >= got) return;
        roll_back(L, S, s, lvl);
        uint32_t w[24];
#pragma unroll
        for (int k = 0; k < 24; ++k) w[k] = 0;
#pragma unroll
        for (int k = 0; k < WORDS; ++k) w[k] = L.word(k);
        w[17] = owner;
        w[18] = uint32_t(m);
        w[19] = uint32_t(m >> 32);
        w[20] = uint32_t(s);
        if (TMAX > 0 && kSym) w[21] = row_level != kNoRow;
        replay_keeping_pick(L, S, s, lvl);
        ring_put(Q, first + rank, w);
    };

    // Pieces shared within the warp are no items of the ring: they are added up
    // within the warp, and its units count as finished when they are too.
    auto share = [&](unsigned idle) -> bool {
        uint32_t whose = 0;
        int its_row = 0;
        return share_in_warp(
            L, S, busy && !fresh, root, lvl,
            TMAX > 0 && row_level != kNoRow ? row_level - kRowShare : last - kMinShareHeight, idle,
            [&](int from, bool) {
                whose = __shfl_sync(kFull, owner, from);
                its_row = __shfl_sync(kFull, row_level, from);
            },
            [&](int level, uint64_t mask) {
                owner = whose;
                root = level;
                if (kSym) {
                    last = sym.last;
                    S.base = sym.start_i;
                    row_level = its_row;
                } else {
                    set_instance(owner);
                }
                S.set(root, mask);
                eval = advance(L, S, lvl, root);
                --finished;  // see report_finished
                walking = false;
                by_walk = false;
                fresh = false;
                busy = true;
            });
    };

    bool share_miss = false;  // warp-uniform: nothing to share at the last try
    uint32_t nap = 256;  // idle back-off, ns
    for (;;) {
        // Start the prefetched unit on lanes whose search has ended.
        if (!busy && pre_stage != 0) {
            if (pre_k < num) {
                MF_FETCH_RECORD();
#pragma unroll
                for (int q = 0; q < kVecs; ++q) {
                    const uint32_t ws[4] = {pre[q].x, pre[q].y, pre[q].z, pre[q].w};
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (4 * q + k < WORDS) L.set_word(4 * q + k, ws[k]);
                }
                ++started;
                bool ok;
                if (kSym) {
                    owner = uint32_t(pre_k);
                    root = sym.start_i;
                    last = sym.last;
                    S.base = root;
                    ok = list_valid(L, root);
                    if constexpr (TMAX > 0)
                        row_level = sym.row > 0 && ok && pages_planar(L, s_tables, kSymCells, root)
                                        ? sym.last + 1 - sym.row : kNoRow;
                } else {
                    owner = pre_owner;
                    root = set_instance(owner);
                    ok = list_valid(L, root < lrules.n + 1 ? root : lrules.n + 1);
                }
                if (!ok) {
                    atomicExch(&Q.hdr->error, kErrMalformed);
                    // As the plain kernel does: the case's count slot says it
                    // was not counted (a Lunnon slot is a whole map's sum and
                    // keeps only the error word).
                    if (kSym) counts[owner] = ~0ULL;
                    ++finished;
                } else if (root > last) {  // nothing left to place: one completion
                    leaves = 1;
                    flush();
                } else {
                    busy = true;
                    fresh = true;
                    walking = false;
                    lvl = root;
                    eval = root;
                }
                pre_k = atomicAdd(&Q.hdr->init_next, 1ULL);
                pre_stage = 1;
            } else {
                pre_stage = 0;
            }
        }
        // Idle lanes share the busy lanes' work.
        const unsigned unfed = __ballot_sync(kFull, !busy && pre_stage == 0);
        if (__popc(unfed) >= kShareLanes && unfed != kFull && !share_miss) share_miss = !share(unfed);
        // Lanes without initial units take split items while the warp's hint
        // says the ring has some (refreshed at bookkeeping, cleared by a miss).
        if (ring_hint) {
            const unsigned need = __ballot_sync(kFull, !busy && pre_stage == 0);
            if (need && (__popc(need) >= kTakeLanes || round + 1 >= period) && take_splits(need))
                ring_hint = false;
        }
        const bool bookkeeping = ++round >= period;
        if (!__any_sync(kFull, busy)) {
            // The whole warp is idle: report, look for split items, decide.
            report_finished(Q.hdr, finished);
            if (lane == 0) {
                if (reported_idle != kWarpTake) {
                    atomicAdd(reinterpret_cast<unsigned long long *>(&Q.hdr->idle_lanes),
                              (unsigned long long)(long long)(kWarpTake - reported_idle));
                    reported_idle = kWarpTake;
                }
            }
            const unsigned need = __ballot_sync(kFull, pre_stage == 0 && lane < kWarpTake);
            const HeaderView now(Q.hdr);
            if (need && now.spawn_tail() != now.spawn_head()) take_splits(need);
            // A lane still holding a prefetched unit keeps the warp alive.
            const bool holding = __any_sync(kFull, pre_stage != 0 && pre_k < num);
            if (__any_sync(kFull, busy) || holding) {
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
        // One round of evaluation per busy lane: a walk takes at most
        // kWalkCap steps and goes on in the next round if unfinished.
        auto at_row = [&]() {
            return TMAX > 0 && busy && eval >= row_level && eval < last && !by_walk;
        };
        if (busy && !at_row()) {
            uint64_t g = 0;
            bool evaluated;
            if (kSym) {
                if (!walking) {
                    srules.begin(L, eval, nodes, swalk);
                    walking = true;
                }
                evaluated = srules.run(L, swalk, kWalkCap);
                if (evaluated) g = srules.result(swalk, nodes);
            } else {
                if (!walking) {
                    lrules.begin(L, eval, nodes, lwalk);
                    walking = true;
                }
                evaluated = lrules.run(L, lwalk, kWalkCap);
                if (evaluated) g = lrules.result(lwalk, nodes);
            }
            if (evaluated) {
                walking = false;
                by_walk = false;
                eval = apply_advance(L, S, lvl, eval, root, last, fresh, g, leaves);
                fresh = false;
                if (eval < 0) {
                    flush();
                    busy = false;
                }
            }
        }
        if constexpr (TMAX > 0) {
            const bool here = at_row();
            const unsigned at = __ballot_sync(kFull, here);
            bool walk = false;
            if (count_rows_now(at, busy, here, row_level, walk)) {
                const int K0 = last - eval;
                uint32_t C = 0, counted = 0;
                typename RowTail::Hist R = 0, H = 0;
                uint32_t W[RowTail::kRow] = {};
                bool ok = false;
                tail.prepare_setup();
                if (here) {
                    auto w = [&](int e) -> int {
                        return kSym ? int(pages.b[last - e]) : last - e - row_len;
                    };
                    const int prev = eval > last + 1 - (kSym ? sym.row : row_len) ? eval - 1 : -1;
                    ok = tail.setup(L, eval, K0, pages, w, prev, C, W, R, H);
                    if (ok) {
                        counted = __popc(C) + (kSym ? 1 : 0);
                        if (!kSym) C &= ~(tail.word(RowTail::Y::kTop)[lane] & 1);
                    } else {
                        by_walk = true;
                    }
                }
                tail.enqueue_roots(ok, K0, C, W, R, H);
                tail.drain(counted, leaves, nodes);
                if (ok) {
                    eval = apply_advance(L, S, lvl, eval, root, last, fresh, 0, leaves);
                    fresh = false;
                    if (eval < 0) {
                        flush();
                        busy = false;
                    }
                }
                __syncwarp();
                round += kTailRounds;
            }
            by_walk |= walk && here;
        }
        if (!bookkeeping) continue;
        round = 0;
        const unsigned idle_mask = __ballot_sync(kFull, !busy);
        report_finished(Q.hdr, finished);
        long long queued = 0;
        if (lane == 0) {
            const int idle_now = __popc(idle_mask);
            if (idle_now != reported_idle) {
                atomicAdd(reinterpret_cast<unsigned long long *>(&Q.hdr->idle_lanes),
                          (unsigned long long)(long long)(idle_now - reported_idle));
                reported_idle = idle_now;
            }
        }
        const HeaderView now(Q.hdr);
        const int quota = split_quota(now, num, warps, queued);
        ring_hint = queued > 0;
        share_miss = false;
        // Feed waiting lanes: busy lanes give away their shallowest untried
        // siblings while lanes wait for work.
        if (quota > 0) donate(quota);
    }
#undef MF_FETCH_RECORD

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

template <int TPB, int LEVELS, int TMAX>
__global__ void __launch_bounds__(TPB, TMAX > 0 ? 4 : 768 / TPB)
    sym_batched_kernel(const uint8_t *__restrict__ edges, SymSource src, unsigned long long num,
                       unsigned long long *counts, unsigned long long *nodes_out, Queue Q,
                       uint32_t period, uint32_t wait_limit, uint32_t spread) {
    extern __shared__ __align__(16) uint8_t smem[];
    using C = Carve<TPB, 16, LEVELS>;
    stage_sym_hop_rules<TPB>(smem, edges, src.start_i, src.last - src.start_i + 1);
    const size_t tables = sym_tables_bytes(src.last - src.start_i + 1);
    const List<TPB> L = C::list(smem, tables);
    typename StackOf<TPB, LEVELS>::type S;
    init_stack<TPB, 16, LEVELS>(S, smem, tables);
    LunnonSource none{};
    persistent_loop<TPB, 16, true, TMAX>(smem, nullptr, src, none, num, counts, nodes_out, Q, period,
                                         wait_limit, spread, L, S,
                                         tail_of_warp<true, TMAX>(smem + tables + C::kThreadBytes));
}

// Shared memory: the maps' neighbour tables and their instance records
// (meta_bytes in all, records at inst_offset), then the carve.  One CTA of 512
// threads fits on an SM by shared memory, so it may take the registers of one
// (left to the compiler: 64, and 56 bytes spilled).
template <int TPB, int LEVELS, int TMAX>
__global__ void __launch_bounds__(TPB, TPB == 512 ? 1 : 0)
    lunnon_batched_kernel(const uint8_t *__restrict__ meta, uint32_t meta_bytes,
                          uint32_t inst_offset, LunnonSource src, unsigned long long num,
                          unsigned long long *counts, unsigned long long *nodes_out, Queue Q,
                          uint32_t period, uint32_t wait_limit, uint32_t spread) {
    extern __shared__ __align__(16) uint8_t smem[];
    using C = Carve<TPB, 17, LEVELS>;
    for (uint32_t k = threadIdx.x; k < meta_bytes / 4; k += TPB)
        reinterpret_cast<uint32_t *>(smem)[k] = __ldg(reinterpret_cast<const uint32_t *>(meta) + k);
    __syncthreads();
    const List<TPB> L = C::list(smem, meta_bytes);
    typename StackOf<TPB, LEVELS>::type S;
    init_stack<TPB, 17, LEVELS>(S, smem, meta_bytes);
    SymSource none{};
    persistent_loop<TPB, 17, false, TMAX>(
        smem, reinterpret_cast<const LunnonInstanceDev *>(smem + inst_offset), none, src, num, counts,
        nodes_out, Q, period, wait_limit, spread, L, S,
        tail_of_warp<false, TMAX>(smem + meta_bytes + C::kThreadBytes));
}

// ------------------------------------------------------- launch helpers --

// MF_STACK_MODE=local forces the local-memory stack (a tuning aid).
bool env_local_stack() {
    static const bool local = [] {
        const char *e = std::getenv("MF_STACK_MODE");
        return e && std::strcmp(e, "local") == 0;
    }();
    return local;
}

// Smallest compiled stack depth that holds `levels` levels (0 = local).
int pick_levels(int levels, bool local = false) {
    if (local || env_local_stack()) return 0;
    if (levels <= 24) return 24;
    if (levels <= 32) return 32;
    if (levels <= 48) return 48;
    return 0;
}

// Size a kernel's persistent grid from the occupancy calculator.  The first
// time a kernel is seen on a device its dynamic shared-memory limit is raised
// once to the device's opt-in maximum (never lowered again, so every later
// launch size stays legal); occupancy results are cached per (device,
// kernel, shared bytes), so a launch recorded into a CUDA graph makes no
// attribute or occupancy calls.
struct FitEntry {
    int dev;
    const void *fn;
    size_t smem;  // 0: the kernel's shared-memory limit has been raised
    int fit;
};
std::mutex g_fit_mu;
FitEntry g_fit[512];
int g_fit_len = 0;

template <class K>
cudaError_t prepare(K kernel, size_t smem, int tpb, int want_per_sm, int &blocks_per_sm) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const void *fn = reinterpret_cast<const void *>(kernel);
    int fit = 0;
    bool raised = false;
    {
        std::lock_guard<std::mutex> lock(g_fit_mu);
        for (int k = 0; k < g_fit_len; ++k) {
            if (g_fit[k].dev != dev || g_fit[k].fn != fn) continue;
            if (g_fit[k].smem == 0) raised = true;
            else if (g_fit[k].smem == smem) fit = g_fit[k].fit;
        }
    }
    if (!raised) {
        int optin = 0;
        e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(g_fit_mu);
        if (g_fit_len < 512) g_fit[g_fit_len++] = FitEntry{dev, fn, 0, 0};
    }
    if (fit == 0) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, tpb, smem);
        if (e != cudaSuccess) return e;
        if (fit < 1) return cudaErrorInvalidConfiguration;
        std::lock_guard<std::mutex> lock(g_fit_mu);
        if (g_fit_len < 512) g_fit[g_fit_len++] = FitEntry{dev, fn, smem, fit};
    }
    blocks_per_sm = want_per_sm > 0 && want_per_sm < fit ? want_per_sm : fit;
    return cudaSuccess;
}

}  // namespace

// ------------------------------------------------------------ launchers --

int device_sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
}

uint64_t workspace_bytes(uint64_t capacity) {
    return 256 + capacity * sizeof(TaskRecord) + capacity * sizeof(unsigned long long);
}

namespace {

Queue carve_queue(void *ws, uint64_t capacity) {
    uint8_t *p = static_cast<uint8_t *>(ws);
    Queue q;
    q.hdr = reinterpret_cast<QueueHeader *>(p);
    q.slots = reinterpret_cast<TaskRecord *>(p + 256);
    q.seq = reinterpret_cast<unsigned long long *>(p + 256 + capacity * sizeof(TaskRecord));
    q.capacity = capacity;
    return q;
}

// Host-side fault injection for tests (mf_test_inject_fault): the next
// persistent launch starts with one split-ring ticket reserved that no lane
// ever publishes, as if a donor's message had been lost.
std::atomic<uint32_t> g_inject{0};

__global__ void phantom_ticket_kernel(QueueHeader *hdr) { hdr->spawn_tail = 1; }

// Levels below the first of map units that are spread as shallow squares' are
// (37,378 states of 1x16 three levels from the end: 109 us over all warps, 87 over
// ten an SM; 40,000 of 1x18 four levels 229 and 203; of five over all 409, with the
// first warps full 470).
constexpr int kShallowMaps = 3;

// Launch size of a persistent launch over `units` initial units searched
// `levels` levels deep: the whole resident grid, or -- for a small job, whose
// units are shallow (at most 10 levels to go, so none of them is heavy) --
// about one warp per four units, with a split ring of at most two cells per
// launched lane (at least 1024).  A tiny map then costs one small launch and
// a short ring reset instead of thousands of warps that start, find nothing
// and leave, and a 512 KB ring initialisation.  Deep units always get the
// whole grid: a single deep unit can hold most of the work.
struct LaunchShape {
    unsigned blocks;
    uint64_t ring;
    uint32_t spread;  // warps that fewer units than lanes are spread over
};

LaunchShape persistent_shape(int sms, int bpsm, int tpb, uint64_t units, int levels,
                             uint64_t ring_knob, int shallow) {
    const uint64_t full = uint64_t(sms) * uint64_t(bpsm);
    if (levels > 10) return LaunchShape{unsigned(full), ring_knob, uint32_t(full * (tpb / 32))};
    const uint64_t warps = (units + 3) / 4;
    const uint64_t per_block = uint64_t(tpb / 32);
    uint64_t blocks = (warps + per_block - 1) / per_block;
    blocks = blocks < 1 ? 1 : (blocks > full ? full : blocks);
    uint64_t ring = 1024;
    while (ring < 2 * blocks * uint64_t(tpb) && ring < ring_knob) ring <<= 1;
    uint64_t spread = blocks * per_block;
    if (levels <= shallow && spread > uint64_t(sms) * kShallowWarps)
        spread = uint64_t(sms) * kShallowWarps;
    return LaunchShape{unsigned(blocks), ring < ring_knob ? ring : ring_knob, uint32_t(spread)};
}

cudaError_t reset_queue(const Queue &Q, uint64_t *counts, uint64_t words, cudaStream_t stream) {
    const uint64_t most = Q.capacity > words ? Q.capacity : words;
    const uint64_t blocks = (most + 255) / 256;
    launch_init_kernel<<<unsigned(blocks < 1024 ? blocks : 1024), 256, 0, stream>>>(
        Q, reinterpret_cast<unsigned long long *>(counts), words);
    if (g_inject.exchange(0) == MF_FAULT_LOST_SPLIT) phantom_ticket_kernel<<<1, 1, 0, stream>>>(Q.hdr);
    return cudaGetLastError();
}

}  // namespace

// Units per warp of a plain launch of units of `levels` levels on CTAs of `tpb`
// threads, `bpsm` of them resident on an SM: spread over all resident warps, shallow
// ones over ten an SM (see kShallow), and where lanes do not share 32 each.
static int plain_units_per_warp(uint64_t num, int bpsm, int tpb, int levels) {
    if (levels <= kNoShare) return 32;
    const uint64_t sms = uint64_t(device_sm_count());
    uint64_t warps = sms * uint64_t(bpsm) * uint64_t(tpb / 32);
    if (levels <= kShallow && warps > sms * kShallowWarps) warps = sms * kShallowWarps;
    const uint64_t k = (num + warps - 1) / (warps ? warps : 1);
    return k < 1 ? 1 : (k > 32 ? 32 : int(k));
}

cudaError_t launch_sym_plain(const uint8_t *d_edges, int start_i, int stop_i,
                             const uint8_t *d_cycles, uint64_t num, uint64_t *d_counts,
                             uint64_t *d_nodes, cudaStream_t stream) {
    if (num == 0) return cudaSuccess;
    constexpr int TPB = 128;
    const int levels = pick_levels(stop_i - 1 - start_i);
    const size_t tables = sym_tables_bytes(stop_i - start_i);
    auto *counts = reinterpret_cast<unsigned long long *>(d_counts);
    auto *nodes = reinterpret_cast<unsigned long long *>(d_nodes);
    int bpsm = 0;
#define MF_SYM_PLAIN(LV)                                                                        \
    do {                                                                                        \
        const size_t smem = tables + Carve<TPB, 16, LV>::kThreadBytes + 8 * TPB;                \
        cudaError_t e = prepare(sym_plain_kernel<TPB, LV>, smem, TPB, 0, bpsm);                 \
        if (e != cudaSuccess) return e;                                                         \
        const int per = plain_units_per_warp(num, bpsm, TPB, stop_i - start_i);                 \
        const uint64_t blocks = (num + per * (TPB / 32) - 1) / (per * (TPB / 32));              \
        sym_plain_kernel<TPB, LV><<<unsigned(blocks), TPB, smem, stream>>>(                     \
            d_edges, start_i, stop_i, d_cycles, num, per, counts, nodes);                       \
    } while (0)
    switch (levels) {
        case 24: MF_SYM_PLAIN(24); break;
        case 32: MF_SYM_PLAIN(32); break;
        case 48: MF_SYM_PLAIN(48); break;
        default: MF_SYM_PLAIN(0); break;
    }
#undef MF_SYM_PLAIN
    return cudaGetLastError();
}

cudaError_t launch_lunnon_plain(const uint8_t *d_table, int n, int dim, int start_leaf,
                                const uint8_t *d_states, uint32_t stride, uint64_t num,
                                uint64_t *d_per_state, uint64_t *d_total, uint64_t *d_nodes,
                                cudaStream_t stream) {
    if (num == 0) return cudaSuccess;
    constexpr int TPB = 128;
    const int table_bytes = (dim * (n + 1) * (n + 1) + 15) / 16 * 16;
    const int levels = pick_levels(n - start_leaf);
    auto *per = reinterpret_cast<unsigned long long *>(d_per_state);
    auto *tot = reinterpret_cast<unsigned long long *>(d_total);
    auto *nodes = reinterpret_cast<unsigned long long *>(d_nodes);
    int bpsm = 0;
#define MF_LUN_PLAIN(LV)                                                                        \
    do {                                                                                        \
        const size_t smem = table_bytes + Carve<TPB, 17, LV>::kThreadBytes + 8 * TPB;           \
        cudaError_t e = prepare(lunnon_plain_kernel<TPB, LV>, smem, TPB, 0, bpsm);              \
        if (e != cudaSuccess) return e;                                                         \
        const int k = plain_units_per_warp(num, bpsm, TPB, n + 1 - start_leaf);                 \
        const uint64_t blocks = (num + k * (TPB / 32) - 1) / (k * (TPB / 32));                  \
        lunnon_plain_kernel<TPB, LV><<<unsigned(blocks), TPB, smem, stream>>>(                  \
            d_table, table_bytes, n, dim, start_leaf, d_states, stride, num, k, per, tot,       \
            nodes);                                                                             \
    } while (0)
    switch (levels) {
        case 24: MF_LUN_PLAIN(24); break;
        case 32: MF_LUN_PLAIN(32); break;
        case 48: MF_LUN_PLAIN(48); break;
        default: MF_LUN_PLAIN(0); break;
    }
#undef MF_LUN_PLAIN
    return cudaGetLastError();
}

cudaError_t launch_sym_batched(const uint8_t *d_edges, int n, int start_i, int stop_i,
                               const uint8_t *d_cycles, uint64_t num, uint64_t *d_counts,
                               uint64_t *d_nodes, void *d_workspace, const BatchKnobs &knobs,
                               cudaStream_t stream, bool clear_nodes) {
    // The node counter is cleared with the counts where it follows them (the
    // host-buffer calls); elsewhere it is the caller's to clear.
    const bool own_nodes = clear_nodes && d_nodes == d_counts + num;
    if (num == 0)
        return reset_queue(carve_queue(d_workspace, knobs.queue_capacity), d_counts, own_nodes, stream);
    cudaError_t e = cudaSuccess;
    const int sms = device_sm_count();
    // The row count pays for units that end at the row or above it; a search to
    // a partial depth has no last row.  100,000 units by list / by rows: 7x7 from
    // 42 cells 0.86 / 0.28 ms, from 43 0.21 / 0.17; 8x8 from 56 0.46 / 0.27, from
    // 57 0.13 / 0.21; 6x6 from 30 0.52 / 0.17, from 31 0.09 / 0.13.
    const int row = stop_i == n * n && n >= 5 && start_i <= stop_i - n ? n : 0;
    const SymSource src{d_cycles, start_i, stop_i - 1, row};
    const int levels = pick_levels(stop_i - 1 - start_i, knobs.stack_mode == 1);
    const size_t tables = sym_tables_bytes(stop_i - start_i);
    auto *counts = reinterpret_cast<unsigned long long *>(d_counts);
    auto *nodes = reinterpret_cast<unsigned long long *>(d_nodes);
    int bpsm = 0;
#define MF_SYM_BATCHED(TPB, LV, TM)                                                              \
    do {                                                                                         \
        const size_t smem = tables + Carve<TPB, 16, LV>::kThreadBytes + tail_bytes<true, TM>(TPB);     \
        e = prepare(sym_batched_kernel<TPB, LV, TM>, smem, TPB, knobs.blocks_per_sm, bpsm);      \
        if (e != cudaSuccess) return e;                                                          \
        const LaunchShape shape =                                                                \
            persistent_shape(sms, bpsm, TPB, num, stop_i - start_i, knobs.queue_capacity,        \
                             TM == 0 ? kShallow : 0);                                            \
        const Queue Q = carve_queue(d_workspace, shape.ring);                                    \
        e = reset_queue(Q, d_counts, num + own_nodes, stream);                                   \
        if (e != cudaSuccess) return e;                                                          \
        sym_batched_kernel<TPB, LV, TM><<<shape.blocks, TPB, smem, stream>>>(                    \
            d_edges, src, num, counts, nodes, Q, knobs.node_budget, knobs.wait_limit,           \
            shape.spread);                                                                       \
    } while (0)
    if (row == 8) {
        MF_SYM_BATCHED(128, 0, 8);
    } else if (row == 7) {
        MF_SYM_BATCHED(128, 0, 7);
    } else if (row == 6) {
        MF_SYM_BATCHED(128, 0, 6);
    } else if (row == 5) {
        MF_SYM_BATCHED(128, 0, 5);
    } else if (knobs.block_threads == 256) {
        switch (levels) {
            case 24: MF_SYM_BATCHED(256, 24, 0); break;
            case 32: MF_SYM_BATCHED(256, 32, 0); break;
            case 48: MF_SYM_BATCHED(256, 48, 0); break;
            default: MF_SYM_BATCHED(256, 0, 0); break;
        }
    } else {
        switch (levels) {
            case 24: MF_SYM_BATCHED(128, 24, 0); break;
            case 32: MF_SYM_BATCHED(128, 32, 0); break;
            case 48: MF_SYM_BATCHED(128, 48, 0); break;
            default: MF_SYM_BATCHED(128, 0, 0); break;
        }
    }
#undef MF_SYM_BATCHED
    return cudaGetLastError();
}

cudaError_t launch_lunnon_batched(const uint8_t *d_meta, uint32_t meta_bytes, uint32_t inst_offset,
                                  int num_inst, int max_levels, int row_levels,
                                  const uint8_t *d_states, const uint32_t *d_state_owner,
                                  uint64_t num, uint64_t *d_counts, uint64_t *d_nodes,
                                  void *d_workspace, const BatchKnobs &knobs, cudaStream_t stream) {
    // The node counter follows the counts and is cleared with them.
    const uint64_t words = uint64_t(num_inst) + (d_nodes == d_counts + num_inst ? 1 : 0);
    if (num == 0)
        return reset_queue(carve_queue(d_workspace, knobs.queue_capacity), d_counts, words, stream);
    cudaError_t e = cudaSuccess;
    const int sms = device_sm_count();
    const uint32_t mb = (meta_bytes + 15) / 16 * 16;
    const LunnonSource src{d_states, d_state_owner, lunnon_state_stride(64)};
    const int levels = pick_levels(max_levels, knobs.stack_mode == 1);
    auto *counts = reinterpret_cast<unsigned long long *>(d_counts);
    auto *nodes = reinterpret_cast<unsigned long long *>(d_nodes);
    int bpsm = 0;
#define MF_LUN_BATCHED(TPB, LV, TM)                                                              \
    do {                                                                                         \
        const size_t smem = mb + Carve<TPB, 17, LV>::kThreadBytes + tail_bytes<false, TM>(TPB);         \
        e = prepare(lunnon_batched_kernel<TPB, LV, TM>, smem, TPB, knobs.blocks_per_sm, bpsm);   \
        if (e != cudaSuccess) return e;                                                          \
        const LaunchShape shape =                                                                \
            persistent_shape(sms, bpsm, TPB, num, max_levels, knobs.queue_capacity,              \
                             TM == 0 ? kShallowMaps : 0);                                        \
        const Queue Q = carve_queue(d_workspace, shape.ring);                                    \
        e = reset_queue(Q, d_counts, words, stream);                                             \
        if (e != cudaSuccess) return e;                                                          \
        lunnon_batched_kernel<TPB, LV, TM><<<shape.blocks, TPB, smem, stream>>>(                 \
            d_meta, mb, inst_offset, src, num, counts, nodes, Q, knobs.node_budget,             \
            knobs.wait_limit, shape.spread);                                                     \
    } while (0)
    // All the maps' tables are in every CTA's shared memory, so many small maps
    // leave room for few CTAs: take the CTA size that keeps more warps on an SM.
    // Where four warps' rows do not fit beside the tables (over 181 KB), the list
    // search still does.
    const size_t warp = tail_bytes<false, 6>(32) + Carve<32, 17, 0>::kThreadBytes;
    const size_t room = 227 * 1024;
    if (row_levels >= kRowLevels && mb + 4 * warp <= room) {
        const size_t small = room / (mb + 4 * warp + 1024) * 4;
        if (mb + 16 * warp <= room && small < 16) MF_LUN_BATCHED(512, 0, 6);
        else MF_LUN_BATCHED(128, 0, 6);
    } else if (knobs.block_threads == 256) {
        switch (levels) {
            case 24: MF_LUN_BATCHED(256, 24, 0); break;
            case 32: MF_LUN_BATCHED(256, 32, 0); break;
            case 48: MF_LUN_BATCHED(256, 48, 0); break;
            default: MF_LUN_BATCHED(256, 0, 0); break;
        }
    } else {
        switch (levels) {
            case 24: MF_LUN_BATCHED(128, 24, 0); break;
            case 32: MF_LUN_BATCHED(128, 32, 0); break;
            case 48: MF_LUN_BATCHED(128, 48, 0); break;
            default: MF_LUN_BATCHED(128, 0, 0); break;
        }
    }
#undef MF_LUN_BATCHED
    return cudaGetLastError();
}

}  // namespace mf

// ------------------------------------------- allocation-free entry point --
//
// mf_sym_count_cases_batched_static: the batched sym kernel with its split
// ring in a fixed device array instead of a caller-provided workspace.  For
// callers that cannot allocate device memory at all -- a process whose HBM is
// owned by another allocator, or a latency-critical caller that must not hit
// the implicit device synchronisation of cudaMalloc/cudaFree -- and therefore
// cannot hand over a workspace either.  Every GPU that loads this library
// holds these arrays until the process exits.

namespace mf {
namespace {

constexpr uint64_t kStaticRingCells = 4096;  // split-ring cells (power of two)
constexpr size_t kStaticWorkspaceBytes =
    256 + kStaticRingCells * (sizeof(TaskRecord) + sizeof(unsigned long long));  // 416.25 KiB

__device__ __align__(256) uint8_t g_static_workspace[kStaticWorkspaceBytes];
__device__ __align__(256) uint8_t g_static_edges[9][4 * kSymCells];  // edge pages per n

struct StaticState {
    bool ready = false;
    unsigned long long ctx_id = 0;  // the CUDA context the addresses belong to
    void *workspace = nullptr;
    uint8_t *edges = nullptr;
};

std::mutex g_static_mu;
StaticState g_static[64];

// Unique id of the calling thread's current CUDA context (0 if none can be
// read).  A device reset destroys the primary context and reloads this
// module with zeroed __device__ arrays; the next context gets a new id.
unsigned long long current_context_id() {
    using GetCurrent = int (*)(void **);
    using GetId = int (*)(void *, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
    });
    void *ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
    return id;
}

// Once per device and context, with that device current: look up the
// arrays' device addresses (a host-side name of a __device__ array is not a
// device address) and fill the edge pages of every board size.  Done again
// if the context changed since (a device reset), so no stale address or
// zeroed edge page is ever used.
int static_setup(int dev, StaticState *&out) {
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticState &s = g_static[dev];
    void *ws = nullptr;
    MF_TRY_CUDA(cudaGetSymbolAddress(&ws, g_static_workspace));  // also brings the context up
    const unsigned long long ctx = current_context_id();
    if (!s.ready || (ctx != 0 && ctx != s.ctx_id)) {
        void *edges = nullptr;
        MF_TRY_CUDA(cudaGetSymbolAddress(&edges, g_static_edges));
        uint8_t host[9][4 * kSymCells] = {};
        for (int n = 2; n <= 8; ++n) sym_edges(n, host[n]);
        MF_TRY_CUDA(cudaMemcpy(edges, host, sizeof(host), cudaMemcpyHostToDevice));
        s.workspace = ws;
        s.edges = static_cast<uint8_t *>(edges);
        s.ctx_id = ctx;
        s.ready = true;
    }
    out = &s;
    return MF_OK;
}

int current_static_state(StaticState *&s) {
    int dev = 0;
    MF_TRY_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_error("device ordinal %d out of range", dev);
        return MF_ERR_ARG;
    }
    return static_setup(dev, s);
}

}  // namespace
}  // namespace mf

extern "C" int32_t mf_sym_count_cases_batched_static(int32_t n, int32_t start_i, int32_t stop_i,
                                                     const uint8_t *d_cycles, uint64_t num_cases,
                                                     uint64_t *d_counts, uint64_t *d_nodes,
                                                     const mf_batch_config *cfg, void *stream) {
    using namespace mf;
    clear_error();
    if (n < 2 || n > 8) {
        set_error("n must be between 2 and 8");
        return MF_ERR_ARG;
    }
    if (start_i < 0 || start_i > stop_i || stop_i > n * n) {
        set_error("need 0 <= start_i <= stop_i <= n*n");
        return MF_ERR_RANGE;
    }
    if (cfg && cfg->queue_capacity > kStaticRingCells) {
        set_error("queue_capacity %llu exceeds the fixed split ring of %llu cells",
                  (unsigned long long)cfg->queue_capacity, (unsigned long long)kStaticRingCells);
        return MF_ERR_CAPACITY;
    }
    if (num_cases > 0xffffffffULL) {
        set_error("at most 2^32-1 cases per call");
        return MF_ERR_ARG;
    }
    if (num_cases && (!d_cycles || !d_counts)) {
        set_error("d_cycles and d_counts are required");
        return MF_ERR_ARG;
    }
    if (reinterpret_cast<uintptr_t>(d_cycles) % 16) {
        set_error("d_cycles must be 16-byte aligned");
        return MF_ERR_ARG;
    }
    if (cfg && cfg->stack_mode == 2) {
        set_error("stack_mode 2 (the 128-bit kernel) has no allocation-free form");
        return MF_ERR_ARG;
    }
    StaticState *s = nullptr;
    if (int rc = current_static_state(s)) return rc;
    BatchKnobs knobs = resolve_knobs(cfg);
    knobs.queue_capacity = kStaticRingCells;
    MF_TRY_CUDA(launch_sym_batched(s->edges + size_t(n) * 4 * kSymCells, n, start_i, stop_i, d_cycles,
                                   num_cases, d_counts, d_nodes, s->workspace, knobs,
                                   static_cast<cudaStream_t>(stream)));
    return MF_OK;
}

extern "C" int32_t mf_sym_static_status(void *stream, void *dst) {
    using namespace mf;
    clear_error();
    if (!dst) {
        set_error("dst is required");
        return MF_ERR_ARG;
    }
    StaticState *s = nullptr;
    if (int rc = current_static_state(s)) return rc;
    MF_TRY_CUDA(cudaMemcpyAsync(dst, s->workspace, sizeof(QueueHeader), cudaMemcpyDefault,
                                static_cast<cudaStream_t>(stream)));
    return MF_OK;
}

extern "C" void mf_test_inject_fault(uint32_t kind) { mf::g_inject.store(kind); }
