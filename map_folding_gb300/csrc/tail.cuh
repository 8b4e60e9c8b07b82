// tail.cuh -- the last row of the search, counted on 32-bit masks.
//
// On both paths the last cells to be placed form a row v_0 .. v_{T-1} of the
// board (the spiral's last side; the last row of a 2-D Lunnon map), and 96 %
// of a 7x7 search's nodes lie there.  Each row cell v_t is held by two arcs:
// one to w_t, its neighbour in the row before, on one page b for the whole
// row, and one to v_{t-1}, on two pages that alternate along the row.  So
// instead of inserting the row's cells into the list and walking both pages
// again at every node, a warp takes 32 "roots" (lists that end where the row
// begins), writes down once per root what the row can see of the list, and
// counts every completion on masks:
//
//   U        the gaps of the list that are in the page-b face of some pending
//            w_x: no row cell can ever go anywhere else.  At most 31 of them
//            (17 on average on 7x7 and 8x8); numbered in list order, so a set
//            of gaps is a 32-bit mask and "after" is "greater".
//   W[x]     the face of w_x on page b: where v_x may still go.
//   P[x]     the gaps before w_x in list order (ones below a bit).
//   planes   the faces of the gaps on the two row pages, as bit planes of face
//            numbers, five each (six for 9x9): the gaps in the face of gap r are those whose
//            plane bits equal r's.
//
// Placing v_t into gap r (bit b) draws the arc (w_t, v_t) on page b; every
// pending face is on one side of it, W[x] &= that side, where gap r itself,
// if W[x] has it, is cut in two and W[x] keeps the half on its side.  Which
// half is one bit h(x, t): every pending W[x] holds at most one piece of each
// gap, so base gaps stay exact positions.  The gaps that the next cell may
// take are r's row-page face & W[x], cut by the row arcs drawn earlier on the same
// page: v_t and v_{t+1} lie on the same side of each.  With A(s, x) = the
// gaps whose piece seen by x is after v_s = h ? -b_s : -2 b_s, an arc (v_s,
// v_{s+1}) encloses A(s, x) ^ A(s+1, x).
//
// The levels are counted from the end: e = T-1-t, so v at level K has K row
// cells after it.  A frame (candidates C of level K, W[K-1..0], the earlier
// picks, the h bits) is one partly counted node.  All lanes of a warp step
// through the levels together: at each level, idle lanes take a frame from
// the level's queue, every lane places its frame's next candidate, and what
// is left of the frame goes back to the queue.  A frame may run on any lane;
// leaves are added up per root slot.
#pragma once

#include "dfs_core.cuh"

namespace mf {
namespace {

// What a warp keeps in shared memory for its rows.  CELLS: the most cells a
// root's list can have.  A level with FILL or more frames is run before a
// shallower one, so no level ever holds more than FILL - 1 + 32.
// BITS: of a face number, enough for half as many faces as cells.
template <int TMAX, int CELLS, int FILL, int BITS>
struct TailLayout {
    static_assert(CELLS <= (BITS == 5 ? 63 : 80) && FILL <= 32 && TMAX >= 2 && TMAX <= 9, "tail layout");
    static constexpr int kCap = FILL + 32;
    // Words of a frame ahead of its W: C, R, H and, where these pass 32 bits,
    // their high bits.
    static constexpr int kHead = TMAX > 8 ? 4 : 3;
    __host__ __device__ static constexpr int quads(int k) { return (kHead + k + 3) / 4; }
    __host__ __device__ static constexpr int cap(int k) { return k == TMAX - 1 ? 32 : kCap; }
    __host__ __device__ static constexpr int frames(int k) {  // offset of level k's queue
        int at = kFrames;
        for (int j = 1; j < k; ++j) at += quads(j) * cap(j) * 16;
        return at;
    }
    static constexpr int kPlane = 0;                         // 2 pages x BITS planes
    static constexpr int kBefore = kPlane + 2 * BITS * 128;  // P of each level
    static constexpr int kTop = kBefore + TMAX * 128;        // Lunnon: bit 0 the gap on the sentinel,
                                                             // bit 1 leaves are nodes too,
                                                             // << 8 the first level with an arc
    static constexpr int kAcc = kTop + 128;                  // leaves of each root
    static constexpr int kRootNodes = kAcc + 128;            // nodes of each root (if asked for)
    static constexpr int kFrames = kRootNodes + 128;
    // Scratch of the set-up, in the frames' place (they are empty then): a word
    // per cell (the face numbers before it, later also the gaps of U before it)
    // and 16 words of face numbers per gap of U.
    static constexpr int kPre = kFrames;
    static constexpr int kGapIds = kPre + CELLS * 128;
    static constexpr int kScratchEnd = kGapIds + 16 * 128;
    static constexpr int kEnd = frames(TMAX);
    static constexpr int kBytes = ((kEnd > kScratchEnd ? kEnd : kScratchEnd) + 127) / 128 * 128;
};

// The row's pages: partner tables of the placed cells (an entry >= the
// number of placed cells: none).
struct TailPages {
    const uint8_t *b;   // page of the arcs (w_t, v_t)
    const uint8_t *a0;  // page of the arc from a cell of an even level
    const uint8_t *a1;  // ... of an odd level
};

// kSym: a square's side, always of TMAX cells; else rows of a Lunnon map, of up
// to TMAX leaves (a longer row starts inside), whose gap on the sentinel counts
// as a node and is not searched; or, where squares' sides shorter than TMAX are
// among them, both (the request server).
template <bool kLong>
struct HistWord {
    using type = uint32_t;
};
template <>
struct HistWord<true> {
    using type = uint64_t;
};

// Most ways to place t row cells into 31 gaps so that their arcs to the row before
// cross nowhere, whatever the list (a bound).  The first arc cuts the gaps, its own
// in two, and the other cells between its sides; as its end goes through the gaps
// in order, cells only ever pass from one side to the other.
constexpr uint64_t most_rows(int t) {
    uint64_t g[10][32] = {};
    for (int n = 0; n < 32; ++n) g[0][n] = 1;
    for (int k = 1; k <= t; ++k)
        for (int n = 1; n < 32; ++n) {
            uint64_t best[10] = {};
            for (int p = 1; p <= n; ++p) {
                uint64_t most = 0;
                for (int j = 0; j < k; ++j) {
                    if (best[j] > most) most = best[j];
                    best[j] = most + g[j][p] * g[k - 1 - j][n + 1 - p];
                }
            }
            for (int j = 0; j < k; ++j)
                if (best[j] > g[k][n]) g[k][n] = best[j];
        }
    return g[t][31];
}

// Whether 32 bits hold a count's sums whatever the roots: a root's leaves in kAcc,
// and all 32 roots' nodes in one lane (a square's last cells are no nodes).  They
// do for rows of up to seven (410,013,942 leaves, 1,308,637,184 nodes); 9x9 rows
// could have 3.7e10 leaves by this bound.
constexpr bool sums_fit(int t, bool square) {
    uint64_t nodes = 1;
    for (int k = 1; k <= t - square; ++k) nodes += most_rows(k);
    return most_rows(t) < (1ULL << 32) && 32 * nodes < (1ULL << 32);
}
static_assert(sums_fit(7, true) && sums_fit(6, false) && !sums_fit(8, true), "sums of a row count");

// Elsewhere the sums go to 64-bit ones once a lane (or root, see kRootNodes) has
// counted this many nodes.  A turn adds at most 31 nodes a level and 31 x 31 at the
// last, 32 lanes' to a root, and at most 31 leaves a node.  (2,000 8x8 cases 58.8 ms
// without, 58.5 with; with the 64-bit sums inside the loop 59.4, and 5,000 7x7 cases
// 2.5 % longer.)
constexpr uint32_t kTailNodes = 1 << 21;
static_assert(uint64_t(kTailNodes + 31 + 7 * 31 + 31 * 31) * 31 * 32 < (1ULL << 32), "sums of a row count");

// With kRootNodes the nodes too are added up per root, not per lane.
template <bool kSym, int TMAX, int CELLS, int FILL, int BITS = 5, bool kRootNodes = false>
struct Tail {
    using Y = TailLayout<TMAX, CELLS, FILL, BITS>;
    static constexpr int kRow = TMAX;
    static constexpr bool kLong = kRootNodes || !sums_fit(TMAX, kSym);
    // R: the gap numbers of the earlier picks, five bits each, the latest
    // lowest; H: the h bits, and the root's slot above them.
    using Hist = typename HistWord<(TMAX > 8)>::type;
    static constexpr int kSlotShift = TMAX > 8 ? 56 : 27;  // the top of the last frame word
    uint8_t *area;
    int lane;
    int cnt[TMAX];  // frames queued per level 1 .. TMAX-1 (warp-uniform)

    __device__ __forceinline__ uint32_t *word(int off) const {
        return reinterpret_cast<uint32_t *>(area + off);
    }
    // Bit of h(ex, es): the half of v_es's gap that the pending level ex keeps.
    __device__ static constexpr int hbit(int ex, int es) { return es * (es - 1) / 2 - 1 + ex; }

    // Clear the set-up's scratch (all lanes call).
    __device__ __forceinline__ void prepare_setup() const {
        uint4 *pre = reinterpret_cast<uint4 *>(area + Y::kPre);
#pragma unroll
        for (int k = 0; k < CELLS * 8; k += 32)
            if (k + lane < CELLS * 8) pre[k + lane] = make_uint4(~0u, ~0u, ~0u, ~0u);
        __syncwarp();
    }

    // Write down a root: the list L of `placed` cells, row levels K0 .. 0 to
    // come, w(e) the row-before neighbour of level e's cell and prev the cell
    // before the first (< 0: none, the row starts here).  Returns false if it
    // has more than 31 gaps.  Fills the root's tables and hands back the frame
    // in registers.
    //
    // One pass over the list in order, with no data-dependent branch so that
    // all lanes stay together: going past the first end of an arc enters a new
    // face, past the second end returns to the face before the first.  (Walking
    // each face by itself took 8 times as long, the lanes' walks being of
    // different lengths.)  A second pass numbers the gaps of U; their face
    // numbers are then turned into planes by a 16 x 16 bit transposition.
    template <class List, class WOf>
    __device__ __forceinline__ bool setup(const List &L, int placed, int K0, const TailPages &pg,
                                          WOf &&w, int prev, uint32_t &C, uint32_t (&W)[TMAX],
                                          Hist &R, Hist &H, bool lunnon = !kSym) const {
        constexpr uint32_t kField = (1u << BITS) - 1;
        constexpr uint32_t kIds = (1u << (3 * BITS)) - 1;
        uint32_t *pre = word(Y::kPre) + lane;
        // Face numbers of the gap at hand and the highest given out: page b in
        // the low field, then a0, a1.
        uint32_t f = 0, top = 0;
        int c = 0;
#pragma unroll 1
        for (int i = 0; i < placed; ++i) {
            pre[c * 32] = f | uint32_t(i) << 20;
            const int after = L.get(c);
            const int q0 = pg.b[c], q1 = pg.a0[c], q2 = pg.a1[c];
            // No placed partner: c's own entry, which changes nothing.
            const uint32_t v0 = pre[(q0 < placed ? q0 : c) * 32];
            const uint32_t v1 = pre[(q1 < placed ? q1 : c) * 32];
            const uint32_t v2 = pre[(q2 < placed ? q2 : c) * 32];
            if (v0 == ~0u) top += 1u;
            if (v1 == ~0u) top += 1u << BITS;
            if (v2 == ~0u) top += 1u << (2 * BITS);
            f = ((v0 == ~0u ? top : v0) & kField) | ((v1 == ~0u ? top : v1) & (kField << BITS)) |
                ((v2 == ~0u ? top : v2) & (kField << (2 * BITS)));
            c = after;
        }
        // Not one cycle (cell 0 met again before the end): left to the list walk.
        if (c != 0 || pre[0] >> 20 != 0) return false;
        // The faces of the w's on page b (a w has no arc there, so its gap is
        // in the face before it).
        uint32_t fw[TMAX];
        uint64_t set = 0;
#pragma unroll
        for (int e = 0; e < TMAX; ++e) {
            fw[e] = 0;
            if (e <= K0) {
                fw[e] = pre[w(e) * 32] & kField;
                set |= 1ULL << fw[e];
            }
        }
        const uint32_t fprev = prev >= 0 ? pre[prev * 32] : 0;
        // U in list order; each cell learns how many of its gaps come before.
        int gaps = 0;
        uint32_t first_in = 0, plane16 = 0, plane17 = 0;
        uint16_t *gap_ids = reinterpret_cast<uint16_t *>(area + Y::kGapIds) + 2 * lane;
#pragma unroll 1
        for (int i = 0; i < placed; ++i) {
            reinterpret_cast<uint8_t *>(pre + c * 32)[3] = uint8_t(gaps);
            c = L.get(c);
            const uint32_t v = pre[c * 32] & kIds;
            const bool in = BITS == 5 ? (uint32_t(set) >> (v & kField)) & 1 : (set >> (v & kField)) & 1;
            if (in && gaps < 32) {
                gap_ids[(gaps & 15) * 64 + (gaps >> 4)] = uint16_t(v);
                if (BITS == 6) {
                    plane16 |= ((v >> 16) & 1) << gaps;
                    plane17 |= ((v >> 17) & 1) << gaps;
                }
            }
            if (!kSym && i == 0) first_in = in;
            gaps += in;
        }
        if (gaps > 31) return false;
        uint32_t a[18];
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] = word(Y::kGapIds)[j * 32 + lane];
        a[16] = plane16;
        a[17] = plane17;
#pragma unroll
        for (int t = 8; t >= 1; t >>= 1) {
            const uint32_t m = t == 8 ? 0x00ff00ffu : t == 4 ? 0x0f0f0f0fu
                               : t == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (!(j & t)) {
                    const uint32_t x = ((a[j] >> t) ^ a[j + t]) & m;
                    a[j + t] ^= x;
                    a[j] ^= x << t;
                }
        }
#pragma unroll
        for (int j = 0; j < 2 * BITS; ++j) word(Y::kPlane)[j * 32 + lane] = a[BITS + j];
        const uint32_t all = (1u << gaps) - 1;
        C = 0;
#pragma unroll
        for (int e = TMAX - 1; e >= 0; --e) {
            uint32_t m = all;
#pragma unroll
            for (int j = 0; j < BITS; ++j) m &= (fw[e] >> j) & 1 ? a[j] : ~a[j];
            W[e] = e <= K0 ? m : 0;
            if (e == K0) C = m;
            word(Y::kBefore)[e * 32 + lane] = e <= K0 ? (1u << (pre[w(e) * 32] >> 24)) - 1 : 0;
        }
        if (!kSym)
            word(Y::kTop)[lane] = (lunnon ? first_in | 2u : 0u) | uint32_t(prev >= 0 ? TMAX : K0) << 8;
        R = 0;
        H = Hist(lane) << kSlotShift;
        if (prev >= 0) {
            // v_{t-1} is a cell of the list: its face on the page of the next
            // arc, and it stands in for all earlier picks (an arc between two
            // equal picks encloses nothing).
            const bool odd = (K0 + 1) & 1;
            const uint32_t fp = odd ? fprev >> (2 * BITS) : fprev >> BITS;
            uint32_t m = ~0u;
#pragma unroll
            for (int j = 0; j < BITS; ++j) {
                const uint32_t plane = word(Y::kPlane)[((odd ? BITS : 0) + j) * 32 + lane];
                m &= (fp >> j) & 1 ? plane : ~plane;
            }
            C &= m;
            const Hist before = pre[prev * 32] >> 24;
#pragma unroll
            for (int j = 0; j < (TMAX > 8 ? 7 : 6); ++j) R |= before << (5 * j);
            H |= (~Hist(0) << hbit(0, K0 + 1)) & ((Hist(1) << hbit(0, TMAX)) - 1);
        }
        return true;
    }

    // Put the root frames of the lanes in `have` into their levels' queues
    // (all lanes call; the set-up's scratch is given up here).
    __device__ __forceinline__ void enqueue_roots(bool have, int K0, uint32_t C, uint32_t (&W)[TMAX],
                                                  Hist R, Hist H) {
        word(Y::kAcc)[lane] = 0;
        if (kRootNodes) word(Y::kRootNodes)[lane] = 0;
        __syncwarp();
        push_roots<TMAX - 1>(have, K0, C, W, R, H);
        __syncwarp();
    }

    template <int K>
    __device__ __forceinline__ void push_roots(bool have, int K0, uint32_t C, uint32_t (&W)[TMAX],
                                               Hist R, Hist H) {
        if constexpr (K >= 1) {
            cnt[K] = 0;
            push<K>(have && K0 == K && C != 0, C, W, R, H);
            push_roots<K - 1>(have, K0, C, W, R, H);
        }
    }

    template <int K>
    __device__ __forceinline__ void push(bool mine, uint32_t C, const uint32_t (&W)[TMAX], Hist R,
                                         Hist H) {
        const unsigned m = __ballot_sync(kFull, mine);
        if (!m) return;
        const int at = cnt[K] + __popc(m & ((1u << lane) - 1));
        cnt[K] += __popc(m);
        if (mine) {
            uint32_t w[4 * Y::quads(K)] = {};
            w[0] = C;
            w[1] = uint32_t(R);
            w[2] = uint32_t(H);
            if constexpr (TMAX > 8)
                w[3] = uint32_t(R >> 32) | uint32_t(H >> 32) << 3;  // 3 bits, 3 bits and the slot
#pragma unroll
            for (int e = 0; e < K; ++e) w[Y::kHead + e] = W[e];
            uint4 *q = reinterpret_cast<uint4 *>(area + Y::frames(K)) + at;
#pragma unroll
            for (int j = 0; j < Y::quads(K); ++j)
                q[j * Y::cap(K)] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
        }
    }

    // Idle lanes (C == 0) take frames of level K.
    template <int K>
    __device__ __forceinline__ void refill(uint32_t &C, uint32_t (&W)[TMAX], uint32_t (&b)[TMAX],
                                           Hist &R, Hist &H) {
        const unsigned idle = __ballot_sync(kFull, C == 0);
        const int want = __popc(idle);
        const int take = want < cnt[K] ? want : cnt[K];
        const int rank = __popc(idle & ((1u << lane) - 1));
        cnt[K] -= take;
        if (C == 0 && rank < take) {
            const uint4 *q = reinterpret_cast<const uint4 *>(area + Y::frames(K)) + cnt[K] + rank;
            uint32_t w[4 * Y::quads(K)];
#pragma unroll
            for (int j = 0; j < Y::quads(K); ++j) {
                const uint4 x = q[j * Y::cap(K)];
                w[4 * j] = x.x;
                w[4 * j + 1] = x.y;
                w[4 * j + 2] = x.z;
                w[4 * j + 3] = x.w;
            }
            C = w[0];
            R = w[1];
            H = w[2];
            if constexpr (TMAX > 8) {
                R |= Hist(w[3] & 7) << 32;
                H |= Hist(w[3] >> 3) << 32;
            }
#pragma unroll
            for (int e = 0; e < K; ++e) W[e] = w[Y::kHead + e];
#pragma unroll
            for (int e = K + 1; e < TMAX; ++e)
                b[e] = 1u << (uint32_t(R >> (5 * (e - K - 1))) & 31);
        }
        __syncwarp();
    }

    // A(es, ex): the gaps whose piece seen by level ex is after v_es.
    __device__ static __forceinline__ uint32_t after(const uint32_t (&b)[TMAX], Hist H, int ex,
                                                     int es) {
        const uint32_t n = 0u - b[es];
        return (H >> hbit(ex, es)) & 1 ? n : n + n;
    }

    __device__ __forceinline__ void count_nodes(int slot, int n, uint32_t &nodes) const {
        if constexpr (kRootNodes) {
            if (n) atomicAdd(word(Y::kRootNodes) + slot, uint32_t(n));
        } else {
            nodes += n;
        }
    }

    // The row's last two cells: for every candidate of the last but one, how many
    // gaps are left for the last.  What depends on the frame alone (the arcs'
    // masks, the planes) is read once for all its candidates, which a lane takes
    // in turn (1.6 on average): there is nothing below to queue.  Queued like the
    // levels above, these steps were a third of all: 50,000 7x7 cases 809 ms, now
    // 738; 6x6 to depth 18 110 and 103 ms.
    __device__ __forceinline__ void last(uint32_t C, const uint32_t (&W)[TMAX],
                                         const uint32_t (&b)[TMAX], Hist H, uint32_t &nodes) const {
        if (!C) return;
        const int slot = int(H >> kSlotShift);
        const uint32_t info = kSym ? 0 : word(Y::kTop)[slot];
        const uint32_t *before = word(Y::kBefore) + slot;
        const uint32_t p0 = before[0], p1 = before[32];
        uint32_t plane[BITS];
#pragma unroll
        for (int j = 0; j < BITS; ++j) plane[j] = word(Y::kPlane)[(BITS + j) * 32 + slot];
        constexpr int kArcs = (TMAX - 2) / 2;  // row arcs on the page: levels 3-2, 5-4, ...
        uint32_t here[kArcs > 0 ? kArcs : 1], there[kArcs > 0 ? kArcs : 1];
#pragma unroll
        for (int j = 0; j < kArcs; ++j) {
            const int es = 2 * j + 3;
            here[j] = after(b, H, 1, es) ^ after(b, H, 1, es - 1);
            there[j] = after(b, H, 0, es) ^ after(b, H, 0, es - 1);
            // A Lunnon row may be shorter than TMAX: no arc leads to its first cell.
            if (!kSym && es > int(info >> 8)) here[j] = there[j] = 0;
        }
        const bool w_up = p0 > p1;
        uint32_t all = 0, leaves = 0;
        do {
            const uint32_t bt = C & (0u - C);
            C ^= bt;
            const uint32_t side = p1 ^ (bt - 1);
            uint32_t next = W[0] & (((p0 >= bt) != w_up ? side : ~side) | bt);
#pragma unroll
            for (int j = 0; j < BITS; ++j) next &= plane[j] & bt ? plane[j] : ~plane[j];
#pragma unroll
            for (int j = 0; j < kArcs; ++j) next &= here[j] & bt ? there[j] : ~there[j];
            all += __popc(next);
            leaves += __popc(next & ~(info & 1));
        } while (C);
        if (!kSym && (info & 2)) count_nodes(slot, int(all), nodes);
        if (leaves) atomicAdd(word(Y::kAcc) + slot, leaves);
    }

    // Level K of a descent: idle lanes take frames, every lane takes its
    // frame's next candidate and queues the rest (up to three times, so that
    // lanes still idle share the candidates of frames just taken: of 32 lanes
    // 21, 26 and 28 busy after one, two and three turns on 7x7 roots; 50,000 7x7
    // cases 890, 832 and 824 ms); then the candidates are placed, and the
    // placed cells' frames go on to the next level.
    template <int K>
    __device__ __forceinline__ void levels(int start, uint32_t &C, uint32_t (&W)[TMAX],
                                           uint32_t (&b)[TMAX], Hist &R, Hist &H,
                                           uint32_t &nodes) {
        if constexpr (K >= 1) {
            if constexpr (K == 1) {
                // Only roots that begin at the row's last but one cell queue here.
                if (cnt[1] > 0) refill<1>(C, W, b, R, H);
                last(C, W, b, H, nodes);
                C = 0;
                return;
            }
            if (K <= start) {
                uint32_t bt = 0;
#pragma unroll 1
                for (int turn = 0; turn < 3; ++turn) {
                    if (cnt[K] > 0) refill<K>(C, W, b, R, H);
                    const uint32_t rest = bt ? 0 : C & (C - 1);
                    if (!bt) bt = C & (0u - C);
                    push<K>(rest != 0, rest, W, R, H);
                    __syncwarp();
                    if (cnt[K] == 0 || __all_sync(kFull, bt != 0)) break;
                }
                uint32_t next = 0;
                if (bt) {
                    const int slot = int(H >> kSlotShift);
                    const uint32_t info = kSym ? 0 : word(Y::kTop)[slot];
                    const int r = 31 - __clz(int(bt));
                    const uint32_t *before = word(Y::kBefore) + slot;
                    const uint32_t *plane = word(Y::kPlane) + (K & 1) * 32 * BITS + slot;
                    uint32_t face = ~0u;
#pragma unroll
                    for (int j = 0; j < BITS; ++j) {
                        const uint32_t p = plane[j * 32];
                        face &= p & bt ? p : ~p;
                    }
                    const uint32_t pt = before[K * 32];
                    const uint32_t side = pt ^ (bt - 1);
                    const uint32_t inside = side | bt, outside = ~side | bt;
                    const bool up = bt > pt;
#pragma unroll
                    for (int e = K - 1; e >= 0; --e) {
                        const uint32_t pe = before[e * 32];
                        const bool in = (pe >= bt) != (pe > pt);
                        W[e] &= in ? inside : outside;
                        if (in != up) H |= Hist(1) << hbit(e, K);
                    }
                    next = face & W[K - 1];
#pragma unroll
                    for (int es = K + 2; es < TMAX; es += 2) {
                        const bool enclosed =
                            ((after(b, H, K, es) ^ after(b, H, K, es - 1)) & bt) != 0;
                        const uint32_t D = after(b, H, K - 1, es) ^ after(b, H, K - 1, es - 1);
                        const uint32_t side_of = enclosed ? D : ~D;
                        // A Lunnon row may be shorter than TMAX: no arc leads
                        // to its first cell.
                        next &= kSym || es <= int(info >> 8) ? side_of : ~0u;
                    }
                    count_nodes(slot, __popc(next), nodes);
                    next &= ~(info & 1);
                    b[K] = bt;
                    R = (R << 5) | Hist(r);
                    if constexpr (TMAX > 8) R &= (Hist(1) << 35) - 1;
                }
                C = next;
            }
            levels<K - 1>(start, C, W, b, R, H, nodes);
        }
    }

    // Take the 32-bit sums (this lane's nodes, its root's leaves and nodes) to
    // the caller's (all lanes call).  A lane adds to other lanes' sums until it is
    // through `last`, and reads other roots' tables there, so the lanes meet first.
    __device__ __forceinline__ void collect(uint32_t &counted, unsigned long long &leaves,
                                            unsigned long long &nodes) const {
        __syncwarp();
        leaves += word(Y::kAcc)[lane];
        nodes += counted;
        counted = 0;
        if (kRootNodes) nodes += word(Y::kRootNodes)[lane];
    }

    // Count the queued frames to the end: the leaves of the lane's root are added
    // to `leaves`, `counted` and the nodes to `nodes`.
    __device__ __forceinline__ void drain(uint32_t counted, unsigned long long &leaves,
                                          unsigned long long &nodes) {
        for (bool more = true; more;) {
            more = run(counted);
            collect(counted, leaves, nodes);
            if (more) {
                word(Y::kAcc)[lane] = 0;
                if (kRootNodes) word(Y::kRootNodes)[lane] = 0;
                __syncwarp();
            }
        }
    }

    // Count queued frames until none is left, or (true) the sums must be taken over.
    __device__ __forceinline__ bool run(uint32_t &nodes) {
        for (;;) {
            int start = 0;
#pragma unroll
            for (int k = 1; k < TMAX; ++k)
                if (cnt[k] > 0) start = k;  // the shallowest level with frames ...
#pragma unroll
            for (int k = TMAX - 1; k >= 1; --k)
                if (cnt[k] >= FILL) start = k;  // ... or the deepest full one
            if (start == 0) return false;
            uint32_t C = 0;
            Hist R = 0, H = 0;
            uint32_t W[TMAX] = {}, b[TMAX] = {};
            levels<TMAX - 1>(start, C, W, b, R, H, nodes);
            if (kLong && __any_sync(kFull, (kRootNodes ? word(Y::kRootNodes)[lane] : nodes) >= kTailNodes))
                return true;
        }
    }
};

// Row counting of the persistent kernels.  Frames that make a level full
// (squares, Lunnon rows), lanes at the row that start a count, and the
// bookkeeping rounds that a count stands for (50,000 7x7 cases: 1,216 ms with
// 16 / 24 / 16; fill 10: 1,312, fill 20: 904 against 832 at a later state, a CTA
// less fitting on an SM; roots 18: 1,294, roots 28: 1,189; rounds 32: 1,232,
// rounds 8: 1,206.  6x6 to depth 18: 116.6 ms with fill 16, 113.4 with 20).
constexpr int kTailFill = 16, kLunnonTailFill = 20;
constexpr int kTailRoots = 28;
constexpr uint32_t kTailRounds = 8;
// Levels above the row from which a subtree may be handed out: below, an item
// is a root or two and costs as much to pass on as to count (4x5 at depth 12,
// with sharing within the warp: 310 us at 4, 244 at 6).
constexpr int kRowSplit = 5;
constexpr int kRowShare = 1;  // the same for a piece shared within the warp
constexpr int kNoRow = 1 << 20;

// Whether the lanes of `at`, which have come to their rows, are to be counted now
// (all 32 lanes call): once kTailRoots of them have, or every busy lane that has a
// row.  Beside lanes of maps without one, which never come, fewer than kFewRoots go
// on by list (`walk`): a count stops the whole warp for some eight rounds, and a
// root by list takes its own lane some 80.  Three 1x20 strips (4.1 ms by themselves)
// and five 4x6 maps (1.1) in one launch: 17.6 ms waiting for all busy lanes, 7.0 so;
// a batch of 64 maps, half its work strips: 12.9 and 8.0 ms (8.4 with 4 or 16 roots
// and counting once seven of eight lanes with rows have come).
constexpr int kFewRoots = 8;
__device__ __forceinline__ bool count_rows_now(unsigned at, bool busy, bool here, int row_level,
                                               bool &walk) {
    walk = false;
    if (!at) return false;
    const int come = __popc(at);
    if (come < kTailRoots && __any_sync(kFull, busy && !here && row_level != kNoRow)) return false;
    walk = come < kFewRoots && __any_sync(kFull, busy && row_level == kNoRow);
    return !walk;
}

// The pages of the last row of a square: the row's last cell is `last`, held
// by last - 1 and by a cell of the row before.  `stride` cells per page.
__device__ __forceinline__ TailPages sym_row_pages(const uint8_t *edge, int last, int stride) {
    TailPages r{edge, edge, edge};
    for (int p = 0; p < 4; ++p) {
        const uint8_t *e = edge + p * stride;
        if (e[last] == last - 1) r.a1 = e;
        else if (e[last] < last) r.b = e;
        if (e[last - 1] == last - 2) r.a0 = e;
    }
    return r;
}

// Whether the arcs of the placed cells cross on no page: a page of k arcs has
// k + 1 faces then and only then.  The row count takes that for granted; a
// unit that a caller made up otherwise is searched by the list walk alone.
template <class List>
__device__ __forceinline__ bool pages_planar(const List &L, const uint8_t *edge, int stride,
                                             int placed) {
    bool planar = true;
#pragma unroll 1
    for (int p = 0; p < 4; ++p) {
        const uint8_t *e = edge + p * stride;
        uint64_t seen[2] = {0, 0};
        int faces = 0, ends = 0;
        for (int g0 = 0; g0 < placed; ++g0) {
            if (((g0 < 64 ? seen[0] : seen[1]) >> (g0 & 63)) & 1) continue;
            int g = g0;
            do {
                if (g < 64) seen[0] |= 1ULL << g;
                else seen[1] |= 1ULL << (g & 63);
                const int c = L.get(g);
                const int q = e[c];
                ends += q < placed;
                g = q < placed ? q : c;
            } while (g != g0);
            ++faces;
        }
        planar &= faces == ends / 2 + 1;
    }
    return planar;
}

}  // namespace
}  // namespace mf
