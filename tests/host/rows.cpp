// The persistent kernels of one block on the CPU (see cuda_runtime.h here).
#include "persistent.inc"  // dfs_kernels.cu: the persistent loop
#include "wide.inc"        // wide_kernels.cu: the 128-bit kernel

namespace mf {
namespace {

struct Ring {
    static constexpr uint64_t kCells = 1024;
    alignas(256) QueueHeader hdr{};
    std::vector<uint64_t> seq = std::vector<uint64_t>(kCells);
    Queue q;
    template <class Slots>
    explicit Ring(Slots *slots) {
        for (uint64_t k = 0; k < kCells; ++k) seq[k] = k;
        q = Queue{&hdr, reinterpret_cast<TaskRecord *>(slots),
                  reinterpret_cast<unsigned long long *>(seq.data()), kCells};
    }
};

// What had been counted when the first warp left.
const uint64_t *g_counts;
uint64_t g_num, *g_at_leave;
void note_leave() {
    for (uint64_t k = 0; k < g_num; ++k) *g_at_leave += g_counts[k];
}
void watch(const QueueHeader &hdr, const uint64_t *counts, uint64_t num, uint64_t *at_leave) {
    g_counts = counts;
    g_num = num;
    g_at_leave = at_leave;
    *at_leave = 0;
    host::leaving = &hdr.warps_out;
    host::on_leave = note_leave;
}

using Ull = unsigned long long;
constexpr uint32_t kPeriod = 64, kWaitLimit = 1u << 30;
uint32_t g_spread;

template <int TMAX>
void run_sym(const uint8_t *edges, const SymSource &src, uint64_t num, uint64_t *counts,
             uint64_t *nodes, const Queue &Q, unsigned seed) {
    auto body = [&] {
        constexpr int TPB = 128;
        using C = Carve<TPB, 16, 0>;
        uint8_t *smem = host::shared;
        stage_sym_hop_rules<TPB>(smem, edges, src.start_i, src.last - src.start_i + 1);
        const size_t tables = sym_tables_bytes(src.last - src.start_i + 1);
        const List<TPB> L = C::list(smem, tables);
        LocalStack S;
        S.base = 0;
        persistent_loop<TPB, 16, true, TMAX>(
            smem, nullptr, src, LunnonSource{}, num, reinterpret_cast<Ull *>(counts),
            reinterpret_cast<Ull *>(nodes), Q, kPeriod, kWaitLimit,
            g_spread, L, S,
            tail_of_warp<true, TMAX>(smem + tables + C::kThreadBytes));
    };
    g_spread = 1 + seed % 4;
    host::launch(128, seed, [](void *f) { (*static_cast<decltype(body) *>(f))(); }, &body);
}

template <int TMAX>
void run_lunnon(const uint8_t *meta, uint32_t bytes, uint32_t inst_offset, const LunnonSource &src,
                uint64_t num, uint64_t *counts, uint64_t *nodes, const Queue &Q, unsigned seed) {
    auto body = [&] {
        constexpr int TPB = 128;
        using C = Carve<TPB, 17, 0>;
        uint8_t *smem = host::shared;
        if (threadIdx.x == 0) std::memcpy(smem, meta, bytes);
        __syncthreads();
        const List<TPB> L = C::list(smem, bytes);
        LocalStack S;
        S.base = 0;
        persistent_loop<TPB, 17, false, TMAX>(
            smem, reinterpret_cast<const LunnonInstanceDev *>(smem + inst_offset), SymSource{}, src,
            num, reinterpret_cast<Ull *>(counts), reinterpret_cast<Ull *>(nodes), Q, kPeriod,
            kWaitLimit, g_spread, L, S, tail_of_warp<false, TMAX>(smem + bytes + C::kThreadBytes));
    };
    g_spread = 1 + seed % 4;
    host::launch(128, seed, [](void *f) { (*static_cast<decltype(body) *>(f))(); }, &body);
}

template <bool kRow>
void run_wide(const uint8_t *edges, int start, const uint8_t *cycles, uint64_t num, uint64_t *counts,
              uint64_t *nodes, const Queue &Q, uint4 *slots, unsigned seed) {
    constexpr int TPB = kRow ? 128 : 64;
    auto body = [&] {
        sym_wide_kernel<TPB, 56, kRow>(edges, start, 80, cycles, kWideCells, num,
                                       reinterpret_cast<Ull *>(counts),
                                       reinterpret_cast<Ull *>(nodes), Q, slots, kPeriod, kWaitLimit,
                                       g_spread);
    };
    g_spread = 1 + seed % (TPB / 32);
    host::launch(TPB, seed, [](void *f) { (*static_cast<decltype(body) *>(f))(); }, &body);
}

}  // namespace
}  // namespace mf

using namespace mf;

extern "C" void host_edges(int32_t n, uint8_t *out) { sym_edges_stride(n, out, kWideCells); }

extern "C" int32_t host_sym(const uint8_t *edges, int32_t n, int32_t start, const uint8_t *cycles,
                            uint64_t num, int32_t rows, uint32_t seed, uint64_t *counts,
                            uint64_t *nodes, uint64_t *at_leave) {
    std::vector<TaskRecord> slots(Ring::kCells);
    Ring ring(slots.data());
    watch(ring.hdr, counts, num, at_leave);
    const SymSource src{cycles, start, n * n - 1, rows ? n : 0};
    switch (rows ? n : 0) {
        case 0: run_sym<0>(edges, src, num, counts, nodes, ring.q, seed); break;
        case 5: run_sym<5>(edges, src, num, counts, nodes, ring.q, seed); break;
        case 6: run_sym<6>(edges, src, num, counts, nodes, ring.q, seed); break;
        case 7: run_sym<7>(edges, src, num, counts, nodes, ring.q, seed); break;
        case 8: run_sym<8>(edges, src, num, counts, nodes, ring.q, seed); break;
        default: return -1;
    }
    return int32_t(ring.hdr.error);
}

extern "C" int32_t host_lunnon(const uint8_t *meta, uint32_t bytes, uint32_t inst_offset,
                               const uint8_t *states, const uint32_t *owner, uint32_t stride,
                               uint64_t num, uint64_t maps, int32_t rows, uint32_t seed,
                               uint64_t *counts, uint64_t *nodes, uint64_t *at_leave) {
    std::vector<TaskRecord> slots(Ring::kCells);
    Ring ring(slots.data());
    watch(ring.hdr, counts, maps, at_leave);
    const LunnonSource src{states, owner, stride};
    if (rows) run_lunnon<6>(meta, bytes, inst_offset, src, num, counts, nodes, ring.q, seed);
    else run_lunnon<0>(meta, bytes, inst_offset, src, num, counts, nodes, ring.q, seed);
    return int32_t(ring.hdr.error);
}

extern "C" int32_t host_wide(const uint8_t *edges, int32_t start, const uint8_t *cycles, uint64_t num,
                             int32_t rows, uint32_t seed, uint64_t *counts, uint64_t *nodes,
                             uint64_t *at_leave) {
    std::vector<uint4> slots(Ring::kCells * kWideRecordWords / 4);
    Ring ring(slots.data());
    watch(ring.hdr, counts, num, at_leave);
    if (rows) run_wide<true>(edges, start, cycles, num, counts, nodes, ring.q, slots.data(), seed);
    else run_wide<false>(edges, start, cycles, num, counts, nodes, ring.q, slots.data(), seed);
    return int32_t(ring.hdr.error);
}
