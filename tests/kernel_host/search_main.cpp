// One search of the kernel on the host: the instance and its team from standard
// input, the control block to standard output.
#include "lanes.h"
#include "search.cuh"

using namespace gastar;

template <class D, int TEAM> bool launch(const InstDesc& d, const LaunchParams& P, uint32_t warps, TeamCtl* ctl,
                                         void* stage, size_t dynamic, uint64_t seed) {
    return host::launch(P.team_ctas, warps * 32, TEAM == TEAM_CLUSTER ? P.team_ctas : 1, dynamic, seed, 500000, [&] {
        if (threadIdx.x == 0) {
            cta().desc = d;
            cta().slice = P.slice_iters;
        }
        __syncthreads();
        run_instance<D, 256, TEAM>(P, TeamRef{P.team_ctas, blockIdx.x, ctl, stage});
    });
}
template <class D> bool launch(int team, const InstDesc& d, const LaunchParams& P, uint32_t warps, TeamCtl* ctl,
                               void* stage, size_t dynamic, uint64_t seed) {
    if (team == TEAM_BLOCK) return launch<D, TEAM_BLOCK>(d, P, warps, ctl, stage, dynamic, seed);
    if (team == TEAM_CLUSTER) return launch<D, TEAM_CLUSTER>(d, P, warps, ctl, stage, dynamic, seed);
    return launch<D, TEAM_RING>(d, P, warps, ctl, stage, dynamic, seed);
}

int main() {
    InstDesc d;
    LaunchParams P;
    std::memset(&d, 0, sizeof(d));
    std::memset((void*)&P, 0, sizeof(P));
    unsigned long long key[4], seed, max_exp;
    uint32_t team, blocks, warps, buckets, slice, table_log2, cap;
    if (std::scanf("%u %u %u %llu %llu %llu %llu %u %u %u", &d.kind, &d.W, &d.H, key, key + 1, key + 2, key + 3, &d.minw,
                   &d.f0, &d.heuristic) != 10 ||
        std::scanf("%u %u %u %u %u %u %u %u %u %u %u %u %llu %u %llu", &team, &blocks, &warps, &d.ew, &d.ew_wide,
                   &d.wide_after, &buckets, &d.delta, &slice, &P.heap_snodes, &table_log2, &cap, &max_exp, &d.max_iter,
                   &seed) != 15)
        return 1;
    std::vector<uint8_t> weights((size_t)d.W * d.H);
    for (auto& w : weights) {
        unsigned v;
        if (std::scanf("%u", &v) != 1) return 1;
        w = (uint8_t)v;
    }
    d.start0 = key[0], d.start1 = key[1], d.goal0 = key[2], d.goal1 = key[3];
    const bool grid = d.kind == KIND_GRID, wide = d.kind == KIND_SLIDING5;
    const uint32_t entry = wide ? 32 : 16, maxn = grid ? 8 : 4, slot = grid ? 1 : wide ? 4 : 2;
    const uint64_t slots = grid ? weights.size() : 1ull << table_log2;
    std::vector<ulonglong2> table(slots * slot / 2 + 1);
    d.weights = weights.data();
    d.table = &table[0].x;
    d.table_words = slots * slot;
    d.table_mask = slots - 1;
    d.table_limit = grid ? ~0ull : slots * 3 / 4;
    d.max_probe = 4096;
    d.max_exp = max_exp;
    d.heaps = blocks * warps;
    d.heap_cap = cap;
    const uint32_t ew = d.ew_wide > d.ew ? d.ew_wide : d.ew;
    std::vector<uint4> nodes((size_t)d.heaps * (cap + 1) * 32 * entry / 16);
    std::vector<uint4> pages(bucket_area_bytes(d.heaps, buckets ? cap : 1, entry) / 16 + 1);
    std::vector<uint4> stage(team_stage_bytes(blocks, warps, ew, maxn, entry) / 16 + 1);
    std::vector<uint32_t> header(2 * d.heaps), touched(1 << 18);
    unsigned long long n_touched = ~0ull;
    d.heap_nodes = nodes.data();
    d.heap_hdr = header.data();
    if (buckets) {
        d.bq_base = pages.data();
        d.bq_pages = cap;
    }
    if (!grid) {
        d.touched = touched.data();
        d.touched_count = &n_touched;
        d.touched_cap = touched.size();
        d.prev_slot_words = slot;
        d.clear_either = 1;
    }
    static InstCtl ctl;
    static TeamCtl team_ctl;
    d.ctl = &ctl;
    P.insts = &d;
    P.n_insts = 1;
    P.team_ctas = blocks;
    P.buckets = buckets;
    P.slice_iters = slice;
    P.barrier_timeout_ns = ~0ull >> 1;
    // Dynamic shared memory as the engine gives it.
    const size_t per_warp = (size_t)(P.heap_snodes - 1) * 32 * entry + (buckets ? 256 : 0);
    const size_t dynamic =
        (team == TEAM_RING ? 0 : 2 * stage_entries_per_buffer(warps, ew, maxn) * entry) + warps * per_warp;
    uint32_t launches = 0;
    while (ctl.life != LIFE_DONE && launches < 5000) {
        team_ctl_init(team_ctl);
        ++launches;
        bool ok;
        switch (d.kind) {
            case KIND_SLIDING3: ok = launch<SlidingDom<3>>(team, d, P, warps, &team_ctl, stage.data(), dynamic, seed + launches); break;
            case KIND_SLIDING4: ok = launch<SlidingDom<4>>(team, d, P, warps, &team_ctl, stage.data(), dynamic, seed + launches); break;
            case KIND_SLIDING5: ok = launch<SlidingDom<5>>(team, d, P, warps, &team_ctl, stage.data(), dynamic, seed + launches); break;
            default: ok = launch<GridDom>(team, d, P, warps, &team_ctl, stage.data(), dynamic, seed + launches); break;
        }
        if (!ok) {
            std::printf("no end\n");
            return host::STUCK;
        }
    }
    std::printf("%u %u %u %llu %llu %llu %llu %llu %u\n", ctl.status, ctl.best, ctl.iterations, ctl.expansions, ctl.stale,
                ctl.generated, ctl.pushes, ctl.table_used, launches);
    return 0;
}
