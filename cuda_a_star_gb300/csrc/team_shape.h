// Shapes of the plain engine's teams and the shared memory of their blocks:
// host arithmetic that needs no GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include "../../include/gastar.h"
#include "engine_types.h"

namespace gastar {

inline uint32_t entry_bytes(uint32_t kind) { return kind == KIND_SLIDING5 ? 32u : 16u; }
inline uint32_t max_neighbours(uint32_t kind) { return kind == KIND_GRID ? 8u : 4u; }
inline uint32_t key_words(uint32_t kind) { return kind == KIND_SLIDING5 ? 2u : 1u; }

// Dynamic shared memory of a block: two stage buffers (one-block and cluster
// teams; `ring`: none, they are in global memory), then per warp its
// shared-memory heap nodes and bucket push scratch.
inline size_t block_smem_bytes(uint32_t kinds, uint32_t warps, uint32_t ew, bool ring,
                               uint32_t heap_snodes = kHeapSmemNodes, bool buckets = false) {
    size_t best = 0;
    for (uint32_t k = 0; k < 4; ++k)
        if (kinds & kind_bit(k)) {
            const size_t stage = ring ? 0 : 2 * stage_entries_per_buffer(warps, ew, max_neighbours(k)) * entry_bytes(k);
            const size_t per_warp = (size_t)(heap_snodes - 1) * 32 * entry_bytes(k) + (buckets ? 256 : 0);
            best = std::max(best, stage + ((size_t)warps * per_warp + 15) / 16 * 16);
        }
    return best;
}

// Team of one plain solve.
struct PlainShape {
    uint32_t ew = 0, W = 0;  // pops per warp-heap, warps per block
    uint32_t ew_wide = 0;    // pops per warp-heap once the search is widened (ew: never)
    uint64_t blocks = 0;     // 0: no such shape
    bool cluster = false;    // several blocks, one thread-block cluster
    bool ring() const { return blocks > 1 && !cluster; }
};

// Pops per warp-heap of a widened search.  A puzzle search with the automatic
// width that passes kWideAfter iterations is a hard one, whose iteration count
// the pops per iteration set rather than its depth; from then on every
// warp-heap pops four times as many (at most 32).  On the 64 15-puzzles of the
// plain benchmark (Q = 16384, 8-wide pops) the hardest took 333 iterations with
// twice the pops and takes 206 with four times; the 64 together 4 % less time.
// 12 15-puzzles on clusters (Q = 512, 256, 128) 24.0, 44.6 and 86.3 ms without
// it, 14.8, 23.3 and 42.3 with it; the hardest 9.4 and 4.6 at Q = 512.
inline uint32_t widened(const PlainShape& s, uint32_t kind, const gastar_config& cfg) {
    return s.blocks > 1 && kind != KIND_GRID && !cfg.expansion_width ? std::min(32u, 4 * s.ew) : s.ew;
}

// Shape of a ring team with the automatic widths: eight warps on every SM,
// popping few entries each.  An iteration lasts as long as its slowest warp,
// and a warp expands its pops in rounds (four grid cells, eight boards), so
// many warps with one or two rounds beat fewer with more.  Measured on 152
// blocks with 16-, 8- and 4-wide pops: 16 15-puzzles 10.6, 8.5 and 9.8 ms
// (4-wide: too few pops).  Grids pop 4 until their frontier (4096^2: ~4000
// cells) fills such pops, which with a pop window of 72 it does first; calls
// with 8- against 4-wide pops, no window and window 72: 2048^2 15.9 and 14.0,
// 14.6 and 13.4 ms; 2896^2 22.5 and 20.8, 20.6 and 20.2; 3200^2 25.4 and 23.8,
// 22.9 and 23.3; 3500^2 28.3 and 27.2, 25.2 and 26.7; 4096^2, searches alone,
// 34.3 and 34.8, 31.0 and 34.0.  Hence the line at 2^23 cells (2896^2).
// Q above 16384 asks for throughput on hard puzzles: pops as wide as it says.
inline PlainShape ring_shape(uint32_t sms, uint32_t kind, uint64_t cells, const gastar_config& cfg, uint64_t Q) {
    PlainShape s;
    const uint64_t warps = 8ull * sms;
    s.W = cfg.warps_per_block ? std::min(16u, cfg.warps_per_block) : 8u;
    if (cfg.expansion_width) s.ew = std::min(32u, cfg.expansion_width);
    else if (kind == KIND_GRID) s.ew = cells >= (1ull << 23) ? 8 : 4;
    else s.ew = (uint32_t)std::min<uint64_t>(Q <= 16384 ? 8 : 32, std::max<uint64_t>(4, (Q + warps - 1) / warps));
    const bool fixed = cfg.expansion_width || cfg.warps_per_block;
    const uint64_t heaps = std::min<uint64_t>((Q + s.ew - 1) / s.ew, fixed ? ~0ull : warps);
    s.blocks = (heaps + s.W - 1) / s.W;
    if (cfg.max_blocks) s.blocks = std::min<uint64_t>(s.blocks, cfg.max_blocks);
    return s;
}

// Shape of a team that is one thread-block cluster (or one block), or none.
// Up to 16 blocks pass their entries and minima through distributed shared
// memory behind one cluster barrier (~400 cycles) instead of the ring's
// fences and flags (~2400), but have a tenth of the SMs: taken for searches
// whose iterations hold a few hundred entries -- Q that small, 8-puzzles
// (181,440 states in all; 0.167 against 0.196 ms) and grids up to 2^17 cells
// (means of two grids, cluster and ring: 200^2 1.06 and 1.24 ms, 300^2 1.70
// and 1.88, 362^2 2.21 and 2.31; 420^2 2.79 and 2.67, 512^2 3.82 and 3.32).
// resident(warps, widest pop, blocks): whether a cluster of that many blocks of that
// shape fits on the GPU.
template <class Resident>
PlainShape cluster_shape(uint32_t kind, uint64_t cells, const gastar_config& cfg, uint64_t Q, Resident resident) {
    PlainShape s;
    const bool fixed = cfg.expansion_width || cfg.warps_per_block;
    s.W = cfg.warps_per_block ? std::min(16u, cfg.warps_per_block) : 8u;
    s.ew = cfg.expansion_width ? std::min(32u, cfg.expansion_width) : 4u;
    if (s.W > 8) return PlainShape();  // their kernel has no cluster teams for single instances
    const bool few = kind == KIND_SLIDING3 || (kind == KIND_GRID && cells <= (1ull << 17));
    uint64_t blocks = (Q + (uint64_t)s.ew * s.W - 1) / ((uint64_t)s.ew * s.W);
    if (blocks > kMaxClusterBlocks) {
        if (fixed || !few) return PlainShape();
        blocks = kMaxClusterBlocks;
    }
    if (cfg.max_blocks) blocks = std::min<uint64_t>(blocks, cfg.max_blocks);
    s.cluster = blocks > 1;
    s.blocks = blocks;
    if (s.cluster && !resident(s.W, widened(s, kind, cfg), (uint32_t)blocks)) return PlainShape();
    return s;
}

// The team of a solve: a cluster where one is taken, else a ring; one block
// where the caller's cap, or the work, leaves no more.  Which kind a team is
// follows from its blocks after the cap: a ring cut down to one block stages
// in shared memory and does not widen.
template <class Resident>
PlainShape plain_shape(uint32_t sms, uint32_t kind, uint64_t cells, const gastar_config& cfg, Resident resident) {
    const uint64_t Q = cfg.num_queues ? cfg.num_queues : 4096;
    PlainShape s = cluster_shape(kind, cells, cfg, Q, resident);
    if (!s.blocks) s = ring_shape(sms, kind, cells, cfg, Q);
    s.ew_wide = widened(s, kind, cfg);
    return s;
}

}  // namespace gastar
