// The GA* search: problem domains and the persistent search kernel.
//
// One "team" of thread blocks works on one instance; each warp of the team
// owns one open list (a warp-heap, optionally behind a bucket front).  An
// iteration is
//   pop    : every warp pops up to `ew` best entries (one per lane), drops
//            stale ones (table g lower than the entry's g) and goal states;
//   expand : a group of lanes per entry, one lane per move, generates the
//            successors, computes g and an incrementally updated h, and does
//            one insert-or-min on the duplicate-detection table per
//            successor; improved successors go to the block's stage area;
//   push   : one-block and cluster teams deal their stage chunks round-robin
//            (rotating offset) to their warps after a barrier, a cluster's
//            through distributed shared memory; in a ring team block c pushes
//            the stage region of block (c + i) mod blocks once that block has
//            flagged it ready (no team barrier);
//   check  : the search ends when the best goal cost is <= min f over all
//            open entries -- over the blocks' slots (one block, cluster) or
//            over the cut every block publishes with its stage region, one
//            hand-off per iteration (ring teams, tested kCutLag iterations
//            later).
// This is the reference's iteration (a_star.h:247-264: extract_nodes, three
// bitonic sorts, mark_duplicates, insert_unique_data, remove_updated_elements,
// insert_nodes_into_queues, two host reductions) as one device-resident loop
// with no host round trip.
#pragma once

#include <type_traits>

#include "device_common.cuh"
#include "engine_types.h"

namespace gastar {

// ---------------------------------------------------------------------------
// Sliding puzzle, n x n.  Keys pack the tile of cell i in bits [B*i, B*i+B)
// (B = 4 for n <= 4 in a uint64, B = 5 for n = 5 in 128 bits).  Moves follow
// the reference's neighbour_generator (a_star_sliding_puzzle.h:84-123):
// move 0/1/2/3 moves the blank row+1 / row-1 / col+1 / col-1, cost 1.
// ---------------------------------------------------------------------------
template <int N> struct SlidingDom {
    static constexpr int KW = N <= 4 ? 1 : 2;
    static constexpr int MAXN = 4;
    static constexpr int B = N <= 4 ? 4 : 5;
    static constexpr int C = N * N;
    using KeyT = std::conditional_t<KW == 1, uint64_t, unsigned __int128>;
    using Tab = std::conditional_t<KW == 1, HashTab64, HashTab128>;

    struct Ctx {
        KeyT goal, start;
        uint32_t ref_h, ref_moves;
        uint8_t md[C][C];  // md[t][p]: Manhattan distance of tile t placed at cell p
    };

    static __device__ __forceinline__ uint32_t field(KeyT k, int i) {
        return uint32_t(k >> (B * i)) & ((1u << B) - 1);
    }
    static __device__ __forceinline__ KeyT key_of(const Entry<KW>& e) {
        if constexpr (KW == 1) return e.k[0];
        else return (KeyT(e.k[1]) << 64) | KeyT(e.k[0]);
    }
    static __device__ __forceinline__ void set_key(Entry<KW>& e, KeyT k) {
        e.k[0] = uint64_t(k);
        if constexpr (KW == 2) e.k[1] = uint64_t(k >> 64);
    }
    static __device__ __forceinline__ KeyT desc_key(uint64_t lo, uint64_t hi) {
        if constexpr (KW == 1) return lo;
        else return (KeyT(hi) << 64) | KeyT(lo);
    }

    // Cell of the blank: the unique all-zero field, found with an AND-fold of
    // the complemented key.
    static __device__ __forceinline__ int blank_of(KeyT k) {
        KeyT y = ~k;
        KeyT z = y & (y >> 1);
        z = z & (z >> 2);
        if constexpr (B == 5) z = z & (y >> 4);
        KeyT mask = 0;
#pragma unroll
        for (int i = 0; i < C; ++i) mask |= KeyT(1) << (B * i);
        z &= mask;
        if constexpr (KW == 1) {
            return (__ffsll((long long)z) - 1) / B;
        } else {
            uint64_t lo = uint64_t(z), hi = uint64_t(z >> 64);
            int bit = lo ? __ffsll((long long)lo) - 1 : 64 + __ffsll((long long)hi) - 1;
            return bit / B;
        }
    }

    static __device__ void load(Ctx& c, const InstDesc& d) {
        const KeyT goal = desc_key(d.goal0, d.goal1);
        for (int i = threadIdx.x; i < C * C; i += blockDim.x) {
            const int t = i / C, p = i % C;
            int gp = 0;
            for (int q = 0; q < C; ++q)
                if ((int)field(goal, q) == t) gp = q;
            int v = abs(gp / N - p / N) + abs(gp % N - p % N);
            c.md[t][p] = d.heuristic == 2 ? 0 : (uint8_t)v;
        }
        if (threadIdx.x == 0) {
            c.goal = goal;
            c.start = desc_key(d.start0, d.start1);
            c.ref_h = d.heuristic == 1;
            c.ref_moves = d.moves == 1;
        }
        __syncthreads();
    }

    static __device__ __forceinline__ Tab make_tab(const InstDesc& d) {
        Tab t;
        t.s = d.table;
        t.mask = d.table_mask;
        t.max_probe = d.max_probe;
        return t;
    }
    static __device__ __forceinline__ uint64_t get(const Tab& t, KeyT k) {
        if constexpr (KW == 1) return tab_get(t, k);
        else return tab_get(t, uint64_t(k), uint64_t(k >> 64));
    }
    static __device__ __forceinline__ uint32_t start_f(const Ctx&, const InstDesc& d) { return d.f0; }
    // Parents are recorded by move code; the root's code is kRootMove.
    static constexpr uint32_t kRootCode = kRootMove;
    static constexpr bool kParentBySlot = false;
    // Two-step lookup of an entry's own value: look_begin issues the home
    // slot's reads (key words k0, k1 and value v), look_end resolves them,
    // probing on when the home slot holds another key.
    static __device__ __forceinline__ void look_begin(const Tab& t, KeyT k, uint64_t& k0, uint64_t& k1, uint64_t& v) {
        if constexpr (KW == 1) {
            k1 = 0;
            tab_look_begin(t, k, k0, v);
        } else {
            tab_look_begin(t, uint64_t(k), uint64_t(k >> 64), k0, k1, v);
        }
    }
    static __device__ __forceinline__ uint64_t look_end(const Tab& t, KeyT k, uint64_t k0, uint64_t k1, uint64_t v) {
        bool empty = k0 == kEmpty;
        if constexpr (KW == 2) empty = empty && k1 == kEmpty;
        if (empty) return kEmpty;
        const KeyT seen = desc_key(k0, k1);
        return seen == k ? v : get(t, k);
    }
    static __device__ __forceinline__ uint32_t code(int m, uint32_t) { return (uint32_t)m; }
    static __device__ __forceinline__ int insert(const Tab& t, KeyT k, uint64_t v, uint64_t& old,
                                                 uint32_t& slot) {
        if constexpr (KW == 1) return tab_insert(t, k, v, old, slot);
        else return tab_insert(t, uint64_t(k), uint64_t(k >> 64), v, old, slot);
    }
    static constexpr bool kDense = false;
    // Two-step claim: claim_begin issues the home slot's compare-and-swap (the
    // words it returned in k0, k1), claim_end resolves it (see tab_claim_end).
    static __device__ __forceinline__ void claim_begin(const Tab& t, KeyT k, uint64_t v, uint32_t& slot, uint64_t& k0,
                                                       uint64_t& k1) {
        if constexpr (KW == 1) tab_claim_begin(t, k, v, slot, k0, k1);
        else tab_claim_begin(t, uint64_t(k), uint64_t(k >> 64), slot, k0, k1);
    }
    static __device__ __forceinline__ int claim_end(const Tab& t, KeyT k, uint64_t v, uint32_t& slot, uint64_t k0,
                                                    uint64_t& k1) {
        if constexpr (KW == 1) return tab_claim_end(t, k, v, slot, k0, k1);
        else return tab_claim_end(t, uint64_t(k), uint64_t(k >> 64), v, slot, k0, k1);
    }
    static __device__ __forceinline__ bool is_goal(const Ctx& c, KeyT k) { return k == c.goal; }
    static __device__ __forceinline__ bool is_start(const Ctx& c, KeyT k) { return k == c.start; }
    // Low byte of an entry's priority word: the blank's cell and the move the
    // entry was reached with (4: the start), so that an expansion neither
    // searches the board for the blank nor looks its parent up.
    static __device__ __forceinline__ uint32_t tag(int m, KeyT nk, uint32_t cell) { return cell << 3 | (uint32_t)m; }
    static __device__ __forceinline__ uint32_t start_tag(KeyT k) { return tag(4, k, (uint32_t)blank_of(k)); }
    // Whether move m leads straight back to the parent of an entry with this tag.
    static __device__ __forceinline__ bool is_back(int m, uint32_t tag) { return (uint32_t)(m ^ 1) == (tag & 7u); }
    // What a lane's move does, fixed for a search: the shift of the blank's
    // cell and the cells it is possible from.
    struct Move {
        int dq;
        uint32_t from;
    };
    static __device__ __forceinline__ Move lane_move(const Ctx& c, int m) {
        constexpr uint32_t all = (1u << C) - 1u, row = (1u << N) - 1u;
        uint32_t left = 0;  // cells of the first column
#pragma unroll
        for (int i = 0; i < N; ++i) left |= 1u << (i * N);
        Move v;
        v.dq = m == 0 ? N : m == 1 ? -N : m == 2 ? 1 : -1;
        v.from = m == 0 ? all & ~(row << (C - N)) : m == 1 ? all & ~row : m == 2 ? all & ~(left << (N - 1)) : all & ~left;
        if (m >= 4 || (c.ref_moves && (m & 1))) v.from = 0;  // the reference's moves 1 and 3 never exist
        return v;
    }

    // The successor by a lane's move: the tile at the new blank cell q slides
    // to the old one p (whose field is zero).  `at` becomes q.
    static __device__ __forceinline__ bool succ(const Ctx& c, const Move& mv, int, KeyT k, uint32_t tag, uint32_t g,
                                                uint32_t h, KeyT& nk, uint32_t& ng, uint32_t& nh, uint32_t& at) {
        const int p = (int)(tag >> 3), q = p + mv.dq;
        if (!(mv.from >> p & 1u)) return false;
        const uint32_t t = field(k, q);
        nk = k ^ (KeyT(t) << (B * q)) ^ (KeyT(t) << (B * p));
        nh = h + c.md[t][p] - c.md[t][q];
        if (c.ref_h) nh = nh + c.md[0][q] - c.md[0][p];
        ng = g + 1;
        at = (uint32_t)q;
        return true;
    }

    // Parent of k when k was reached with move m: the blank moves back.
    static __device__ __forceinline__ KeyT parent(const Ctx&, const Tab&, KeyT k, uint32_t m) {
        const int p = blank_of(k);
        const int q = (m == 0) ? p - N : (m == 1) ? p + N : (m == 2) ? p - 1 : p + 1;
        const uint32_t t = field(k, q);
        return (k & ~(KeyT((1u << B) - 1) << (B * q))) | (KeyT(t) << (B * p));
    }
};

// ---------------------------------------------------------------------------
// Weighted grid, 8-connected (a_star_pathfinding.h:147-209).  Key = cell index
// y*W + x.  Move m shifts (x, y) by (DX[m], DY[m]); entering a cell costs its
// weight; weight 0 is impassable.  The duplicate-detection table is a dense
// value array indexed by cell.
// ---------------------------------------------------------------------------
// GridDom::dx(m) + 1 and GridDom::dy(m) + 1 in bits 2m..2m+1.
constexpr uint32_t kGridDxPack = 2u | 0u << 2 | 1u << 4 | 1u << 6 | 2u << 8 | 2u << 10 | 0u << 12 | 0u << 14;
constexpr uint32_t kGridDyPack = 1u | 1u << 2 | 2u << 4 | 0u << 6 | 2u << 8 | 0u << 10 | 2u << 12 | 0u << 14;

struct GridDom {
    static constexpr int KW = 1;
    static constexpr int MAXN = 8;
    using KeyT = uint64_t;
    using Tab = DenseTab;
    // Key: cell index | x << 32 | y << 48 (sides are at most 65535); the table
    // is indexed by the cell.
    static __host__ __device__ __forceinline__ KeyT make_key(uint32_t cell, uint32_t x, uint32_t y) {
        return (KeyT)cell | (KeyT)x << 32 | (KeyT)y << 48;
    }

    struct Ctx {
        const uint8_t* w;
        KeyT start;
        uint32_t W, H, goal, gx, gy, minw, href;
    };

    static constexpr __host__ __device__ int dx(int m) { return (m == 0 || m == 4 || m == 5) ? 1 : (m == 1 || m == 6 || m == 7) ? -1 : 0; }
    static constexpr __host__ __device__ int dy(int m) { return (m == 2 || m == 4 || m == 6) ? 1 : (m == 3 || m == 5 || m == 7) ? -1 : 0; }
    static __device__ __forceinline__ uint32_t inv(uint32_t m) { return m < 4 ? (m ^ 1) : 11 - m; }

    static __device__ __forceinline__ KeyT key_of(const Entry<1>& e) { return e.k[0]; }
    static __device__ __forceinline__ void set_key(Entry<1>& e, KeyT k) { e.k[0] = k; }

    static __device__ void load(Ctx& c, const InstDesc& d) {
        if (threadIdx.x == 0) {
            c.w = d.weights;
            c.W = d.W;
            c.H = d.H;
            c.goal = (uint32_t)d.goal0;
            const uint32_t st = (uint32_t)d.start0;
            c.start = make_key(st, st % d.W, st / d.W);
            c.gx = c.goal % d.W;
            c.gy = c.goal / d.W;
            c.minw = d.minw;
            c.href = d.heuristic;
        }
        __syncthreads();
    }
    static __device__ __forceinline__ Tab make_tab(const InstDesc& d) { return Tab{d.table}; }
    static __device__ __forceinline__ uint64_t get(const Tab& t, KeyT k) { return __ldcg(t.v + (uint32_t)k); }
    static __device__ __forceinline__ uint32_t start_f(const Ctx&, const InstDesc& d) { return d.f0; }
    static constexpr uint32_t kRootCode = kRootMove;
    static constexpr bool kParentBySlot = false;
    static constexpr bool kDense = true;
    // The cell is the slot: one atomicMin claims and lowers it.
    static __device__ __forceinline__ uint64_t lower(const Tab& t, KeyT k, uint64_t v) {
        return atomicMin(t.v + (uint32_t)k, (unsigned long long)v);
    }
    static __device__ __forceinline__ int insert(const Tab& t, KeyT k, uint64_t v, uint64_t& old,
                                                 uint32_t& slot) {
        old = lower(t, k, v);
        slot = (uint32_t)k;
        return old == kEmpty ? 1 : 0;
    }
    static __device__ __forceinline__ bool is_goal(const Ctx& c, KeyT k) { return (uint32_t)k == c.goal; }
    // Low byte of an entry's priority word: the move it was reached with.
    static __device__ __forceinline__ uint32_t tag(int m, KeyT, uint32_t) { return (uint32_t)m; }
    static __device__ __forceinline__ uint32_t start_tag(KeyT) { return kRootMove; }
    static __device__ __forceinline__ bool is_back(int m, uint32_t tag) {
        return tag != kRootMove && (uint32_t)m == inv(tag);
    }
    // What a lane's move does, fixed for a search.
    struct Move {
        int dx, dy, dcell;
    };
    static __device__ __forceinline__ Move lane_move(const Ctx& c, int m) {
        Move v;
        v.dx = (int)((kGridDxPack >> (2 * m)) & 3u) - 1;
        v.dy = (int)((kGridDyPack >> (2 * m)) & 3u) - 1;
        v.dcell = v.dy * (int)c.W + v.dx;
        return v;
    }
    static __device__ __forceinline__ uint32_t heur(const Ctx& c, int x, int y) {
        // 0: Chebyshev x min weight (admissible); 1: Manhattan (the reference's,
        // a_star_pathfinding.h:219-221); 2: zero.
        const uint32_t ax = (uint32_t)abs(x - (int)c.gx), ay = (uint32_t)abs(y - (int)c.gy);
        if (c.href == 1) return ax + ay;
        if (c.href == 2) return 0;
        return (ax > ay ? ax : ay) * c.minw;
    }
    // The cell a lane's move enters from k and its h; false off the board.
    static __device__ __forceinline__ bool step(const Ctx& c, const Move& mv, KeyT k, KeyT& nk, uint32_t& nh) {
        const int nx = (int)((uint32_t)(k >> 32) & 0xffffu) + mv.dx, ny = (int)(uint32_t)(k >> 48) + mv.dy;
        if ((uint32_t)nx >= c.W || (uint32_t)ny >= c.H) return false;
        nk = make_key((uint32_t)k + (uint32_t)mv.dcell, (uint32_t)nx, (uint32_t)ny);
        nh = heur(c, nx, ny);
        return true;
    }
    static __device__ __forceinline__ uint32_t weight(const Ctx& c, KeyT k) { return __ldg(c.w + (uint32_t)k); }
};

// ---------------------------------------------------------------------------
// Block-shared state.
// ---------------------------------------------------------------------------
struct CtaShared {
    TeamSlot slot[kSlots];  // iteration records of a one-block team
    TeamSlot agg;           // this block's share of the current iteration (multi-block teams)
    uint32_t agg_minheap, agg_err_prev;  // this block's heaps' min f and error of the previous push
    unsigned long long run[2];   // claims, expansions of the iterations tested so far
    unsigned long long mine[2];  // claims, expansions of this block (multi-block teams)
    unsigned long long base[2];  // claims, expansions before this launch
    unsigned long long wcnt[kMaxWarps][3];  // per warp: stale, generated, pushed in this launch
    unsigned long long t_start;  // search start on the device clock
    uint32_t dec_status, dec_best, dec_fmin, push_count, push_ok;  // ring teams: its two threads -> block
    // Cluster teams, warp 0 -> block: best, error, least open f, chunks in
    // all, entries per chunk; per block the chunks before its own, its entries.
    uint32_t plan[8], plan_before[kMaxClusterBlocks], plan_count[kMaxClusterBlocks];
    InstDesc desc;
    alignas(16) uint32_t inst;
    uint32_t ok, slice, pad1;  // slice: iterations before suspending (0 = to the end)
    union {
        SlidingDom<3>::Ctx s3;
        SlidingDom<4>::Ctx s4;
        SlidingDom<5>::Ctx s5;
        GridDom::Ctx g;
    } ctx;
};

extern __shared__ uint4 g_dyn_smem[];

// The block's shared state.  A function-local variable rather than a reference
// handed down: every access is then a shared-memory instruction instead of a
// generic one, and costs no register for the address.
__device__ __forceinline__ CtaShared& cta() {
    __shared__ CtaShared s;
    return s;
}
template <class D> __device__ __forceinline__ typename D::Ctx& shared_ctx() {  // plugins
    __shared__ typename D::Ctx c;
    return c;
}
__device__ __forceinline__ void slot_clear(TeamSlot& t) {
    t.count = t.err = t.claims = t.exps = t.perr = 0;
    t.minstage = t.best = t.minheap = kInf;
}
template <> __device__ __forceinline__ SlidingDom<3>::Ctx& shared_ctx<SlidingDom<3>>() { return cta().ctx.s3; }
template <> __device__ __forceinline__ SlidingDom<4>::Ctx& shared_ctx<SlidingDom<4>>() { return cta().ctx.s4; }
template <> __device__ __forceinline__ SlidingDom<5>::Ctx& shared_ctx<SlidingDom<5>>() { return cta().ctx.s5; }
template <> __device__ __forceinline__ GridDom::Ctx& shared_ctx<GridDom>() { return cta().ctx.g; }

// Barrier over the blocks of a multi-block team: one atomic arrival on a
// counter that only grows, a poll until it reaches the end of this barrier's
// range, a bounded wait (deadline on the device clock), and an abort flag so
// that one block giving up releases the others.
__device__ __forceinline__ bool team_sync_grid(TeamCtl* tc, uint32_t nctas, uint64_t timeout_ns) {
    CtaShared& sm = cta();
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t ok = 1;
        // Release: the block's writes (ordered before thread 0 by the block
        // barrier) become visible before the arrival does.
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        const unsigned long long old = atomicAdd(&tc->arrive, 1ull);
        const unsigned long long target = (old / nctas + 1) * nctas;
        const volatile unsigned long long* va = &tc->arrive;
        const volatile uint32_t* vab = &tc->abort;
        if (*va < target) {
            const uint64_t t0 = globaltimer_ns();
            for (uint32_t spin = 1;; ++spin) {
                if (*va >= target) break;
                if (*vab) {
                    ok = 0;
                    break;
                }
                if ((spin & 255u) == 0 && globaltimer_ns() - t0 > timeout_ns) {
                    atomicExch(&tc->abort, 1u);
                    ok = 0;
                    break;
                }
                if (spin > 64) __nanosleep(32);
            }
        }
        // Acquire: the other blocks' writes before their arrivals are visible.
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        if (*vab) ok = 0;
        sm.ok = ok;
    }
    __syncthreads();
    return sm.ok != 0;
}

__device__ __forceinline__ uint32_t ld_vol(const uint32_t* p) { return *(const volatile uint32_t*)p; }
__device__ __forceinline__ uint64_t ld_vol64(const unsigned long long* p) {
    return *(const volatile unsigned long long*)p;
}

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// Strong relaxed reads: followed by fence_acq_rel_gpu they form acquire
// patterns.  Strong relaxed writes: after fence_acq_rel_gpu they form release
// patterns.
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void red_relaxed_add_u32(uint32_t* p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits (one thread) until the ready word *p carries iteration `target`
// (high half >= target), given `w`, a value of *p read before and ordered by
// an acquire fence since; returns the word in `w`.  Bounded like
// team_wait_u32 below; returns with acquire ordering.
__device__ __forceinline__ bool team_wait_ready(const unsigned long long* p, uint32_t target,
                                                unsigned long long& w, TeamCtl* tc, uint64_t timeout_ns) {
    if ((uint32_t)(w >> 32) >= target) return true;
    const volatile uint32_t* vab = &tc->abort;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t spin = 1;; ++spin) {
        w = ld_acquire_u64(p);
        if ((uint32_t)(w >> 32) >= target) return true;
        if (*vab) return false;
        if ((spin & 255u) == 0 && globaltimer_ns() - t0 > timeout_ns) {
            atomicExch(&tc->abort, 1u);
            return false;
        }
        if (spin > 64) __nanosleep(32);
    }
}

// Waits (one thread) until *p >= target, given `seen`, a value of *p read
// before and ordered by an acquire fence since: bounded by the deadline,
// released by the team's abort flag; a timeout raises the flag.  Returns with
// acquire ordering: the writes the waited-for block made before raising *p
// are visible.
__device__ __forceinline__ bool team_wait_u32(const uint32_t* p, uint32_t target, uint32_t seen, TeamCtl* tc,
                                              uint64_t timeout_ns) {
    if (seen >= target) return true;
    const volatile uint32_t* vab = &tc->abort;
    const uint64_t t0 = globaltimer_ns();
    for (uint32_t spin = 1;; ++spin) {
        if (ld_acquire_u32(p) >= target) return true;
        if (*vab) return false;
        if ((spin & 255u) == 0 && globaltimer_ns() - t0 > timeout_ns) {
            atomicExch(&tc->abort, 1u);
            return false;
        }
        if (spin > 64) __nanosleep(32);
    }
}

// The blocks working on one instance.
struct TeamRef {
    uint32_t ctas;  // blocks in the team (1 = one block, barriers are __syncthreads)
    uint32_t rank;  // this block's rank in the team
    TeamCtl* ctl;   // control block of a multi-block team (device)
    void* stage;    // stage buffers of a multi-block team (device)
};

// Lanes of a warp that expand one entry: a power of two, one lane per move
// (domains with more than 32 moves take them 32 at a time).
constexpr int lanes_per_entry(int maxn) {
    int l = 1;
    while (l < maxn && l < 32) l *= 2;
    return l;
}
template <int LPE> __device__ constexpr uint32_t group_mask() {
    return LPE == 32 ? 0xffffffffu : (1u << (LPE & 31)) - 1u;
}


// How the blocks of a team work together: one block; the blocks of one
// thread-block cluster, through each other's shared memory; any number of
// blocks, through a ring of stage buffers in global memory.
enum TeamKind : int { TEAM_BLOCK, TEAM_CLUSTER, TEAM_RING };

// Barrier over the cluster's blocks; orders their shared and global memory.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// 16 bytes at shared-memory address `p` of the cluster's block `rank`.
__device__ __forceinline__ uint4 ld_cluster(const void* p, uint32_t rank) {
    uint4 v;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("{\n\t.reg .u32 ra;\n\tmapa.shared::cluster.u32 ra, %4, %5;\n\t"
                 "ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [ra];\n\t}"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(a), "r"(rank)
                 : "memory");
    return v;
}
template <int KW> __device__ __forceinline__ Entry<KW> ld_stage_cluster(const Entry<KW>* p, uint32_t rank) {
    Entry<KW> e;
#pragma unroll
    for (int v = 0; v < entry_vecs<KW>(); ++v) {
        const uint4 a = ld_cluster(reinterpret_cast<const uint4*>(p) + v, rank);
        set_word(e, 2 * v, (uint64_t(a.y) << 32) | a.x);
        set_word(e, 2 * v + 1, (uint64_t(a.w) << 32) | a.z);
    }
    return e;
}

template <class D, int MAXT, int TEAM>
__device__ __noinline__ void run_instance(const LaunchParams& P, const TeamRef tm) {
    constexpr int KW = D::KW;
    constexpr int MAXN = D::MAXN;
    constexpr bool ring = TEAM == TEAM_RING, cluster = TEAM == TEAM_CLUSTER;
    constexpr bool multi = ring || cluster;  // several blocks
    using E = Entry<KW>;
    using KeyT = typename D::KeyT;
    constexpr int LPE = lanes_per_entry(MAXN);  // lanes per entry: one per move
    constexpr int EPR = 32 / LPE;               // entries per expansion round
    // Rounds whose probes are in flight together.  Blocks of 9 to 16 warps
    // have 128 registers per thread: their grids take two rounds (152 grids of
    // 1000 x 1000, one block each: 28.9 -> 24.1 ms, with four 24.6), as far as
    // no register spills (with 120 bytes of spills two rounds took 34 ms);
    // their boards, bound by claims in cold tables, lose by it (15-puzzles
    // 21.7 -> 23.2 us an iteration).
    constexpr int RB = MAXT > 256 ? (D::kDense ? 2 : 1) : KW == 1 ? 4 : 2;
    // The 16-warp kernel has 128 registers a thread and mostly pops 32 at
    // once; the second way to pop cost its grids 100 bytes more of spilled
    // registers (152 grids of 1000 x 1000 one block each: 39 -> 43 ms).
    constexpr bool kFewPath = MAXT <= 256;
    CtaShared& sm = cta();
    const InstDesc& d = sm.desc;
    typename D::Ctx& ctx = shared_ctx<D>();
    const int lane = threadIdx.x & 31, warp = (int)uniform(threadIdx.x >> 5), W = blockDim.x >> 5;
    const uint32_t rank = multi ? tm.rank : 0u;
    InstCtl* const ctl = d.ctl;
    const bool leader = rank == 0 && threadIdx.x == 0;
    const uint32_t hid = rank * W + warp;
    // Blocks and clusters stage in shared memory (two buffers), ring teams in
    // global memory.
    const uint32_t region_cap =
        (uint32_t)stage_entries_per_buffer(W, d.ew_wide > d.ew ? d.ew_wide : d.ew, MAXN);  // widest pop of the search
    E* const snodes_all = reinterpret_cast<E*>(g_dyn_smem) + (ring ? 0u : 2 * region_cap);

    auto tsync = [&]() -> bool {
        if constexpr (ring) return team_sync_grid(tm.ctl, tm.ctas, P.barrier_timeout_ns);
        if constexpr (cluster) cluster_sync();
        else __syncthreads();
        return true;
    };

    D::load(ctx, d);

    WarpHeap<KW> hp;
    hp.nodes = reinterpret_cast<E*>(d.heap_nodes) + (size_t)hid * (d.heap_cap + 1) * 32;
    const uint32_t snodes = uniform(P.heap_snodes ? P.heap_snodes : kHeapSmemNodes) - 1;  // per warp: buffer + nodes
    hp.sn = snodes - 1;
    hp.snodes = snodes_all + warp * snodes * 32;
    hp.cap = uniform(d.heap_cap);
    // Bucket front: pages, links and free stacks in the instance's bucket
    // area; the push scratch (64 words per warp) in shared memory after the
    // heap nodes.
    Buckets<KW> bq;
    bq.P = uniform(P.buckets ? d.bq_pages : 0u);
    bq.pages = reinterpret_cast<E*>(d.bq_base) + (size_t)hid * bq.P * 32;
    bq.upd = reinterpret_cast<uint32_t*>(snodes_all + W * snodes * 32) + warp * 64;
    // Word tables of the bucket area, past every warp's pages: links, free
    // stacks (as many words each), saved states.
    auto bq_words = [&]() {
        return reinterpret_cast<uint32_t*>(reinterpret_cast<E*>(d.bq_base) + (size_t)d.heaps * bq.P * 32);
    };
    bq.link = bq_words() + (size_t)hid * bq.P;
    bq.fs_off = d.heaps * bq.P;
    bq_init(bq, lane);

    const uint32_t life = uniform(ld_vol(&ctl->life));
    if (!ring && threadIdx.x < kSlots) slot_clear(sm.slot[threadIdx.x]);
    if (lane < 3) sm.wcnt[warp][lane] = 0;
    uint32_t status = kInf;  // kInf while running / suspended
    uint32_t best_r;         // best goal cost seen (identical in every thread)
    bool have_prev;          // the previous iteration's slot holds the heaps' min
    if (life == LIFE_FRESH) {
        // Clear the table (0xff = empty key and value) across the whole team:
        // only the slots the previous solve claimed when they were recorded
        // (a length above the list's capacity means they were not) and few,
        // otherwise the whole table.  Listed offsets are the previous solve's, in the
        // same buffer; its table may have been larger than this solve's.
        const uint64_t stride = (uint64_t)(multi ? tm.ctas : 1u) * blockDim.x;
        const uint64_t tid = (uint64_t)rank * blockDim.x + threadIdx.x;
        // Where either clear will do, scattered stores costing about a
        // 32-byte sector each against streaming ones, the list is used while
        // it covers under a quarter of the table's words.
        const uint64_t cnt = d.touched ? ld_vol64(d.touched_count) : 0;
        if (d.touched && cnt <= d.touched_cap &&
            (!d.clear_either || cnt * d.prev_slot_words * 4 < d.table_words)) {
            for (uint64_t i = tid; i < cnt; i += stride) {
                const uint32_t w = __ldcg(d.touched + i);
                if (w == kTouchedHole) continue;
                for (uint32_t j = 0; j < d.prev_slot_words; ++j) __stcg(d.table + w + j, kEmpty);
            }
        } else {
            uint4* tp = reinterpret_cast<uint4*>(d.table);
            const uint64_t n16 = d.table_words / 2;
            for (uint64_t i = tid; i < n16; i += stride) __stcg(tp + i, make_uint4(~0u, ~0u, ~0u, ~0u));
            if ((d.table_words & 1) && tid == 0)  // odd cell count: last word
                __stcg(d.table + d.table_words - 1, kEmpty);
        }
        heap_init(hp);
        if (!tsync()) status = ST_BARRIER;
        if (hid == 0) {
            E s = inf_entry<KW>();
            s.prio = make_prio(D::start_f(ctx, d), 0, D::start_tag(ctx.start));
            D::set_key(s, ctx.start);
            heap_push(hp, lane == 0 ? s : inf_entry<KW>(), 1u, lane);
        }
        if (leader) {
            uint64_t old;
            uint32_t slot = 0;
            D::insert(D::make_tab(d), ctx.start, make_val(0, D::kRootCode), old, slot);
            if (d.touched) {
                *d.touched_count = 1;
                d.touched[0] = slot;
            }
            atomicAdd(&ctl->table_used, 1ull);
            ctl->t_start = globaltimer_ns();
        }
        best_r = uniform_if(D::is_goal(ctx, ctx.start)) ? 0u : kInf;
        have_prev = true;  // the start is the only open entry; every slot starts empty
    } else {
        heap_restore<kFewPath>(hp, d.heap_hdr + 2 * hid, lane);
        bq_restore(bq, bq_words() + 2 * (size_t)d.heaps * bq.P + (size_t)hid * kBucketStateWords, lane);
        best_r = uniform(ld_vol(&ctl->best));
        have_prev = false;
    }
    // Ring teams: each block stages into its own region of the ring
    // buffers and aggregates its counters and minima in shared memory; thread
    // 0 publishes them (ready word, cut slot).
    E* const stage0 = ring ? reinterpret_cast<E*>(tm.stage) : reinterpret_cast<E*>(g_dyn_smem);
    unsigned long long* const ready =
        ring ? reinterpret_cast<unsigned long long*>(stage0 + (size_t)kStageRing * tm.ctas * region_cap) : nullptr;
    if (ring && threadIdx.x == 0) {
        for (uint32_t r = 0; r < kStageRing; ++r) ready[(size_t)r * tm.ctas + rank] = 0;
        if (rank == 0)
            for (uint32_t k = 0; k < kCuts; ++k) {
                CutSlot& c = tm.ctl->cut[k];
                c.minf = kInf;
                c.claims = c.exps = 0;
                c.best = kInf;
                c.lossy = c.err = c.count = 0;
            }
    }
    if (status == kInf && !tsync()) status = ST_BARRIER;

    const int sub = lane & (LPE - 1);
    const typename D::Move mv = D::lane_move(ctx, sub);
    // This warp's current claim-list chunk (none reserved yet).
    unsigned long long t_base = 0;
    uint32_t t_used = kTouchedChunk;
    uint32_t fmin = uniform(D::start_f(ctx, d));  // min f over the open list at the last check
    uint32_t it = 0;
    const uint32_t slice = uniform(sm.slice);
    const uint32_t it0 = uniform(ld_vol(&ctl->iterations));
    if (threadIdx.x == 0) {
        slot_clear(sm.agg);
        sm.agg_minheap = kInf;
        sm.agg_err_prev = 0;
        // Budgets are tested against these (no global reads per iteration).
        sm.base[0] = ld_vol64(&ctl->table_used);
        sm.base[1] = ld_vol64(&ctl->expansions);
        sm.t_start = *(const volatile uint64_t*)&ctl->t_start;
        sm.run[0] = sm.run[1] = sm.mine[0] = sm.mine[1] = 0;
    }
    __syncthreads();
    // The first cut of a ring team holds the heaps as they are now.
    if (ring) {
        const uint32_t mf = open_minf(hp, bq);
        if (lane == 0 && mf != kInf) atomicMin(&sm.agg_minheap, mf);
    }
    while (status == kInf) {
        TeamSlot* const S = &sm.slot[it % kSlots];
        // Where this block's warps record the iteration: its slot, or for ring
        // teams the block aggregate.
        TeamSlot* const Sw = ring ? &sm.agg : S;
        E* const stage = ring ? stage0 + ((size_t)(it % kStageRing) * tm.ctas + rank) * region_cap
                               : reinterpret_cast<E*>(g_dyn_smem) + (it & 1) * region_cap;
        const typename D::Tab tab = D::make_tab(d);
        if (!ring && threadIdx.x == 0) {
            // Slot it+1 was last read right after the barrier of iteration
            // it-2; every warp is past that point, and none writes it before
            // the barrier of this iteration.
            slot_clear(sm.slot[(it + 1) % kSlots]);
            if (!cluster && it) {  // the previous iteration's counts are complete
                const TeamSlot& pv = sm.slot[(it + kSlots - 1) % kSlots];
                sm.run[0] += pv.claims;
                sm.run[1] += pv.exps;
            }
        }
        if (!ring && leader) {
            uint32_t err = 0;
            if (sm.base[0] + sm.run[0] > d.table_limit) err = ST_TABLE_FULL;
            else if (d.max_exp && sm.base[1] + sm.run[1] >= d.max_exp) err = ST_BUDGET;
            else if (d.max_iter && it0 + it + 1 >= d.max_iter) err = ST_BUDGET;
            else if (d.timeout_ns && globaltimer_ns() - sm.t_start > d.timeout_ns) err = ST_TIMEOUT;
            if (err) atomicMax(&S->err, err);
        }

        // ---- pop: up to ew entries per warp-heap, inside the window ----
        // With delta set, only entries with f <= fmin + delta are expanded
        // (delta-stepping); the rest wait for later iterations.
        const uint64_t lim = (d.delta && (uint64_t)fmin + d.delta < 0xffffffffull)
                                 ? ((uint64_t)(fmin + d.delta + 1) << 32)
                                 : kInfPrio;
        E e;
        const uint32_t cnt =
            open_pop<kFewPath>(hp, bq, uniform(d.wide_after && it0 + it >= d.wide_after ? d.ew_wide : d.ew), lim, e, lane);
        bool act = (uint32_t)lane < cnt;
        const KeyT k = D::key_of(e);
        const uint32_t g = prio_g(e.prio);
        uint32_t self = 0, goal_g = kInf, n_stale = 0;
        if (act && D::is_goal(ctx, k)) {
            // The goal is never expanded (a_star.h:80-83); its cost counts
            // unless a lower g for it is already known.
            if ((uint32_t)(D::get(tab, k) >> 32) >= g) goal_g = g;
            act = false;
        }
        if constexpr (D::kParentBySlot) {
            // Plugins record parents by slot: the entry's own slot is needed
            // before its successors are inserted.
            bool stale = false;
            if (act && (uint32_t)(D::get_self(tab, k, self) >> 32) < g) {
                stale = true;
                act = false;
            }
            n_stale = __popc(__ballot_sync(kFull, stale));
        }

        // ---- expand: one lane per (entry, move) ----
        // Lane l of round r takes move l % LPE of entry r * EPR + l / LPE.
        // Bound by round trips to L2/HBM and by the SM's rate of scattered
        // accesses (measured per SM: one L2 load per cycle, one L2 atomic per
        // 2.1, seven cycles per random HBM sector); per round one probe
        // instruction covers EPR whole neighbourhoods (a grid cell's three
        // rows share sectors), RB rounds' probes are in flight together, and
        // a warp that popped few entries runs few rounds.  A plain 4096^2
        // grid pops four entries per warp and iteration: with one lane per
        // entry and the moves in sequence its expansion took 8.9 k cycles of
        // a 27 k cycle iteration; this alone took it from 74.4 to 48.9 ms, and
        // it is 3.4 k of 11.4 k cycles now (31 ms).  The
        // lane of the move straight back to the parent, which has no
        // successor, checks whether the entry is stale.
        const uint32_t live = __ballot_sync(kFull, act);
        // The popped lanes as a vote: the round tests below are then uniform
        // branches to the compiler too.
        const uint32_t popped = __ballot_sync(kFull, (uint32_t)lane < cnt);
        const uint32_t lt = (1u << lane) - 1u;
        uint32_t n_gen = 0, n_claim = 0, pushed = 0, fstage = kInf;
        uint32_t flags = 0;  // 1: the table is full, 2: a cost out of range
        for (uint32_t r0 = 0; r0 < (uint32_t)LPE && (popped >> (r0 * EPR)) != 0; r0 += RB) {
#pragma unroll 1
            for (int mg = 0; mg < MAXN; mg += LPE) {
                const int m = mg + sub;
                KeyT nk[RB];
                uint32_t ng[RB], nf[RB], wt[RB];
                uint64_t old[RB], seen[RB], own_v[RB];
                uint32_t slot[RB];
                uint32_t code[RB];  // parent as recorded in the table
                uint32_t at[RB];    // puzzles: the blank's cell
                bool ok[RB], own[RB];
                // Issue: nothing here waits for a probe, so RB rounds' probes
                // are in flight together.
#pragma unroll
                for (int j = 0; j < RB; ++j) {
                    ok[j] = own[j] = false;
                    if (r0 + j >= (uint32_t)LPE || (popped >> ((r0 + j) * EPR)) == 0) continue;  // warp-uniform
                    const int src = (int)((r0 + j) * EPR) + lane / LPE;
                    const E x = shfl_idx(e, src);
                    const KeyT xk = D::key_of(x);
                    const uint32_t xg = prio_g(x.prio), tag = prio_pm(x.prio);
                    uint32_t xself = 0, nh = 0;
                    if constexpr (D::kParentBySlot) xself = __shfl_sync(kFull, self, src);
                    const bool on = ((live >> src) & 1u) && m < MAXN;
                    if constexpr (!D::kParentBySlot) own[j] = on && D::is_back(m, tag);
                    ng[j] = xg;
                    if constexpr (D::kDense) {
                        // The neighbour's weight and value load together; a
                        // value that is already as good needs no atomic
                        // (four of five do not: 7.5 M of 9.8 M generated on
                        // a 1021^2 grid), and a load costs half an atomic.
                        ok[j] = on && !own[j] && D::step(ctx, mv, xk, nk[j], nh);
                        if (own[j]) nk[j] = xk;
                        if (ok[j] || own[j]) old[j] = D::get(tab, nk[j]);
                        if (ok[j]) wt[j] = D::weight(ctx, nk[j]);
                        nf[j] = nh;
                    } else {
                        ok[j] = on && !own[j] &&
                                D::succ(ctx, mv, m, xk, tag, xg, prio_f(x.prio) - xg, nk[j], ng[j], nh, at[j]);
                        n_gen += __popc(__ballot_sync(kFull, ok[j]));
                        if (ok[j] && ng[j] > kMaxG) {
                            flags |= 2u;
                            ok[j] = false;
                        }
                        nf[j] = ng[j] + nh;
                        ok[j] = ok[j] && nf[j] < best_r;  // cannot beat the best goal found
                        code[j] = D::code(m, xself);
                        if (ok[j]) D::claim_begin(tab, nk[j], make_val(ng[j], code[j]), slot[j], seen[j], old[j]);
                        if constexpr (!D::kParentBySlot) {
                            if (own[j]) {
                                nk[j] = xk;
                                D::look_begin(tab, xk, seen[j], old[j], own_v[j]);
                            }
                        }
                    }
                }
                if constexpr (D::kDense) {
#pragma unroll
                    for (int j = 0; j < RB; ++j) {
                        if (r0 + j >= (uint32_t)LPE || (popped >> ((r0 + j) * EPR)) == 0) continue;
                        // Stale: the table's g went below the entry's own.
                        const uint32_t sb = __ballot_sync(kFull, own[j] && (uint32_t)(old[j] >> 32) < ng[j]);
                        const bool stale = (sb >> (lane & ~(LPE - 1)) & group_mask<LPE>()) != 0;
                        n_stale += __popc(sb);
                        ok[j] = ok[j] && !stale && wt[j] != 0;  // 0: obstacle
                        n_gen += __popc(__ballot_sync(kFull, ok[j]));
                        if (ok[j]) ng[j] += wt[j];
                        if (ok[j] && ng[j] > kMaxG) {
                            flags |= 2u;
                            ok[j] = false;
                        }
                        nf[j] += ng[j];
                        const uint64_t v = make_val(ng[j], (uint32_t)m);
                        ok[j] = ok[j] && nf[j] < best_r && v < old[j];
                        if (ok[j]) old[j] = D::lower(tab, nk[j], v);
                    }
                }
                uint32_t acc_at[RB], clm_at[RB];
                uint32_t total = 0, claimed = 0;
#pragma unroll
                for (int j = 0; j < RB; ++j) {
                    acc_at[j] = clm_at[j] = kInf;
                    if (r0 + j >= (uint32_t)LPE || (popped >> ((r0 + j) * EPR)) == 0) continue;
                    bool stale = false;
                    int cl = -1;
                    if constexpr (D::kDense) {
                        if (ok[j]) cl = old[j] == kEmpty ? 1 : 0;
                    } else {
                        if (ok[j]) cl = D::claim_end(tab, nk[j], make_val(ng[j], code[j]), slot[j], seen[j],
                                                     old[j]);
                        if (ok[j] && cl < 0) flags |= 1u;
                        if constexpr (!D::kParentBySlot) {
                            // A stale entry's successors are real paths and
                            // stay in the table, but are not queued; the
                            // entry with the lower g covers them.
                            const bool st =
                                own[j] && (uint32_t)(D::look_end(tab, nk[j], seen[j], old[j], own_v[j]) >> 32) < ng[j];
                            const uint32_t sb = __ballot_sync(kFull, st);
                            stale = (sb >> (lane & ~(LPE - 1)) & group_mask<LPE>()) != 0;
                            n_stale += __popc(sb);
                        }
                    }
                    const bool in = ok[j] && cl >= 0;
                    const bool acc = in && !stale && (uint32_t)(old[j] >> 32) > ng[j];
                    const uint32_t ab = __ballot_sync(kFull, acc), cb = __ballot_sync(kFull, in && cl == 1);
                    if (acc) {
                        acc_at[j] = total + __popc(ab & lt);
                        fstage = nf[j] < fstage ? nf[j] : fstage;
                        if (D::is_goal(ctx, nk[j]) && ng[j] < goal_g) goal_g = ng[j];
                    }
                    if (in && cl == 1) clm_at[j] = claimed + __popc(cb & lt);
                    total += __popc(ab);
                    claimed += __popc(cb);
                }
                n_claim += claimed;
                pushed += total;
                // Stage the improved successors: one atomic per warp reserves the range.
                if (total) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(&Sw->count, total);
                    base = __shfl_sync(kFull, base, 0);
#pragma unroll
                    for (int j = 0; j < RB; ++j) {
                        if (acc_at[j] != kInf) {
                            E out = inf_entry<KW>();
                            out.prio = make_prio(nf[j], ng[j], D::tag(m, nk[j], D::kDense ? 0u : at[j]));
                            D::set_key(out, nk[j]);
                            st_stage<ring>(stage + base + acc_at[j], out);
                        }
                    }
                }
                if (d.touched && claimed) {  // record claimed slots for the next solve's clear
                    // Fill the warp's chunk; a group that overruns it
                    // continues in a newly reserved one.
                    const uint32_t room = kTouchedChunk - t_used;
                    unsigned long long nb = 0;
                    if (claimed > room) {
                        if (lane == 0) nb = atomicAdd(d.touched_count, (unsigned long long)kTouchedChunk);
                        nb = __shfl_sync(kFull, nb, 0);
                    }
#pragma unroll
                    for (int j = 0; j < RB; ++j) {
                        if (clm_at[j] != kInf) {
                            const uint32_t pos = clm_at[j];
                            const unsigned long long at = pos < room ? t_base + t_used + pos : nb + (pos - room);
                            if (at < d.touched_cap) d.touched[at] = slot[j];
                        }
                    }
                    if (claimed > room) {
                        t_base = nb;
                        t_used = claimed - room;
                    } else {
                        t_used += claimed;
                    }
                }
            }
        }
        {
            // The counts are warp-uniform; minima over the lanes with one
            // reduction each.
            const uint32_t smin = __reduce_min_sync(kFull, fstage);
            goal_g = __reduce_min_sync(kFull, goal_g);
            // One reduction for both flags, not a vote each: grids never raise
            // the first (the rule at uniform()).
            flags = uniform(flags);
            if (lane == 0) {
                const uint32_t n_exp = __popc(live) - (D::kParentBySlot ? 0u : n_stale);
                sm.wcnt[warp][0] += n_stale;
                sm.wcnt[warp][1] += n_gen;
                sm.wcnt[warp][2] += pushed;
                if (n_exp) atomicAdd(&Sw->exps, n_exp);
                if (n_claim) atomicAdd(&Sw->claims, n_claim);
                if (smin != kInf) atomicMin(&Sw->minstage, smin);
                if (goal_g != kInf) atomicMin(&Sw->best, goal_g);
                if (flags & 1u) atomicMax(&Sw->err, (uint32_t)ST_TABLE_FULL);
                if (flags & 2u) atomicMax(&Sw->err, (uint32_t)ST_COST_RANGE);
            }
        }
        if constexpr (ring) {
            // ---- one hand-off per iteration: publish cut `it` and this
            // block's stage region, then wait for the region this block
            // pushes and test cut it - kCutLag (a_star.h:260-262) ----
            // Thread 0 publishes the region and waits for the one it takes;
            // the second warp's first thread (of a one-warp block, thread 0
            // in between) does the same for the cuts.  A chain of round trips
            // to L2 (fence 1.0 k cycles, store to load 1.4 k or more), so the
            // region, which the push waits for, goes first and by itself (behind the cut's
            // updates: grid 1021^2 6.11 ms, so: 5.91).
            __syncthreads();  // every warp's stage writes and counters are done
            const uint32_t cut_thread = W > 1 ? 32u : 0u;
            unsigned long long* const rw = ready + (size_t)(it % kStageRing) * tm.ctas;
            unsigned long long wfrom = 0;
            uint32_t from = 0, mine = 0;
            if (threadIdx.x == 0) {
                from = (rank + it) % tm.ctas;
                // The awaited word is read first, relaxed; its round trip
                // overlaps the fence, which orders it before what follows
                // (acquire) and every warp's stage writes, ordered before
                // thread 0 by the block barrier, before the ready word (release).
                wfrom = ld_relaxed_u64(rw + from);
                mine = sm.agg.count;
                sm.agg.count = 0;
                fence_acq_rel_gpu();
                st_relaxed_u64(rw + rank, ((unsigned long long)(it + 1) << 32) | mine);
            }
            if (threadIdx.x == cut_thread) {
                CutSlot* cuts = tm.ctl->cut;
                const CutSlot* t = cuts + (it + kCuts - kCutLag) % kCuts;
                const uint32_t tseen = it >= kCutLag ? ld_relaxed_u32(&t->count) : 0u;
                const uint32_t lossy = sm.agg.err ? sm.agg.err : sm.agg_err_prev;
                uint32_t err = 0;
                if (rank == 0) {
                    if (it >= 2 * kCutLag + 2) {  // every block has read it; none writes it yet
                        CutSlot* r = cuts + (it - 2 * kCutLag - 2) % kCuts;
                        r->minf = kInf;
                        r->claims = r->exps = 0;
                        r->best = kInf;
                        r->lossy = r->err = r->count = 0;
                    }
                    if (d.max_iter && it0 + it + 1 >= d.max_iter) err = ST_BUDGET;
                    if (d.timeout_ns && globaltimer_ns() - sm.t_start > d.timeout_ns) err = ST_TIMEOUT;
                }
                // Cut `it` covers this block's heaps after the previous push
                // (a superset of what is left after this iteration's pops) and
                // what this iteration staged.
                CutSlot* c = cuts + it % kCuts;
                const uint32_t cm = sm.agg_minheap < sm.agg.minstage ? sm.agg_minheap : sm.agg.minstage;
                if (cm != kInf) atomicMin(&c->minf, cm);
                // The team's counts are for its budgets only.
                if (sm.agg.claims && d.table_limit != ~0ull)
                    atomicAdd(&c->claims, (unsigned long long)sm.agg.claims);
                if (sm.agg.exps && d.max_exp) atomicAdd(&c->exps, (unsigned long long)sm.agg.exps);
                sm.mine[0] += sm.agg.claims;
                sm.mine[1] += sm.agg.exps;
                if (sm.agg.best != kInf) atomicMin(&c->best, sm.agg.best);
                if (lossy) atomicCAS(&c->lossy, 0u, lossy);
                if (err) atomicCAS(&c->err, 0u, err);
                // The cut's updates, and every warp's reads of the last
                // region, precede the arrival (release); the early read
                // precedes everything after (acquire).
                fence_acq_rel_gpu();
                red_relaxed_add_u32(&c->count, 1u);
                sm.agg.err = sm.agg.claims = sm.agg.exps = 0;  // not the count
                sm.agg.minstage = sm.agg.best = kInf;
                sm.agg_minheap = kInf;
                sm.agg_err_prev = 0;
                uint32_t dec = kInf, dbest = kInf, dfmin = kInf;
                if (it >= kCutLag) {
                    // Waits only while a block is more than kCutLag iterations behind.
                    if (!team_wait_u32(&t->count, tm.ctas, tseen, tm.ctl, P.barrier_timeout_ns)) {
                        dec = ST_BARRIER;
                    } else {
                        const uint32_t open_f = ld_vol(&t->minf);
                        dbest = ld_vol(&t->best);
                        uint32_t tl = ld_vol(&t->lossy), te = ld_vol(&t->err);
                        // Budgets from the team's totals, the same in every block.
                        if (d.table_limit != ~0ull) sm.run[0] += ld_vol64(&t->claims);
                        if (d.max_exp) sm.run[1] += ld_vol64(&t->exps);
                        if (!tl && sm.base[0] + sm.run[0] > d.table_limit) tl = ST_TABLE_FULL;
                        if (!te && d.max_exp && sm.base[1] + sm.run[1] >= d.max_exp) te = ST_BUDGET;
                        const uint32_t bb = dbest < best_r ? dbest : best_r;
                        if (tl) dec = tl;  // an iteration that lost entries proves nothing
                        else if (bb != kInf && bb <= open_f) dec = ST_OK;
                        else if (te) dec = te;
                        else if (open_f == kInf) dec = ST_NO_PATH;
                        dfmin = open_f;
                    }
                }
                sm.dec_status = dec;
                sm.dec_best = dbest;
                sm.dec_fmin = dfmin;
            }
            if (threadIdx.x == 0) {
                uint32_t got = 1;
                if (from == rank)
                    wfrom = mine;
                else if (!team_wait_ready(rw + from, it + 1, wfrom, tm.ctl, P.barrier_timeout_ns))
                    got = 0;
                sm.push_count = (uint32_t)wfrom;
                sm.push_ok = got;
            }
            __syncthreads();
            {
                const uint32_t db = uniform(sm.dec_best), df = uniform(sm.dec_fmin);
                best_r = db < best_r ? db : best_r;
                if (df != kInf) fmin = df;
                status = uniform(sm.push_ok) ? uniform(sm.dec_status) : (uint32_t)ST_BARRIER;
            }
            if (status != kInf) break;
        } else {
            if (!tsync()) {
                status = ST_BARRIER;
                break;
            }
            // ---- termination test (a_star.h:260-262), one iteration behind ----
            // Open entries now: heaps after the previous push (>= that slot's
            // min) minus this iteration's pops, plus this iteration's stage.
            const TeamSlot* pv = &sm.slot[(it + kSlots - 1) % kSlots];
            uint32_t err, open_f, sb;
            if constexpr (cluster) {
                // One warp per block reads the blocks' slots through
                // distributed shared memory (lane j block j's), reduces them
                // and plans the push; the others wait for its record (all
                // warps reading all slots took no less, 1.5 k cycles).
                if (warp == 0) {
                    uint4 a = make_uint4(0, kInf, kInf, 0), q = make_uint4(0, 0, kInf, 0);
                    uint2 n = make_uint2(0, 0);
                    if ((uint32_t)lane < tm.ctas) {
                        a = ld_cluster(&S->count, (uint32_t)lane);
                        q = ld_cluster(&pv->claims, (uint32_t)lane);
                        if (rank == 0) {
                            const uint4 c = ld_cluster(&S->claims, (uint32_t)lane);
                            n = make_uint2(c.x, c.y);
                        }
                    }
                    if (!have_prev) q.z = kInf, q.w = 0;
                    const uint32_t b_min = __reduce_min_sync(kFull, a.z);
                    const uint32_t e_max = __reduce_max_sync(kFull, a.w > q.w ? a.w : q.w);
                    const uint32_t f_min = __reduce_min_sync(kFull, a.y < q.z ? a.y : q.z);
                    if (rank == 0) {  // the team's counts, for the budgets
                        const uint32_t nc = __reduce_add_sync(kFull, n.x), ne = __reduce_add_sync(kFull, n.y);
                        if (lane == 0) {
                            sm.run[0] += nc;
                            sm.run[1] += ne;
                        }
                    }
                    const uint32_t NW = tm.ctas * (uint32_t)W;
                    const uint32_t total = __reduce_add_sync(kFull, a.x);
                    // A block's last chunk may be short: a chunk of slack per
                    // block keeps the chunks at one per warp.
                    const uint32_t room = W > 1 ? NW - tm.ctas : NW;
                    const uint32_t per = (total + room - 1) / room;
                    const uint32_t cs = per < 32 ? (per ? per : 1u) : 32u;
                    const uint32_t chunks = (a.x + cs - 1) / cs;
                    uint32_t upto = chunks;  // chunks of blocks 0..lane
#pragma unroll
                    for (int o = 1; o < (int)kMaxClusterBlocks; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(kFull, upto, o);
                        if (lane >= o) upto += t;
                    }
                    if (lane < (int)kMaxClusterBlocks) {
                        sm.plan_before[lane] = upto - chunks;
                        sm.plan_count[lane] = a.x;
                    }
                    if (lane == (int)kMaxClusterBlocks - 1) {
                        sm.plan[0] = b_min;
                        sm.plan[1] = e_max;
                        sm.plan[2] = f_min;
                        sm.plan[3] = upto;
                        sm.plan[4] = cs;
                    }
                }
                __syncthreads();
                sb = uniform(ld_vol(&sm.plan[0]));
                err = uniform(ld_vol(&sm.plan[1]));
                open_f = uniform(ld_vol(&sm.plan[2]));
            } else {
                sb = uniform(ld_vol(&S->best));
                err = uniform(ld_vol(&S->err));
                open_f = uniform(ld_vol(&S->minstage));
                if (have_prev) {
                    const uint32_t pe = uniform(ld_vol(&pv->perr)), mf = uniform(ld_vol(&pv->minheap));
                    err = pe > err ? pe : err;
                    open_f = mf < open_f ? mf : open_f;
                }
            }
            best_r = sb < best_r ? sb : best_r;
            // An iteration that lost entries (full table or heap) proves nothing.
            if (err == ST_TABLE_FULL || err == ST_HEAP_FULL || err == ST_COST_RANGE) status = err;
            else if (have_prev && best_r != kInf && best_r <= open_f) status = ST_OK;
            else if (err) status = err;
            else if (have_prev && open_f == kInf) status = ST_NO_PATH;
            if (status != kInf) break;
            if (open_f != kInf) fmin = open_f;
        }

        // ---- push ----
        // One-block teams deal the block's stage chunks round-robin with a
        // rotating offset; cluster teams deal all blocks' chunks the same way
        // over all of the cluster's warps; in a ring team block r takes the
        // region of block (r + it) mod blocks, so work moves between blocks
        // every iteration, and its warps deal that region's chunks.
        // Chunks hold up to 32 entries, fewer when that gives every warp a
        // share: a warp expands its pops in rounds.
        {
            bool hfull = false;
            if constexpr (cluster) {
                const uint32_t NW = tm.ctas * (uint32_t)W;
                const uint32_t nch = uniform(ld_vol(&sm.plan[3])), cs = uniform(ld_vol(&sm.plan[4]));
                for (uint32_t c = (hid + NW - it % NW) % NW; c < nch; c += NW) {
                    // The block whose chunks c falls among.
                    const uint32_t before = lane < (int)kMaxClusterBlocks ? ld_vol(&sm.plan_before[lane]) : kInf;
                    const uint32_t from = 31 - __clz(__ballot_sync(kFull, (uint32_t)lane < tm.ctas && before <= c));
                    const uint32_t at = (c - uniform(ld_vol(&sm.plan_before[from]))) * cs;
                    const uint32_t left = uniform(ld_vol(&sm.plan_count[from])) - at;
                    const uint32_t m = left < cs ? left : cs;
                    const E x = (uint32_t)lane < m ? ld_stage_cluster(stage + at + lane, from) : inf_entry<KW>();
                    if (!open_push(hp, bq, x, m, lane)) {
                        hfull = true;
                        break;
                    }
                }
            } else {
                uint32_t total;
                const E* src;
                uint32_t first;
                if constexpr (ring) {
                    const uint32_t from = (rank + it) % tm.ctas;
                    total = uniform(sm.push_count);
                    src = stage0 + ((size_t)(it % kStageRing) * tm.ctas + from) * region_cap;
                    first = ((uint32_t)warp + it) % (uint32_t)W;
                } else {
                    total = uniform(ld_vol(&S->count));
                    src = stage;
                    first = ((uint32_t)warp + (uint32_t)W - it % (uint32_t)W) % (uint32_t)W;
                }
                const uint32_t per = (total + (uint32_t)W - 1) / (uint32_t)W;
                const uint32_t cs = per < 32 ? per : 32u;
                const uint32_t nch = cs ? (total + cs - 1) / cs : 0u;
                for (uint32_t c = first; c < nch; c += (uint32_t)W) {
                    const uint32_t idx = c * cs + (uint32_t)lane;
                    const uint32_t m = total - c * cs < cs ? total - c * cs : cs;
                    E x = (uint32_t)lane < m ? ld_stage<ring>(src + idx) : inf_entry<KW>();
                    if (!open_push(hp, bq, x, m, lane)) {
                        hfull = true;
                        break;
                    }
                }
            }
            const uint32_t mf = open_minf(hp, bq);
            if (lane == 0) {
                atomicMin(ring ? &sm.agg_minheap : &S->minheap, mf);
                if (hfull) atomicCAS(ring ? &sm.agg_err_prev : &S->perr, 0u, (uint32_t)ST_HEAP_FULL);
            }
        }
        ++it;
        have_prev = true;
        if (slice && it >= slice) break;  // suspend
    }

    if (lane == 0) atomicMax(&ctl->max_nodes, hp.max_n);
    if (d.touched)  // the unused rest of the warp's chunk
        for (uint32_t i = t_used + (uint32_t)lane; i < kTouchedChunk; i += 32)
            if (t_base + i < d.touched_cap) d.touched[t_base + i] = kTouchedHole;
    {  // this launch's counters
        if constexpr (cluster) cluster_sync();  // no block reads another's slots or stage any more
        else __syncthreads();
        if (threadIdx.x == 0) {
            if constexpr (cluster) {
                if (rank == 0) {  // the team's
                    sm.mine[0] = sm.run[0];
                    sm.mine[1] = sm.run[1];
                }
            } else if constexpr (!ring) {
                // Iterations 0 .. it - 1 were counted when the next one began;
                // the one the loop left by, or the last before a suspension:
                const uint32_t last = status == kInf ? it - 1 : it;
                const TeamSlot& t = sm.slot[last % kSlots];
                sm.mine[0] = sm.run[0] + t.claims;
                sm.mine[1] = sm.run[1] + t.exps;
            }
            if (sm.mine[1]) atomicAdd(&ctl->expansions, sm.mine[1]);
            if (sm.mine[0]) atomicAdd(&ctl->table_used, sm.mine[0]);
        }
        if (lane == 0) {
            if (sm.wcnt[warp][0]) atomicAdd(&ctl->stale, sm.wcnt[warp][0]);
            if (sm.wcnt[warp][1]) atomicAdd(&ctl->generated, sm.wcnt[warp][1]);
            if (sm.wcnt[warp][2]) atomicAdd(&ctl->pushes, sm.wcnt[warp][2]);
        }
    }
    if (status == kInf) {
        // Suspending: fold in what the iterations not tested yet found -- a
        // goal popped there is in no heap any more -- and stop on entries
        // they lost.
        if constexpr (ring) {
            if (threadIdx.x == 0) {
                CutSlot* c = tm.ctl->cut + it % kCuts;
                if (sm.agg.best != kInf) atomicMin(&c->best, sm.agg.best);
                const uint32_t lossy = sm.agg.err ? sm.agg.err : sm.agg_err_prev;
                if (lossy) atomicCAS(&c->lossy, 0u, lossy);
            }
            if (!tsync()) {
                status = ST_BARRIER;
            } else {
                if (threadIdx.x == 0) {
                    uint32_t b = best_r, lossy = 0;
                    for (uint32_t x = it > kCutLag ? it - kCutLag : 0; x <= it; ++x) {
                        const CutSlot* c = tm.ctl->cut + x % kCuts;
                        const uint32_t cb = ld_vol(&c->best);
                        b = cb < b ? cb : b;
                        if (!lossy) lossy = ld_vol(&c->lossy);
                    }
                    sm.dec_best = b;
                    sm.dec_status = lossy ? lossy : kInf;
                }
                __syncthreads();
                best_r = uniform(sm.dec_best);
                status = uniform(sm.dec_status);
            }
        } else if constexpr (cluster) {
            uint32_t pe = 0;  // raised by the last push of any block
            if ((uint32_t)lane < tm.ctas)
                pe = ld_cluster(&sm.slot[(it + kSlots - 1) % kSlots].claims, (uint32_t)lane).w;
            if (it > 0 && __reduce_max_sync(kFull, pe) != 0) status = ST_HEAP_FULL;
            cluster_sync();
        } else if (it > 0 && uniform(ld_vol(&sm.slot[(it + kSlots - 1) % kSlots].perr)) == ST_HEAP_FULL) {
            status = ST_HEAP_FULL;  // raised by the last push
        }
    }
    if (status == kInf) {  // suspended: keep the search state resident
        heap_save(hp, d.heap_hdr + 2 * hid, lane);
        bq_save(bq, bq_words() + 2 * (size_t)d.heaps * bq.P + (size_t)hid * kBucketStateWords, lane);
        if (leader) {
            ctl->best = best_r;
            ctl->iterations = it0 + it;
            __threadfence();
            ctl->life = LIFE_RUNNING;
        }
    } else if (leader) {
        ctl->best = best_r;
        ctl->iterations = it0 + it;
        ctl->status = status;
        ctl->t_end = globaltimer_ns();
        __threadfence();
        ctl->life = LIFE_DONE;
    }
}

template <uint32_t KINDS, int MAXT, int TEAM>
__device__ __forceinline__ void dispatch(const LaunchParams& P, const TeamRef tm) {
    switch (cta().desc.kind) {
        case KIND_SLIDING3:
            if constexpr ((KINDS & kind_bit(KIND_SLIDING3)) != 0) run_instance<SlidingDom<3>, MAXT, TEAM>(P, tm);
            break;
        case KIND_SLIDING4:
            if constexpr ((KINDS & kind_bit(KIND_SLIDING4)) != 0) run_instance<SlidingDom<4>, MAXT, TEAM>(P, tm);
            break;
        case KIND_SLIDING5:
            if constexpr ((KINDS & kind_bit(KIND_SLIDING5)) != 0) run_instance<SlidingDom<5>, MAXT, TEAM>(P, tm);
            break;
        case KIND_GRID:
            if constexpr ((KINDS & kind_bit(KIND_GRID)) != 0) run_instance<GridDom, MAXT, TEAM>(P, tm);
            break;
        default:
            break;
    }
}

// The block's next instance into its shared state; false: none is left.  A
// function of its own so that nothing of it, hoisted out of the caller's loop,
// holds registers across a search: the 16-warp kernel's one-block searches
// spilled 120 bytes for grids and 132 for boards with it in the loop, 8 and 44
// without (spill loads; 24-puzzles 228, ring-team grids 68).
inline __device__ __noinline__ bool take_instance(const LaunchParams& P) {
    CtaShared& sm = cta();
    if (threadIdx.x == 0) sm.inst = atomicAdd(P.next, 1u);
    __syncthreads();
    const uint32_t i = sm.inst;
    if (i >= P.n_insts) return false;
    if (threadIdx.x == 0) {
        const uint32_t slot = P.order ? P.order[i] : i;
        sm.desc = P.insts[slot];
        sm.slice = P.slices ? P.slices[slot] : P.slice_iters;
    }
    __syncthreads();
    return true;
}

// Persistent search kernel.
//  * plain (team_ctas > 1): every block works on instance 0 (one cluster, or a
//    cooperative launch);
//  * batch/serve: blocks of the heavy teams first take heavy instances together
//    (grids), then every block takes instances one block each from a work counter.
// MAXT bounds the block size: 256 threads (8 warps) leave the compiler up to
// 255 registers per thread; the all-kinds kernel has a second instantiation
// for 16-warp blocks (batch/serve), capped at 128 registers.
template <uint32_t KINDS, int MAXT = 256>
__global__ void __launch_bounds__(MAXT, 1) search_kernel(const __grid_constant__ LaunchParams P) {
    CtaShared& sm = cta();
    // Single-kind kernels are the plain engine's; the all-kinds kernel of
    // 16-warp blocks serves both.
    constexpr bool plain = KINDS != kKindsAll || MAXT > 256, many = KINDS == kKindsAll;
    if (plain && P.team_ctas > 1) {
        if (threadIdx.x == 0) {
            sm.desc = P.insts[0];
            sm.slice = P.slice_iters;
        }
        __syncthreads();
        if constexpr (plain) {
            const TeamRef tm{P.team_ctas, blockIdx.x, P.team, P.stage};
            if constexpr (MAXT <= 256)
                if (P.cluster) {
                    dispatch<KINDS, MAXT, TEAM_CLUSTER>(P, tm);
                    return;
                }
            dispatch<KINDS, MAXT, TEAM_RING>(P, tm);
        }
        return;
    }
    if (many && P.n_heavy && blockIdx.x < P.heavy_teams * P.heavy_team) {
        const uint32_t t = blockIdx.x / P.heavy_team, rank = blockIdx.x % P.heavy_team;
        if (P.cluster) {
            if constexpr (many) {
                for (;;) {
                    if (rank == 0 && threadIdx.x == 0) sm.inst = atomicAdd(P.heavy_next, 1u);
                    cluster_sync();
                    const uint32_t i = uniform(ld_cluster(&sm.inst, 0).x);
                    cluster_sync();  // read by all before the first block's next use of it, or its exit
                    if (i >= P.n_heavy) break;
                    if (threadIdx.x == 0) {
                        const uint32_t slot = P.heavy_order[i];
                        sm.desc = P.insts[slot];
                        sm.slice = P.slices ? P.slices[slot] : P.slice_iters;
                    }
                    __syncthreads();
                    dispatch<kind_bit(KIND_GRID), MAXT, TEAM_CLUSTER>(P, TeamRef{P.heavy_team, rank, nullptr, nullptr});
                    __syncthreads();
                }
            }
        } else {
            TeamCtl* tc = P.heavy_ctl + t;
            const TeamRef tm{P.heavy_team, rank, tc,
                             reinterpret_cast<char*>(P.heavy_stage) + (size_t)t * P.heavy_stage_bytes};
            for (;;) {
                // Every block of the team is done with the previous instance here.
                if (!team_sync_grid(tc, P.heavy_team, P.barrier_timeout_ns)) break;
                if (rank == 0 && threadIdx.x == 0) {
                    for (uint32_t k = 0; k < kCuts; ++k) {
                        tc->cut[k].minf = kInf;
                        tc->cut[k].claims = tc->cut[k].exps = 0;
                        tc->cut[k].best = kInf;
                        tc->cut[k].lossy = 0;
                        tc->cut[k].err = 0;
                        tc->cut[k].count = 0;
                    }
                    tc->inst = atomicAdd(P.heavy_next, 1u);
                }
                if (!team_sync_grid(tc, P.heavy_team, P.barrier_timeout_ns)) break;
                const uint32_t i = ld_vol(&tc->inst);
                if (i >= P.n_heavy) break;
                if (threadIdx.x == 0) {
                    const uint32_t slot = P.heavy_order[i];
                    sm.desc = P.insts[slot];
                    sm.slice = P.slices ? P.slices[slot] : P.slice_iters;
                }
                __syncthreads();
                if constexpr (many) dispatch<kind_bit(KIND_GRID), MAXT, TEAM_RING>(P, tm);
            }
        }
        __syncthreads();
    }
    while (take_instance(P)) {
        dispatch<KINDS, MAXT, TEAM_BLOCK>(P, TeamRef{1, 0, nullptr, nullptr});
        __syncthreads();
    }
}

// Path rebuild (a_star.h:268-281 walked one <<<1,1>>> launch per step): for
// each finished puzzle one thread follows parent moves from the goal to the
// start and writes the states goal-first (grids: walk_grid_path, a warp per
// instance).  An instance that has the arena to itself (a launch of one)
// writes as it walks; otherwise it walks twice -- once to count, once to
// write into a slice of the shared arena reserved with one atomic.
template <class D>
__device__ void walk_path(const InstDesc& d, typename D::Ctx& ctx, unsigned long long* arena,
                          unsigned long long arena_words, unsigned long long* arena_used, bool own_arena,
                          unsigned long long base_off = 0) {
    InstCtl* ctl = d.ctl;
    const typename D::Tab tab = D::make_tab(d);
    // Every step lowers g by at least 1, so a walk longer than best + 1 states
    // means a damaged table.
    const uint64_t limit = (uint64_t)ctl->best + 2;
    if (own_arena) {
        const uint64_t cap = arena_words / D::KW;
        uint64_t len = 0;
        for (typename D::KeyT k = ctx.goal;;) {
            if (len >= cap || len > limit) {  // the host retries with room for best + 1 states
                ctl->status = ST_PATH_CAP;
                ctl->path_len = 0;
                return;
            }
            unsigned long long* o = arena + len * D::KW;
            o[0] = (uint64_t)k;
            if constexpr (D::KW == 2) o[1] = (uint64_t)(k >> 64);
            ++len;
            if (D::is_start(ctx, k)) break;
            const uint64_t v = D::get(tab, k);
            const uint32_t m = (uint32_t)v;
            if (v == kEmpty || m == D::kRootCode) {
                ctl->status = ST_PATH_CAP;
                ctl->path_len = 0;
                return;
            }
            k = D::parent(ctx, tab, k, m);
        }
        ctl->path_len = (uint32_t)len;
        ctl->path_off = base_off;
        atomicAdd(arena_used, (unsigned long long)(len * D::KW));
        return;
    }
    uint64_t len = 1;
    for (typename D::KeyT k = ctx.goal; !D::is_start(ctx, k); ++len) {
        const uint64_t v = D::get(tab, k);
        const uint32_t m = (uint32_t)v;
        if (v == kEmpty || m == D::kRootCode || len > limit) {
            ctl->status = ST_PATH_CAP;
            ctl->path_len = 0;
            return;
        }
        k = D::parent(ctx, tab, k, m);
    }
    const unsigned long long words = len * D::KW;
    const unsigned long long off = atomicAdd(arena_used, words);
    ctl->path_len = (uint32_t)len;
    if (off + words > arena_words) {
        ctl->status = ST_PATH_CAP;
        return;
    }
    ctl->path_off = off;
    typename D::KeyT k = ctx.goal;
    for (uint64_t i = 0; i < len; ++i) {
        unsigned long long* o = arena + off + i * D::KW;
        o[0] = (uint64_t)k;
        if constexpr (D::KW == 2) o[1] = (uint64_t)(k >> 64);
        if (i + 1 < len) k = D::parent(ctx, tab, k, (uint32_t)D::get(tab, k));
    }
}

// Builds the domain context without the block-wide table fill (one thread).
template <int N> __device__ void sliding_ctx_min(typename SlidingDom<N>::Ctx& c, const InstDesc& d) {
    c.goal = SlidingDom<N>::desc_key(d.goal0, d.goal1);
    c.start = SlidingDom<N>::desc_key(d.start0, d.start1);
}

// Grid path rebuild by one warp.  A dependent table load per step costs a
// DRAM round trip (~0.6 us; a 8192^2 grid's path has ~9k steps), so the warp
// loads the values of a kPathWin x kPathWin window of cells in one round
// trip (lane j reads column j of every row, 32 loads in flight) into shared
// memory, and lane 0 follows parent moves inside it.  Parents lead toward the
// start, so the window is placed with the current cell kPathMargin cells from
// its edge away from the start: up to ~28 steps per load.
constexpr int kPathWin = 32, kPathMargin = 3, kPathWarps = 4;

static __device__ __forceinline__ int path_win_origin(int c, int s, int n) {
    int o = s < c ? c - (kPathWin - 1 - kPathMargin) : s > c ? c - kPathMargin : c - kPathWin / 2;
    if (o > n - kPathWin) o = n - kPathWin;
    return o < 0 ? 0 : o;
}

// Walks the grid path of `d` from the goal to the start (the whole warp
// calls it).  With `out`, lane 0 writes the cells goal-first, at most `cap`
// of them (`capped` is set when there were more).  Returns the number of
// states, or 0 for a damaged table: a cell without a move, a move leaving the
// grid, or more than `limit` states.
static __device__ uint64_t walk_grid_warp(const InstDesc& d, unsigned long long* win, unsigned long long* out,
                                   uint64_t cap, uint64_t limit, int lane, bool& capped) {
    const int W = (int)d.W, H = (int)d.H;
    const int sx = (int)(d.start0 % d.W), sy = (int)(d.start0 / d.W);
    int cx = (int)(d.goal0 % d.W), cy = (int)(d.goal0 / d.W);
    unsigned long long len = 0;
    int state = 0;  // 0: walking, 1: at the start, 2: damaged table
    bool cp = false;
    while (state == 0) {
        const int x0 = path_win_origin(cx, sx, W), y0 = path_win_origin(cy, sy, H);
        const int x = x0 + lane;
        unsigned long long v[kPathWin];
#pragma unroll
        for (int r = 0; r < kPathWin; ++r)
            v[r] = (x < W && y0 + r < H) ? __ldcg(d.table + (size_t)(y0 + r) * W + x) : kEmpty;
#pragma unroll
        for (int r = 0; r < kPathWin; ++r) win[r * kPathWin + lane] = v[r];
        __syncwarp();
        if (lane == 0) {
            // Window-local coordinates; a step is one shared-memory load and
            // a few integer operations (dx, dy from 2-bit fields).  Inside
            // the window a cell outside the grid holds kEmpty (loaded so), so
            // the grid bounds are checked only when the walk leaves it.
            int lx = cx - x0, ly = cy - y0;
            const int slx = sx - x0, sly = sy - y0;
            unsigned long long cell = (unsigned long long)cy * W + cx;
            for (;;) {
                if (out) {
                    if (len < cap) out[len] = cell;
                    else cp = true;
                }
                ++len;
                if (lx == slx && ly == sly) {
                    state = 1;
                    break;
                }
                const unsigned long long t = win[ly * kPathWin + lx];
                const uint32_t m = (uint32_t)t;
                if (len > limit || t == kEmpty || m >= 8) {
                    state = 2;
                    break;
                }
                const int dx = (int)((kGridDxPack >> (2 * m)) & 3u) - 1;
                const int dy = (int)((kGridDyPack >> (2 * m)) & 3u) - 1;
                lx -= dx;
                ly -= dy;
                cell -= (long long)dx + (long long)dy * W;
                if ((unsigned)lx >= (unsigned)kPathWin || (unsigned)ly >= (unsigned)kPathWin) break;
            }
            cx = x0 + lx;
            cy = y0 + ly;
            if (state == 0 && (cx < 0 || cx >= W || cy < 0 || cy >= H)) state = 2;
        }
        state = __shfl_sync(kFull, state, 0);
        cx = __shfl_sync(kFull, cx, 0);
        cy = __shfl_sync(kFull, cy, 0);
        len = __shfl_sync(kFull, len, 0);
        __syncwarp();  // the window is rewritten next
    }
    capped = __shfl_sync(kFull, (int)cp, 0) != 0;
    return state == 1 ? len : 0;
}

// walk_path for grids, by a whole warp (same arena protocol and statuses).
static __device__ void walk_grid_path(const InstDesc& d, unsigned long long* win, unsigned long long* arena,
                               unsigned long long arena_words, unsigned long long* arena_used, bool own_arena,
                               int lane, unsigned long long base_off) {
    InstCtl* ctl = d.ctl;
    const uint64_t limit = (uint64_t)ctl->best + 2;
    bool capped = false;
    if (own_arena) {
        const uint64_t len = walk_grid_warp(d, win, arena, arena_words, limit, lane, capped);
        if (lane != 0) return;
        if (!len || capped) {  // the host retries with room for best + 1 states
            ctl->status = ST_PATH_CAP;
            ctl->path_len = 0;
            return;
        }
        ctl->path_len = (uint32_t)len;
        ctl->path_off = base_off;
        atomicAdd(arena_used, (unsigned long long)len);
        return;
    }
    const uint64_t len = walk_grid_warp(d, win, nullptr, 0, limit, lane, capped);
    if (!len) {
        if (lane == 0) {
            ctl->status = ST_PATH_CAP;
            ctl->path_len = 0;
        }
        return;
    }
    unsigned long long off = 0;
    if (lane == 0) {
        off = atomicAdd(arena_used, (unsigned long long)len);
        ctl->path_len = (uint32_t)len;
    }
    off = __shfl_sync(kFull, off, 0);
    if (off + len > arena_words) {
        if (lane == 0) ctl->status = ST_PATH_CAP;
        return;
    }
    if (lane == 0) ctl->path_off = off;
    walk_grid_warp(d, win, arena + off, len, limit, lane, capped);
}

// One warp per finished instance: grids walk windows (walk_grid_path),
// puzzles walk on lane 0.  Blocks of kPathWarps warps, a window of shared
// memory per warp.  With `offs` (n + 1 prefix offsets) instance i owns arena
// words [offs[i], offs[i+1]) and writes as it walks; otherwise a launch of
// one owns the arena and larger launches reserve slices with an atomic.
static __global__ void __launch_bounds__(kPathWarps * 32)
    path_kernel(const InstDesc* insts, uint32_t n, unsigned long long* arena, unsigned long long arena_words,
                unsigned long long* arena_used, const unsigned long long* offs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * kPathWarps + warp;
    if (i >= n) return;  // warp-uniform from here on: every lane reads the same instance
    const InstDesc& d = insts[i];
    if (d.ctl->life != LIFE_DONE || d.ctl->status != ST_OK) return;
    const bool own = offs || n == 1;
    const unsigned long long base = offs ? offs[i] : 0ull;
    unsigned long long* a = arena + base;
    const unsigned long long words = offs ? offs[i + 1] - base : arena_words;
    if (d.kind == KIND_GRID) {
        unsigned long long* win = reinterpret_cast<unsigned long long*>(g_dyn_smem) + warp * kPathWin * kPathWin;
        walk_grid_path(d, win, a, words, arena_used, own, lane, base);
        return;
    }
    if (lane != 0) return;
    switch (d.kind) {
        case KIND_SLIDING3: {
            SlidingDom<3>::Ctx c;
            sliding_ctx_min<3>(c, d);
            walk_path<SlidingDom<3>>(d, c, a, words, arena_used, own, base);
            break;
        }
        case KIND_SLIDING4: {
            SlidingDom<4>::Ctx c;
            sliding_ctx_min<4>(c, d);
            walk_path<SlidingDom<4>>(d, c, a, words, arena_used, own, base);
            break;
        }
        case KIND_SLIDING5: {
            SlidingDom<5>::Ctx c;
            sliding_ctx_min<5>(c, d);
            walk_path<SlidingDom<5>>(d, c, a, words, arena_used, own, base);
            break;
        }
        default:
            break;
    }
}

}  // namespace gastar
