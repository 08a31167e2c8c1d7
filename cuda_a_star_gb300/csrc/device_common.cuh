// Device building blocks of the GA* engine: entries, warp sorting networks,
// the warp-cooperative batched binary heap and the duplicate-detection tables.
//
// Reference (michalborkowski96/cuda_a_star) counterparts:
//   HeapEntry / QueueValue ordering        heaps.h:14-23, a_star.h:55-66
//   HeapsDevice::extract/insert/remove     heaps.h:93-160   -> WarpHeap (below)
//   FancyHashmap mass insert + statuses    fancy_hashmap.h:32-167, 336-340
//                                          -> insert-or-min with CAS (below)
//   bitonic_sort network (global memory)   bitonic_sort.h:107-143
//                                          -> register/shuffle networks (below)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gastar {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint64_t kEmpty = ~0ull;      // empty table key / value
constexpr uint64_t kInfPrio = ~0ull;    // priority of a padding entry
constexpr uint32_t kInf = 0xffffffffu;
constexpr uint32_t kRootMove = 0xffu;   // parent move of the start state

// Device status codes; the numeric values are the gastar_status values of the C ABI.
enum : uint32_t {
    ST_OK = 0, ST_NO_PATH = 1, ST_BUDGET = 2, ST_TIMEOUT = 3, ST_HEAP_FULL = 4,
    ST_TABLE_FULL = 5, ST_PATH_CAP = 6, ST_BARRIER = 7, ST_BAD_INPUT = 8, ST_COST_RANGE = 13,
};
static_assert(ST_HEAP_FULL > ST_BUDGET && ST_HEAP_FULL > ST_TIMEOUT && ST_TABLE_FULL > ST_HEAP_FULL &&
                  ST_COST_RANGE > ST_TABLE_FULL,
              "an iteration's status is the largest code raised: lost entries before budgets");
enum : uint32_t { LIFE_FRESH = 0, LIFE_RUNNING = 1, LIFE_DONE = 2 };

__host__ __device__ __forceinline__ uint64_t mix64(uint64_t x) {
    // SplitMix64 output function (Steele, Lea, Flood 2014).
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

// Priority word: f in bits 63..32, (2^24-1 - g) in bits 31..8 and a tag of
// the domain in bits 7..0 (the move that produced the entry; puzzles: with the
// blank's cell), so that one unsigned comparison gives
// the reference's order "lower f first, equal f -> higher g first"
// (QueueValue::operator<, a_star.h:58-63) and a popped entry knows its parent
// move without a table lookup.  Costs are limited to kMaxG.
constexpr uint32_t kMaxG = 0xffffffu;
__host__ __device__ __forceinline__ uint64_t make_prio(uint32_t f, uint32_t g, uint32_t pm = 0xffu) {
    return (uint64_t(f) << 32) | (uint64_t(kMaxG - g) << 8) | (pm & 0xffu);
}
__host__ __device__ __forceinline__ uint32_t prio_f(uint64_t p) { return uint32_t(p >> 32); }
__host__ __device__ __forceinline__ uint32_t prio_g(uint64_t p) { return kMaxG - (uint32_t(p >> 8) & kMaxG); }
__host__ __device__ __forceinline__ uint32_t prio_pm(uint64_t p) { return uint32_t(p) & 0xffu; }

// Table value word: g in the high half, parent move in the low byte; one
// 64-bit atomicMin keeps the lowest g and, among equal g, the lowest move.
__host__ __device__ __forceinline__ uint64_t make_val(uint32_t g, uint32_t move) {
    return (uint64_t(g) << 32) | move;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A value that is the same in every lane, as a warp reduction's result.  The
// compiler takes what a load, a shuffle or threadIdx yields for per-lane data
// and guards every branch on it with convergence code; the result of a
// reduction or a vote is uniform to it, and so are the branches.
//
// Rule: no vote or reduction may have an operand that is a compile-time constant
// in any instantiation; code that some domains never run goes under `if
// constexpr`.  A vote on a constant (grids: a flag that only hash tables raise)
// left all lanes of every warp waiting on the GPU.  Its source was well formed:
// the lanes of a warp came to every full-mask operation together when the same
// code was run on the host, and every branch around one is on a vote's or a
// reduction's result.  So it is kept out by a test that compiles every
// instantiation for the host (tests/test_vote_predicates.py).
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_or_sync(kFull, v); }
__device__ __forceinline__ bool uniform_if(bool c) { return __any_sync(kFull, c) != 0; }

// ---------------------------------------------------------------------------
// Heap entries: a priority word and KW 64-bit key words (KW = 1..4), padded to
// a multiple of 16 bytes: 16 B for 64-bit keys, 32 B for 128..192-bit keys,
// 48 B for 256-bit keys.
// ---------------------------------------------------------------------------
template <int KW> struct alignas(16) Entry {
    static constexpr int NK = KW + ((KW % 2 == 0) ? 1 : 0);  // key words incl. padding
    uint64_t prio;
    uint64_t k[NK];
};
template <int KW> __host__ __device__ constexpr int entry_vecs() { return (1 + Entry<KW>::NK) / 2; }

template <int KW> __device__ __forceinline__ Entry<KW> inf_entry() {
    Entry<KW> e;
    e.prio = kInfPrio;
#pragma unroll
    for (int j = 0; j < Entry<KW>::NK; ++j) e.k[j] = 0;
    return e;
}

template <int KW> __device__ __forceinline__ Entry<KW> shfl_idx(const Entry<KW>& e, int src) {
    Entry<KW> r;
    r.prio = __shfl_sync(kFull, e.prio, src);
#pragma unroll
    for (int j = 0; j < Entry<KW>::NK; ++j) r.k[j] = j < KW ? __shfl_sync(kFull, e.k[j], src) : 0;
    return r;
}

template <int KW> __device__ __forceinline__ Entry<KW> shfl_xor(const Entry<KW>& e, int m) {
    Entry<KW> r;
    r.prio = __shfl_xor_sync(kFull, e.prio, m);
#pragma unroll
    for (int j = 0; j < Entry<KW>::NK; ++j) r.k[j] = j < KW ? __shfl_xor_sync(kFull, e.k[j], m) : 0;
    return r;
}

template <int KW> __device__ __forceinline__ void set_word(Entry<KW>& e, int w, uint64_t v) {
    if (w == 0) e.prio = v;
    else e.k[w - 1] = v;
}
template <int KW> __device__ __forceinline__ uint64_t get_word(const Entry<KW>& e, int w) {
    return w == 0 ? e.prio : e.k[w - 1];
}

// L2-coherent loads/stores (heap nodes and stage buffers are handed between
// launches and, in multi-block teams, between blocks).
template <int KW> __device__ __forceinline__ Entry<KW> ld_entry(const Entry<KW>* p) {
    Entry<KW> e;
    const uint4* s = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int v = 0; v < entry_vecs<KW>(); ++v) {
        const uint4 a = __ldcg(s + v);
        set_word(e, 2 * v, (uint64_t(a.y) << 32) | a.x);
        set_word(e, 2 * v + 1, (uint64_t(a.w) << 32) | a.z);
    }
    return e;
}
template <int KW> __device__ __forceinline__ void st_entry(Entry<KW>* p, const Entry<KW>& e) {
    uint4* d = reinterpret_cast<uint4*>(p);
#pragma unroll
    for (int v = 0; v < entry_vecs<KW>(); ++v) {
        const uint64_t a = get_word(e, 2 * v), b = get_word(e, 2 * v + 1);
        __stcg(d + v, make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32)));
    }
}

// Stage-buffer access: shared memory for one-block teams (plain generic
// accesses), global memory shared by the blocks of a multi-block team
// (L2-coherent accesses, since the buffer is refilled every iteration).
template <bool GLOBAL, int KW> __device__ __forceinline__ Entry<KW> ld_stage(const Entry<KW>* p) {
    if constexpr (GLOBAL) return ld_entry(p);
    Entry<KW> e;
    const uint4* s = reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int v = 0; v < entry_vecs<KW>(); ++v) {
        const uint4 a = s[v];
        set_word(e, 2 * v, (uint64_t(a.y) << 32) | a.x);
        set_word(e, 2 * v + 1, (uint64_t(a.w) << 32) | a.z);
    }
    return e;
}
template <bool GLOBAL, int KW> __device__ __forceinline__ void st_stage(Entry<KW>* p, const Entry<KW>& e) {
    if constexpr (GLOBAL) {
        st_entry(p, e);
        return;
    }
    uint4* d = reinterpret_cast<uint4*>(p);
#pragma unroll
    for (int v = 0; v < entry_vecs<KW>(); ++v) {
        const uint64_t a = get_word(e, 2 * v), b = get_word(e, 2 * v + 1);
        d[v] = make_uint4(uint32_t(a), uint32_t(a >> 32), uint32_t(b), uint32_t(b >> 32));
    }
}

// ---------------------------------------------------------------------------
// Warp sorting networks over one entry per lane (ascending by prio).
// Every compare-exchange decides from the same predicate in both lanes of a
// pair, so equal priorities never duplicate or drop an entry.
// ---------------------------------------------------------------------------
template <int KW> __device__ __forceinline__ Entry<KW> bitonic_clean(Entry<KW> x, int lane) {
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
        Entry<KW> y = shfl_xor(x, j);
        bool lower = !(lane & j);
        bool sw = lower ? (y.prio < x.prio) : (x.prio < y.prio);
        if (sw) x = y;
    }
    return x;
}

// Sorts by (f, g): the network moves only the priority words, with the lane in
// place of the tag (half the shuffles of 16-byte entries, a quarter of 32-byte
// ones), and the entries follow in one step.  Entries of equal f and g come in
// lane order, which the merges below, comparing whole words, do not mind: what
// they return is in (f, g) order too.
template <int KW> __device__ __forceinline__ Entry<KW> sort32(const Entry<KW>& x, int lane) {
    uint64_t k = (x.prio & ~0xffull) | (uint32_t)lane;
#pragma unroll
    for (int n = 2; n <= 32; n <<= 1) {
#pragma unroll
        for (int j = n >> 1; j > 0; j >>= 1) {
            const uint64_t y = __shfl_xor_sync(kFull, k, j);
            const bool lower = !(lane & j), asc = (n == 32) || !(lane & n);
            if ((lower == asc) == (y < k)) k = y;
        }
    }
    return shfl_idx(x, (int)(k & 31u));
}

// Merges two ascending 32-entry vectors: lo = 32 smallest, hi = 32 largest,
// both ascending.
template <int KW>
__device__ __forceinline__ void merge2(const Entry<KW>& a, const Entry<KW>& b, Entry<KW>& lo,
                                       Entry<KW>& hi, int lane) {
    Entry<KW> br = shfl_idx(b, 31 - lane);
    bool bl = br.prio < a.prio;
    lo = bl ? br : a;
    hi = bl ? a : br;
    lo = bitonic_clean(lo, lane);
    hi = bitonic_clean(hi, lane);
}

// Element idx (0..63) of the concatenation lo ++ hi; all lanes must call.
template <int KW>
__device__ __forceinline__ Entry<KW> pick(const Entry<KW>& lo, const Entry<KW>& hi, int idx) {
    Entry<KW> a = shfl_idx(lo, idx & 31);
    Entry<KW> b = shfl_idx(hi, idx & 31);
    return idx < 32 ? a : b;
}

// ---------------------------------------------------------------------------
// Warp-cooperative batched binary heap.
//
// One warp owns one heap.  A node holds 32 entries sorted ascending; the heap
// order is node-wise (every entry of a node <= every entry of its children),
// so the root holds the 32 best entries of the tree.  A partial buffer of
// < 32 entries and nodes 0..sn-1 (the top levels; sn is chosen per launch
// from the shared memory left on the SM) live in shared memory for the
// lifetime of a launch, the rest are 512-byte (or 1 KiB) blocks in global
// memory read and written with one coalesced access per lane.  Root and
// buffer stay out of registers: they are touched a few times per iteration,
// and the 16-warp kernel has 128 registers per thread (holding them there
// spilled ~500 bytes per thread, whose local-memory traffic was 15x the
// search's own loads).  Replaces the reference's one-thread-per-heap
// binary heaps with their key->slot index (heaps.h:93-177, device_hashmap.h):
// stale entries are dropped at pop time instead of being erased (lazy
// deletion).
// ---------------------------------------------------------------------------

template <int KW> struct WarpHeap {
    Entry<KW>* nodes;   // (cap + 1) * 32 entries; node `cap` stores the saved partial buffer
    Entry<KW>* snodes;  // shared memory: the partial buffer, then nodes 0..sn-1
    uint32_t cap;       // tree nodes available (>= sn)
    uint32_t sn;        // nodes below sn live in shared memory
    uint32_t N;         // full nodes in the tree (warp-uniform)
    uint32_t pc;        // entries in the partial buffer (warp-uniform)
    uint32_t pf;        // their least f (kInf: none; warp-uniform)
    uint32_t ro;        // entries of the root already popped: its first ones (warp-uniform)
    uint32_t max_n;     // high-water mark of N
    bool sorted;        // they are in ascending order (warp-uniform)
};

// The partial buffer collects pushes in arrival order and is sorted only when
// a pop needs its best entries or it overflows into the tree: a search that
// keeps a warp at a few entries per iteration (grids, small puzzles) then
// neither sorts nor merges anything.
template <int KW> __device__ __forceinline__ Entry<KW> ld_part(const WarpHeap<KW>& h, int lane) {
    return (uint32_t)lane < h.pc ? ld_stage<false>(h.snodes + lane) : inf_entry<KW>();
}
template <int KW> __device__ __forceinline__ Entry<KW> ld_part_sorted(const WarpHeap<KW>& h, int lane) {
    const Entry<KW> p = ld_part(h, lane);
    return h.sorted ? p : sort32(p, lane);
}
template <int KW> __device__ __forceinline__ uint32_t least_f(const Entry<KW>& e) {
    return __reduce_min_sync(kFull, prio_f(e.prio));
}
template <int KW> __device__ __forceinline__ void st_part(const WarpHeap<KW>& h, int lane, const Entry<KW>& e) {
    st_stage<false>(h.snodes + lane, e);
}
template <int KW>
__device__ __forceinline__ Entry<KW> ld_node(const WarpHeap<KW>& h, uint32_t idx, int lane) {
    if (idx < h.sn) return ld_stage<false>(h.snodes + (idx + 1) * 32 + lane);
    return ld_entry(h.nodes + (size_t)idx * 32 + lane);
}
// The root without its popped entries, moved to the front.
template <int KW> __device__ __forceinline__ Entry<KW> ld_root(const WarpHeap<KW>& h, int lane) {
    return (uint32_t)lane + h.ro < 32 ? ld_stage<false>(h.snodes + 32 + h.ro + lane) : inf_entry<KW>();
}
template <int KW>
__device__ __forceinline__ void st_node(const WarpHeap<KW>& h, uint32_t idx, int lane, const Entry<KW>& e) {
    if (idx < h.sn) st_stage<false>(h.snodes + (idx + 1) * 32 + lane, e);
    else st_entry(h.nodes + (size_t)idx * 32 + lane, e);
}
// Priority of the largest entry of node idx (one read, broadcast to the warp).
template <int KW> __device__ __forceinline__ uint64_t node_max(const WarpHeap<KW>& h, uint32_t idx) {
    if (idx < h.sn) return *reinterpret_cast<const volatile uint64_t*>(&h.snodes[(idx + 1) * 32 + 31].prio);
    return __ldcg(reinterpret_cast<const unsigned long long*>(&h.nodes[(size_t)idx * 32 + 31].prio));
}

// Starts bringing global node idx (each lane its own entry) into L2, so a
// dependent load of it later waits for L2 instead of DRAM.
template <int KW> __device__ __forceinline__ void prefetch_node(const WarpHeap<KW>& h, uint32_t idx, int lane) {
    if (idx >= h.sn && idx < h.N) {
        const Entry<KW>* a = h.nodes + (size_t)idx * 32 + lane;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
    }
}

template <int KW> __device__ __forceinline__ void heap_init(WarpHeap<KW>& h) {
    h.N = 0;
    h.pc = 0;
    h.pf = kInf;
    h.ro = 0;
    h.max_n = 0;
    h.sorted = true;
}

// `hdr`: the heap's saved {N, pc | ro << 8}.
template <bool FEW, int KW> __device__ __forceinline__ void heap_restore(WarpHeap<KW>& h, const uint32_t* hdr, int lane) {
    h.N = uniform(__ldcg(hdr));
    h.pc = uniform(__ldcg(hdr + 1));
    h.ro = FEW ? h.pc >> 8 : 0;
    h.pc &= 0xffu;
    h.max_n = h.N;
    const Entry<KW> part = (uint32_t)lane < h.pc ? ld_entry(h.nodes + (size_t)h.cap * 32 + lane) : inf_entry<KW>();
    st_part(h, lane, part);
    h.pf = least_f(part);
    h.sorted = false;
    for (uint32_t i = 0; i < h.N && i < h.sn; ++i) st_node(h, i, lane, ld_entry(h.nodes + (size_t)i * 32 + lane));
    __syncwarp();
}

template <int KW> __device__ __forceinline__ void heap_save(const WarpHeap<KW>& h, uint32_t* hdr, int lane) {
    __syncwarp();
    for (uint32_t i = 0; i < h.N && i < h.sn; ++i) st_entry(h.nodes + (size_t)i * 32 + lane, ld_node(h, i, lane));
    st_entry(h.nodes + (size_t)h.cap * 32 + lane, ld_part(h, lane));
    if (lane == 0) {
        __stcg(hdr, h.N);
        __stcg(hdr + 1, h.pc | h.ro << 8);
    }
}

// Least f of the heap (kInf when it is empty; the warp calls it after the
// last change is visible to every lane).
template <int KW> __device__ __forceinline__ uint32_t heap_minf(const WarpHeap<KW>& h) {
    const uint32_t r = h.N ? prio_f(*reinterpret_cast<const volatile uint64_t*>(&h.snodes[32 + h.ro].prio)) : kInf;
    return r < h.pf ? r : h.pf;
}

// Restores the node order from the root (new content `cur`, not stored yet) down.
template <int KW> __device__ void heap_sift_down(WarpHeap<KW>& h, Entry<KW> cur, int lane) {
    uint32_t idx = 0;
    for (;;) {
        uint32_t l = 2 * idx + 1, r = l + 1;
        if (l >= h.N) break;
        Entry<KW> L = ld_node(h, l, lane);
        // The next level is a child of l or r: start all four on their way.
        prefetch_node(h, 2 * l + 1, lane);
        prefetch_node(h, 2 * l + 2, lane);
        prefetch_node(h, 2 * r + 1, lane);
        prefetch_node(h, 2 * r + 2, lane);
        uint64_t cmax = __shfl_sync(kFull, cur.prio, 31);
        uint64_t lmin = __shfl_sync(kFull, L.prio, 0);
        if (r >= h.N) {
            if (uniform_if(cmax > lmin)) {
                Entry<KW> lo, hi;
                merge2(cur, L, lo, hi, lane);
                st_node(h, l, lane, hi);
                cur = lo;
            }
            break;
        }
        Entry<KW> R = ld_node(h, r, lane);
        uint64_t rmin = __shfl_sync(kFull, R.prio, 0);
        if (uniform_if(cmax <= (lmin < rmin ? lmin : rmin))) break;
        uint64_t lmax = __shfl_sync(kFull, L.prio, 31);
        uint64_t rmax = __shfl_sync(kFull, R.prio, 31);
        Entry<KW> A, B;
        merge2(L, R, A, B, lane);
        const bool left = uniform_if(lmax >= rmax);
        const uint32_t big = left ? l : r, small = left ? r : l;
        st_node(h, big, lane, B);  // B.max = max(lmax, rmax): big's subtree stays ordered
        Entry<KW> lo, hi;
        merge2(cur, A, lo, hi, lane);
        st_node(h, idx, lane, lo);
        cur = hi;
        idx = small;
    }
    st_node(h, idx, lane, cur);
    __syncwarp();
}

// Pops of up to this many entries take them off the root's and the buffer's
// front: a count of smaller buffer entries per root lane (two shuffles for
// each entry popped) in place of a merge, and the tree is gone through once per
// root instead of once per pop.  A pop is a chain of shuffles and shared-memory
// loads, bound by their latency.  Wider pops use up a root at once and merge
// it with the buffer.  On 152 blocks, with the shorter sort: 15-puzzles
// (8 popped) 5.20 -> 4.74 ms, grids 1021^2 7.08 -> 6.11 ms, 4096^2 36.6 -> 31.6 ms.
constexpr uint32_t kFewPops = 8;
template <int KW> __device__ void heap_refill(WarpHeap<KW>& h, int lane);

// Pops up to E (1..32) best entries whose priority is below `lim`; lane
// l < return value receives one.
template <bool FEW, int KW>
__device__ uint32_t heap_pop(WarpHeap<KW>& h, uint32_t E, uint64_t lim, Entry<KW>& out, int lane) {
    if (h.N == 0) {
        Entry<KW> part = ld_part(h, lane);
        const uint32_t bm = __ballot_sync(kFull, part.prio < lim);
        uint32_t c = __popc(bm);
        if (c > E) {  // the E best of them
            if (!h.sorted) part = sort32(part, lane);
            h.sorted = true;
            c = E;
        } else if (c && c < h.pc && !h.sorted) {  // all of them, moved to the front
            const uint32_t below = bm & ((1u << lane) - 1u);
            const uint32_t to = (bm >> lane & 1u) ? __popc(below) : c + (uint32_t)lane - __popc(below);
            __syncwarp();
            if ((uint32_t)lane < h.pc) st_stage<false>(h.snodes + to, part);
            __syncwarp();
            part = ld_part(h, lane);
        }
        out = (uint32_t)lane < c ? part : inf_entry<KW>();
        if (c) {
            const Entry<KW> t = shfl_idx(part, (lane + (int)c) & 31);
            const Entry<KW> rest = (uint32_t)lane + c < h.pc ? t : inf_entry<KW>();
            h.pc -= c;
            st_part(h, lane, rest);
            h.pf = least_f(rest);
            __syncwarp();
        }
        return c;
    }
    // The root's entries are above no child's: the least of root and buffer
    // are the heap's, as many of them as the root holds.
    if (FEW && h.N > 1 && 32 - h.ro < E) E = 32 - h.ro;  // (buckets: a wider pop than the last)
    const Entry<KW> part = ld_part_sorted(h, lane);
    const Entry<KW> root = ld_root(h, lane);
    h.sorted = true;  // every way on stores it back in order
    if (FEW && E <= kFewPops) {
        // Take the first kr of the root and the first entries of the buffer:
        // no merge, no way down the tree.
        const uint32_t in_root = __popc(__ballot_sync(kFull, root.prio < lim));
        const uint32_t all = in_root + __popc(__ballot_sync(kFull, part.prio < lim));
        const uint32_t take = E < all ? E : all;
        uint32_t before = 0;  // buffer entries below this lane's root entry
#pragma unroll
        for (int j = 0; j < (int)kFewPops; ++j) before += __shfl_sync(kFull, part.prio, j) < root.prio;
        const uint32_t kr = __popc(__ballot_sync(kFull, (uint32_t)lane < in_root && (uint32_t)lane + before < take));
        const uint32_t kp = take - kr;
        const Entry<KW> from_part = shfl_idx(part, (lane - (int)kr) & 31);
        out = (uint32_t)lane < kr ? root : (uint32_t)lane < take ? from_part : inf_entry<KW>();
        const Entry<KW> t = shfl_idx(part, (lane + (int)kp) & 31);
        const Entry<KW> rest = (uint32_t)lane + kp < h.pc ? t : inf_entry<KW>();
        h.pc -= kp;
        st_part(h, lane, rest);
        h.pf = least_f(rest);
        h.ro += kr;
        __syncwarp();
        if (h.N > 1) {
            if (h.ro + E > 32) heap_refill(h, lane);
        } else if (h.ro == 32) {
            h.N = 0;
            h.ro = 0;
        }
        return take;
    }
    prefetch_node(h, h.N - 1, lane);  // the last node refills the root when the buffer runs short
    Entry<KW> lo, hi;
    merge2(root, part, lo, hi, lane);
    {
        const uint32_t below = __popc(__ballot_sync(kFull, lo.prio < lim));
        if (below < E) E = below;
        if (E == 0) {
            st_part(h, lane, part);
            __syncwarp();
            out = inf_entry<KW>();
            return 0;
        }
    }
    const uint32_t valid = 32 - h.ro + h.pc, rest = valid - E;
    h.ro = 0;
    out = (uint32_t)lane < E ? lo : inf_entry<KW>();
    const int i1 = (int)E + lane, i2 = (int)E + 32 + lane;
    Entry<KW> r1 = pick(lo, hi, i1 & 63);
    Entry<KW> r2 = pick(lo, hi, i2 & 63);
    if ((uint32_t)i1 >= valid) r1 = inf_entry<KW>();
    if ((uint32_t)i2 >= valid) r2 = inf_entry<KW>();
    if (rest >= 32) {
        st_part(h, lane, r2);
        h.pc = rest - 32;
        h.pf = least_f(r2);
        heap_sift_down(h, r1, lane);
    } else if (h.N == 1) {
        h.N = 0;
        st_part(h, lane, r1);
        h.pc = rest;
        h.pf = least_f(r1);
        __syncwarp();
    } else {
        Entry<KW> last = ld_node(h, h.N - 1, lane);
        h.N -= 1;
        Entry<KW> lo2, hi2;
        merge2(last, r1, lo2, hi2, lane);
        st_part(h, lane, hi2);
        h.pc = rest;
        h.pf = least_f(hi2);
        heap_sift_down(h, lo2, lane);
    }
    return E;
}

// Adds a full node top-down along the path to the new leaf: every node on the
// path keeps the 32 smallest of itself and the carried node.
template <int KW> __device__ bool heap_insert_node(WarpHeap<KW>& h, Entry<KW> F, int lane) {
    if (h.N >= h.cap) return false;
    if (h.N) {
        const uint32_t p = h.N + 1;
        const int levels = 31 - __clz(p);
        // The path is fixed by the new leaf's index: fetch the maximum of
        // every node on it in one parallel load (lane j <- depth j), so only
        // the nodes that need a merge cost a dependent access.
        uint64_t pmax = kInfPrio;
        if (lane < levels) pmax = node_max(h, (p >> (levels - lane)) - 1);
        for (int b = levels - 1; b >= 1; --b) prefetch_node(h, (p >> b) - 1, lane);  // the nodes themselves
        for (int b = levels; b >= 1; --b) {
            const uint32_t idx = (p >> b) - 1;
            uint64_t fmin = __shfl_sync(kFull, F.prio, 0);
            if (uniform_if(fmin < __shfl_sync(kFull, pmax, levels - b))) {
                Entry<KW> M = ld_node(h, idx, lane);
                // Popped entries of the root stay least, so that a full node
                // goes on.
                if (idx == 0 && (uint32_t)lane < h.ro) M.prio = 0;
                Entry<KW> lo, hi;
                merge2(M, F, lo, hi, lane);
                st_node(h, idx, lane, lo);
                F = hi;
            }
        }
    }
    st_node(h, h.N, lane, F);
    __syncwarp();
    h.N += 1;
    if (h.N > h.max_n) h.max_n = h.N;
    return true;
}

// Pushes the entries of the lanes in `mask` (the other lanes hold padding
// entries).
template <int KW>
__device__ bool heap_push(WarpHeap<KW>& h, Entry<KW> x, uint32_t mask, int lane) {
    const uint32_t tot = h.pc + __popc(mask);
    if (tot < 32) {
        if (mask >> lane & 1u) st_stage<false>(h.snodes + h.pc + __popc(mask & ((1u << lane) - 1u)), x);
        const uint32_t f = least_f(x);
        h.pf = f < h.pf ? f : h.pf;
        h.pc = tot;
        h.sorted = false;
        __syncwarp();
        return true;
    }
    x = sort32(x, lane);
    Entry<KW> lo, hi;
    merge2(ld_part_sorted(h, lane), x, lo, hi, lane);
    // The largest 32 form a new node; the smallest stay in the partial buffer,
    // where the next pop sees them first.
    const uint32_t off = tot - 32;
    Entry<KW> node = pick(lo, hi, (int)off + lane);
    const Entry<KW> rest = (uint32_t)lane < off ? lo : inf_entry<KW>();
    st_part(h, lane, rest);
    h.pc = off;
    h.pf = least_f(rest);
    h.sorted = true;
    return heap_insert_node(h, node, lane);
}

// Fills the root again: what it has left and the tree's last node (there is
// one below it) give the new root content and as many entries for the buffer.
template <int KW> __device__ void heap_refill(WarpHeap<KW>& h, int lane) {
    const uint32_t left = 32 - h.ro;
    const Entry<KW> last = ld_node(h, h.N - 1, lane);
    Entry<KW> lo, hi;
    merge2(last, ld_root(h, lane), lo, hi, lane);
    h.N -= 1;
    h.ro = 0;
    heap_sift_down(h, lo, lane);
    if (left) heap_push(h, hi, (1u << left) - 1u, lane);
}

// ---------------------------------------------------------------------------
// Bucket front of a warp's open list.
//
// Entries whose f lies in the window [lo, lo + 32) go to one of 32 buckets
// (bucket = f mod 32; lane b keeps bucket b's state), each a stack of 32-entry
// pages in global memory.  Every other entry -- and every entry once the
// pages run out -- goes to the warp-heap.  A pop takes from whichever holds
// the lower f; the buckets are exact in f and last-in first-out within one f,
// which favours the deepest entries among equal f as the heap's g tie-break
// does, so the open list's minimum stays exact.  A push is a few shuffles and
// stores, a pop one coalesced page load, where the heap merges 32-entry nodes
// level by level (two 64-entry merges of ~44 shuffles each per level).
// Pages come from a cache of free page ids held in registers (lane l < fc
// holds one), then from never-used pages (bump), then from a stack in global
// memory of pages freed while the cache was full.
// ---------------------------------------------------------------------------
constexpr uint32_t kNoPage = 0xffffffffu;

template <int KW> struct Buckets {
    Entry<KW>* pages;  // P pages of 32 entries (global memory)
    uint32_t* link;    // the page below each page in its bucket's stack (global memory)
    uint32_t* upd;     // per-bucket scratch of a push (64 words, shared memory)
    uint32_t fs_off;   // link + fs_off: pages freed while the register cache was full
    uint32_t P;        // pages (0 = buckets off)
    uint32_t bump;     // pages >= bump were never used (warp-uniform)
    uint32_t nfs;      // entries on fstack (warp-uniform)
    uint32_t fc;       // free page ids cached in registers (warp-uniform)
    uint32_t cache;    // lane l < fc: a free page id
    uint32_t lo;       // window start (warp-uniform)
    uint32_t head;     // lane b: top page of bucket b (kNoPage = empty)
    uint32_t hcnt;     // lane b: entries in that page (the pages below are full)
};

template <int KW> __device__ __forceinline__ void bq_init(Buckets<KW>& q, int) {
    q.bump = 0;
    q.nfs = 0;
    q.fc = 0;
    q.cache = kNoPage;
    q.lo = 0;
    q.head = kNoPage;
    q.hcnt = 0;
}

// f of the lowest non-empty bucket, or kInf.
template <int KW> __device__ __forceinline__ uint32_t bq_min_f(const Buckets<KW>& q) {
    const uint32_t mask = __ballot_sync(kFull, q.head != kNoPage);
    if (!mask) return kInf;
    const uint32_t s = q.lo & 31u;
    const uint32_t rot = s ? (mask >> s) | (mask << (32 - s)) : mask;
    return q.lo + (uint32_t)(__ffs(rot) - 1);
}

// Least f over a warp's open list (kInf when it is empty).
template <int KW> __device__ __forceinline__ uint32_t open_minf(const WarpHeap<KW>& h, const Buckets<KW>& q) {
    const uint32_t hf = heap_minf(h);
    if (!q.P) return hf;
    const uint32_t bf = bq_min_f(q);
    return hf < bf ? hf : bf;
}

// Returns a freed page to the cache, or to the global stack when it is full.
template <int KW> __device__ __forceinline__ void bq_free(Buckets<KW>& q, uint32_t page, int lane) {
    if (q.fc < 32) {
        if ((uint32_t)lane == q.fc) q.cache = page;
        q.fc += 1;
    } else {
        if (lane == 0) __stcg(q.link + q.fs_off + q.nfs, page);
        q.nfs += 1;
    }
}

// Adds x (lanes < m valid; lanes >= m hold inf entries).  Returns false when
// the heap is full (entries were lost).
template <int KW>
__device__ bool open_push(WarpHeap<KW>& h, Buckets<KW>& q, Entry<KW> x, uint32_t m, int lane) {
    if (m == 0) return true;
    const bool valid = (uint32_t)lane < m;
    bool placed = false;
    if (q.P) {
        const uint32_t f = prio_f(x.prio);
        if (!__any_sync(kFull, q.head != kNoPage))  // empty: the window starts at the least f
            q.lo = __reduce_min_sync(kFull, valid ? f : kInf);
        const bool inwin = valid && f >= q.lo && f - q.lo < 32u;
        const uint32_t b = f & 31u;
        const uint32_t lt = (1u << lane) - 1u;
        const uint32_t grp = __match_any_sync(kFull, inwin ? b : 32u + (uint32_t)lane);
        const uint32_t r = __popc(grp & lt), n = __popc(grp);
        const uint32_t hd = __shfl_sync(kFull, q.head, (int)b), hc = __shfl_sync(kFull, q.hcnt, (int)b);
        const bool leader = inwin && r == 0;
        const uint32_t room = hd == kNoPage ? 0u : 32u - hc;
        const bool need = inwin && n > room;
        // One new page per overflowing bucket: cached ids first, then
        // never-used pages, then the global stack.
        const uint32_t nmask = __ballot_sync(kFull, leader && need);
        const uint32_t want = __popc(nmask);
        const uint32_t fresh = q.P - q.bump, avail = q.fc + fresh + q.nfs;
        uint32_t page = kNoPage;
        {
            const uint32_t idx = __popc(nmask & lt);
            const uint32_t cached = __shfl_sync(kFull, q.cache, (int)((q.fc - 1 - idx) & 31u));
            if (leader && need && idx < avail) {
                if (idx < q.fc) page = cached;
                else if (idx < q.fc + fresh) page = q.bump + (idx - q.fc);
                else page = __ldcg(q.link + q.fs_off + q.nfs - 1 - (idx - q.fc - fresh));
            }
        }
        {
            uint32_t take = want < avail ? want : avail;
            const uint32_t from_cache = take < q.fc ? take : q.fc;
            q.fc -= from_cache;
            take -= from_cache;
            const uint32_t from_bump = take < fresh ? take : fresh;
            q.bump += from_bump;
            q.nfs -= take - from_bump;
        }
        page = __shfl_sync(kFull, page, __ffs(grp) - 1);
        if (inwin) {
            if (r < room) {
                st_entry(q.pages + (size_t)hd * 32 + hc + r, x);
                placed = true;
            } else if (page != kNoPage) {
                st_entry(q.pages + (size_t)page * 32 + (r - room), x);
                placed = true;
            }
        }
        if (leader) {
            uint32_t nh = hd, nc = hc;
            if (n <= room) {
                nc = hc + n;
            } else {
                if (hd != kNoPage) nc = 32;
                if (page != kNoPage) {
                    __stcg(q.link + page, hd);
                    nh = page;
                    nc = n - room;
                }
            }
            q.upd[2 * b] = nh;
            q.upd[2 * b + 1] = nc;
        }
        const uint32_t umask = __reduce_or_sync(kFull, leader ? (1u << b) : 0u);
        __syncwarp();
        if ((umask >> lane) & 1u) {
            q.head = q.upd[2 * lane];
            q.hcnt = q.upd[2 * lane + 1];
        }
        __syncwarp();
    }
    const bool rest = valid && !placed;
    const uint32_t rm = __ballot_sync(kFull, rest);
    if (!rm) return true;
    return heap_push(h, rest ? x : inf_entry<KW>(), rm, lane);
}

// Pops up to E (1..32) entries with priority below `lim` (a multiple of 2^32
// or kInfPrio); lane l < return value receives one.
template <bool FEW, int KW>
__device__ uint32_t open_pop(WarpHeap<KW>& h, Buckets<KW>& q, uint32_t E, uint64_t lim, Entry<KW>& out,
                             int lane) {
    out = inf_entry<KW>();
    uint32_t taken = 0;
    for (int round = 0; round < 4 && taken < E; ++round) {
        const uint32_t bf = q.P ? bq_min_f(q) : kInf, hf = uniform(heap_minf(h));
        const uint32_t mf = hf < bf ? hf : bf;
        if (mf == kInf || ((uint64_t)mf << 32) >= lim) break;
        const uint64_t bp = bf == kInf ? kInfPrio : ((uint64_t)bf << 32);
        const uint32_t i = (uint32_t)lane - taken;  // this lane's index among the new ones
        if (hf < bf) {  // the heap holds lower f: take its entries below the buckets' f
            Entry<KW> e;
            const uint32_t c = heap_pop<FEW>(h, E - taken, bp < lim ? bp : lim, e, lane);
            const Entry<KW> sh = shfl_idx(e, (lane - (int)taken) & 31);
            if ((uint32_t)lane >= taken && i < c) out = sh;
            taken += c;
            if (c == 0 || !q.P) break;
        } else {
            const int bl = (int)(bf & 31u);
            const uint32_t hd = __shfl_sync(kFull, q.head, bl), hc = uniform(__shfl_sync(kFull, q.hcnt, bl));
            const uint32_t k = E - taken < hc ? E - taken : hc;
            // The page's entries and, when it empties, its link load together.
            const uint32_t nx = hc == k ? __ldcg(q.link + hd) : kNoPage;
            if ((uint32_t)lane >= taken && i < k) out = ld_entry(q.pages + (size_t)hd * 32 + (hc - k + i));
            if (hc == k) {  // the page is empty: the next one comes up, this one is free
                if (lane == bl) {
                    q.head = nx;
                    q.hcnt = nx == kNoPage ? 0u : 32u;
                }
                bq_free(q, hd, lane);
            } else if (lane == bl) {
                q.hcnt = hc - k;
            }
            taken += k;
        }
    }
    const uint32_t bf = q.P ? bq_min_f(q) : kInf;
    if (bf != kInf) q.lo = bf;  // the window follows the lowest non-empty bucket
    return taken;
}

// The bucket state of a suspended search stays beside its pages: lane l
// saves its bucket's head page and count and its cached free page; lane 0
// the window start, the never-used and free-stack counts and the cache size.
template <int KW> __device__ __forceinline__ void bq_save(const Buckets<KW>& q, uint32_t* state, int lane) {
    if (!q.P) return;
    __stcg(state + lane, q.head);
    __stcg(state + 32 + lane, q.hcnt);
    __stcg(state + 64 + lane, q.cache);
    if (lane == 0) {
        __stcg(state + 96, q.lo);
        __stcg(state + 97, q.bump);
        __stcg(state + 98, q.nfs);
        __stcg(state + 99, q.fc);
    }
}
template <int KW> __device__ __forceinline__ void bq_restore(Buckets<KW>& q, const uint32_t* state, int lane) {
    if (!q.P) return;
    q.head = __ldcg(state + lane);
    q.hcnt = __ldcg(state + 32 + lane);
    q.cache = __ldcg(state + 64 + lane);
    q.lo = uniform(__ldcg(state + 96));
    q.bump = uniform(__ldcg(state + 97));
    q.nfs = uniform(__ldcg(state + 98));
    q.fc = uniform(__ldcg(state + 99));
}

// ---------------------------------------------------------------------------
// Duplicate-detection tables.  insert-or-min returns the previous value word;
// the caller keeps a successor iff its g is strictly below the old g.  This is
// the reference's NEW -> INSERTED / UPDATED / REJECTED classification
// (fancy_hashmap.h:32-81, 155-167) as one atomic per successor.
// ---------------------------------------------------------------------------

// Claims come in two steps: claim_begin issues the home slot's atomic,
// claim_end resolves it -- probing on when the slot holds another key,
// lowering the value of a known key -- and returns -1 full, 0 found or
// 1 claimed, with `old` the value word before this update.

__device__ __forceinline__ void cas128(unsigned long long* addr, uint64_t c0, uint64_t c1,
                                       uint64_t n0, uint64_t n1, uint64_t& o0, uint64_t& o1) {
    asm volatile(
        "{\n\t.reg .b128 cmp, swp, dst;\n\t"
        "mov.b128 cmp, {%2, %3};\n\t"
        "mov.b128 swp, {%4, %5};\n\t"
        "atom.global.cas.b128 dst, [%6], cmp, swp;\n\t"
        "mov.b128 {%0, %1}, dst;\n\t}"
        : "=l"(o0), "=l"(o1)
        : "l"(c0), "l"(c1), "l"(n0), "l"(n1), "l"(addr)
        : "memory");
}

// 64-bit keys: slot = {key, value}, 16 bytes; linear probing.  Every atomic
// on a slot is one 16-byte compare-and-swap of the pair: a new key is claimed
// with its value in one round trip, a known key costs none more unless its
// value drops.
struct HashTab64 {
    unsigned long long* s;
    uint64_t mask;
    uint32_t max_probe;
};

// Lowers the value of a found key to `val` unless it is already <= val;
// `seen` is the value the claim read.  Returns the value before the update.
// Values only fall, so every failed exchange is followed by a strictly lower
// value; the retry bound is far beyond the number of concurrent updaters.
__device__ __forceinline__ uint64_t tab_min_at(const HashTab64& t, uint32_t slot, uint64_t key, uint64_t val,
                                               uint64_t seen) {
    uint64_t cur = seen;
    for (uint32_t r = 0; cur > val && r < 4096; ++r) {
        uint64_t o0, o1;
        cas128(t.s + slot, key, cur, key, val, o0, o1);
        if (o1 == cur) break;
        cur = o1;
    }
    return cur;
}
__device__ __forceinline__ void tab_claim_begin(const HashTab64& t, uint64_t key, uint64_t val, uint32_t& slot,
                                                uint64_t& o0, uint64_t& o1) {
    slot = 2 * (uint32_t)(mix64(key) & t.mask);
    cas128(t.s + slot, kEmpty, kEmpty, key, val, o0, o1);
}
// (o0, o1): what claim_begin's exchange returned; o1 becomes the value before.
__device__ __forceinline__ int tab_claim_end(const HashTab64& t, uint64_t key, uint64_t val, uint32_t& slot,
                                             uint64_t o0, uint64_t& o1) {
    for (uint32_t p = 1;; ++p) {
        if (o0 == kEmpty && o1 == kEmpty) return 1;
        if (o0 == key) {
            if (o1 > val) o1 = tab_min_at(t, slot, key, val, o1);
            return 0;
        }
        if (p >= t.max_probe) return -1;
        slot = 2 * ((slot / 2 + 1) & (uint32_t)t.mask);
        cas128(t.s + slot, kEmpty, kEmpty, key, val, o0, o1);
    }
}
// Returns 1 when the key was newly claimed, 0 when found, -1 when full.
__device__ __forceinline__ int tab_insert(const HashTab64& t, uint64_t key, uint64_t val, uint64_t& old,
                                          uint32_t& slot) {
    uint64_t o0;
    tab_claim_begin(t, key, val, slot, o0, old);
    return tab_claim_end(t, key, val, slot, o0, old);
}

// Issues the home-slot load of a lookup (key and value in one 16-byte load).
__device__ __forceinline__ void tab_look_begin(const HashTab64& t, uint64_t key, uint64_t& k, uint64_t& v) {
    const uint64_t i = mix64(key) & t.mask;
    const ulonglong2 kv = __ldcg(reinterpret_cast<const ulonglong2*>(t.s + 2 * i));
    k = kv.x;
    v = kv.y;
}

__device__ __forceinline__ uint64_t tab_get(const HashTab64& t, uint64_t key) {
    uint64_t i = mix64(key) & t.mask;
    for (uint32_t p = 0; p < t.max_probe; ++p) {
        // Key and value in one 16-byte load (they are written together).
        const ulonglong2 kv = __ldcg(reinterpret_cast<const ulonglong2*>(t.s + 2 * i));
        if (kv.x == key) return kv.y;
        if (kv.x == kEmpty) return kEmpty;
        i = (i + 1) & t.mask;
    }
    return kEmpty;
}

// 128-bit keys: slot = {k0, k1, value, pad}, 32 bytes (one sector).  The key
// is claimed with a 16-byte compare-and-swap; reads of the key pair also go
// through the 16-byte atomic so a half-written pair is never observed.
struct HashTab128 {
    unsigned long long* s;
    uint64_t mask;
    uint32_t max_probe;
};

__device__ __forceinline__ uint64_t hash128(uint64_t k0, uint64_t k1) {
    return mix64(k0 ^ mix64(k1 + 0x9e3779b97f4a7c15ull));
}

__device__ __forceinline__ void tab_claim_begin(const HashTab128& t, uint64_t k0, uint64_t k1, uint32_t& slot,
                                                uint64_t& o0, uint64_t& o1) {
    slot = 4 * (uint32_t)(hash128(k0, k1) & t.mask);
    cas128(t.s + slot, kEmpty, kEmpty, k0, k1, o0, o1);
}
// (o0, o1): the key words claim_begin's exchange returned; o1 becomes the
// value before.  The value word beside the key is lowered with atomicMin.
__device__ __forceinline__ int tab_claim_end(const HashTab128& t, uint64_t k0, uint64_t k1, uint64_t val,
                                             uint32_t& slot, uint64_t o0, uint64_t& o1) {
    for (uint32_t p = 1;; ++p) {
        const int claimed = (o0 == kEmpty && o1 == kEmpty);
        if (claimed || (o0 == k0 && o1 == k1)) {
            o1 = atomicMin(t.s + slot + 2, (unsigned long long)val);
            return claimed;
        }
        if (p >= t.max_probe) return -1;
        slot = 4 * ((slot / 4 + 1) & (uint32_t)t.mask);
        cas128(t.s + slot, kEmpty, kEmpty, k0, k1, o0, o1);
    }
}
__device__ __forceinline__ int tab_insert(const HashTab128& t, uint64_t k0, uint64_t k1,
                                          uint64_t val, uint64_t& old, uint32_t& slot) {
    uint64_t o0;
    tab_claim_begin(t, k0, k1, slot, o0, old);
    return tab_claim_end(t, k0, k1, val, slot, o0, old);
}

__device__ __forceinline__ uint64_t tab_get(const HashTab128& t, uint64_t k0, uint64_t k1) {
    uint64_t i = hash128(k0, k1) & t.mask;
    for (uint32_t p = 0; p < t.max_probe; ++p) {
        unsigned long long* ks = t.s + 4 * i;
        uint64_t o0, o1;
        cas128(ks, kEmpty, kEmpty, kEmpty, kEmpty, o0, o1);  // atomic 16-byte read
        if (o0 == k0 && o1 == k1) return __ldcg(ks + 2);
        if (o0 == kEmpty && o1 == kEmpty) return kEmpty;
        i = (i + 1) & t.mask;
    }
    return kEmpty;
}

// Issues the home slot's reads of a lookup: the key pair (one 16-byte atomic)
// and the value word.
__device__ __forceinline__ void tab_look_begin(const HashTab128& t, uint64_t k0, uint64_t k1, uint64_t& o0,
                                               uint64_t& o1, uint64_t& v) {
    unsigned long long* ks = t.s + 4 * (hash128(k0, k1) & t.mask);
    cas128(ks, kEmpty, kEmpty, kEmpty, kEmpty, o0, o1);
    v = __ldcg(ks + 2);
}

// Dense table for grids: the cell index is the slot (a perfect hash).
struct DenseTab {
    unsigned long long* v;
};

}  // namespace gastar
