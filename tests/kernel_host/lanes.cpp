#include "lanes.h"

#include <ucontext.h>

namespace host {
namespace {

enum State { READY, AT_WARP_OP, AT_BLOCK_BARRIER, AT_CLUSTER_BARRIER, DONE };
constexpr size_t kStack = 128 << 10, kStatic = 32 << 10;

struct Fiber {
    ucontext_t ctx;
    std::unique_ptr<char[]> stack{new char[kStack]};
    uint32_t thread, block;
    State state = READY;
    bool gave_way = false;
    Op op;
    uint64_t val, aux;
};
std::vector<std::unique_ptr<Fiber>> fibers;
Fiber* cur;
ucontext_t scheduler;
uint32_t n_blocks, n_threads, cluster_size;
size_t dynamic_bytes;
std::vector<std::unique_ptr<uint4[]>> memory[3];
std::function<void()> body;

void entry() {
    body();
    cur->state = DONE;
    swapcontext(&cur->ctx, &scheduler);
}
void wait(State s) {
    Fiber* f = cur;
    f->state = s;
    swapcontext(&f->ctx, &scheduler);
}
[[noreturn]] void fail(int code, const char* what) {
    std::printf("%s\n", what);
    std::fflush(stdout);
    std::_Exit(code);
}

uint64_t combine(Op op, const uint64_t* in, const uint64_t* aux, int l) {
    uint64_t r = op == MIN ? ~0ull : 0;
    switch (op) {
        case SHFL: return in[aux[l] & 31];
        case XOR: return in[(l ^ aux[l]) & 31];
        case UP: return l >= (int)aux[l] ? in[l - aux[l]] : in[l];
        case SYNC: return 0;
        default: break;
    }
    for (int j = 0; j < 32; ++j) switch (op) {
            case BALLOT: r |= (uint64_t)(in[j] != 0) << j; break;
            case MIN: r = in[j] < r ? in[j] : r; break;
            case MAX: r = in[j] > r ? in[j] : r; break;
            case ADD: r += in[j]; break;
            case OR: r |= in[j]; break;
            case MATCH: r |= (uint64_t)(in[j] == in[l]) << j; break;
            default: break;
        }
    return r;
}

// Runs a warp until its lanes wait for others; false: nothing moved.
bool run_warp(std::unique_ptr<Fiber>* w) {
    bool moved = false;
    for (int rep = 0; rep < 64; ++rep) {
        bool ran = false, gave = false;
        for (int l = 0; l < 32; ++l)
            if (w[l]->state == READY) {
                cur = w[l].get();
                cur->gave_way = false;
                swapcontext(&scheduler, &cur->ctx);
                ran = moved = true;
                gave |= cur->gave_way;
            }
        int at = 0, ready = 0;
        for (int l = 0; l < 32; ++l) {
            at += w[l]->state == AT_WARP_OP;
            ready += w[l]->state == READY;
        }
        if (at == 32) {
            uint64_t in[32], aux[32];
            for (int l = 0; l < 32; ++l) {
                if (w[l]->op != w[0]->op) fail(LANES_APART, "lanes of a warp at different operations");
                in[l] = w[l]->val;
                aux[l] = w[l]->aux;
            }
            for (int l = 0; l < 32; ++l) {
                w[l]->val = combine(w[0]->op, in, aux, l);
                w[l]->state = READY;
            }
            ran = moved = true;
        } else if (at && !ready) {
            fail(LANES_APART, "lanes of a warp at an operation that the others do not come to");
        }
        if (!ran || gave) break;
    }
    return moved;
}

bool release(uint32_t first, uint32_t n, State s) {
    uint32_t at = 0, done = 0;
    for (uint32_t i = first; i < first + n; ++i) {
        at += fibers[i]->state == s;
        done += fibers[i]->state == DONE;
    }
    if (!at || at + done != n) return false;
    if (done) fail(LANES_APART, "threads at a barrier that others have left for good");
    for (uint32_t i = first; i < first + n; ++i) fibers[i]->state = READY;
    return true;
}

}  // namespace

Dim thread_index() { return {cur->thread}; }
Dim block_index() { return {cur->block}; }
Dim block_size() { return {n_threads}; }
uint64_t warp_op(Op op, uint64_t v, uint64_t aux) {
    cur->op = op;
    cur->val = v;
    cur->aux = aux;
    Fiber* f = cur;
    wait(AT_WARP_OP);
    return f->val;
}
void block_barrier() { wait(AT_BLOCK_BARRIER); }
void cluster_barrier() { wait(cluster_size > 1 ? AT_CLUSTER_BARRIER : AT_BLOCK_BARRIER); }
void give_way() {
    Fiber* f = cur;
    f->gave_way = true;
    swapcontext(&f->ctx, &scheduler);
}
char* block_memory(int which) { return (char*)memory[which][cur->block].get(); }
const void* in_block(const void* p, uint32_t rank) {
    const uint32_t b = cur->block / cluster_size * cluster_size + rank;
    for (int m = 0; m < 3; ++m) {
        const char* base = (const char*)memory[m][cur->block].get();
        const size_t n = m == 0 ? dynamic_bytes : kStatic;
        if ((const char*)p >= base && (const char*)p < base + n)
            return (const char*)memory[m][b].get() + ((const char*)p - base);
    }
    fail(BAD_ADDRESS, "an address outside the block's shared memory");
}

bool launch(uint32_t blocks, uint32_t threads, uint32_t cluster, size_t dynamic, uint64_t seed, uint64_t rounds,
            std::function<void()> kernel) {
    std::mt19937_64 rng(seed);
    body = kernel;
    n_blocks = blocks;
    n_threads = threads;
    cluster_size = cluster ? cluster : 1;
    dynamic_bytes = dynamic;
    fibers.clear();
    for (int m = 0; m < 3; ++m) {
        memory[m].clear();
        const size_t n = (m == 0 ? dynamic : kStatic) / 16 + 4;
        for (uint32_t b = 0; b < blocks; ++b) {
            memory[m].emplace_back(new uint4[n]);
            std::memset((void*)memory[m][b].get(), 0xa5, n * 16);
        }
    }
    for (uint32_t b = 0; b < blocks; ++b)
        for (uint32_t t = 0; t < threads; ++t) {
            fibers.emplace_back(new Fiber);
            Fiber& f = *fibers.back();
            f.thread = t;
            f.block = b;
            getcontext(&f.ctx);
            f.ctx.uc_stack.ss_sp = f.stack.get();
            f.ctx.uc_stack.ss_size = kStack;
            f.ctx.uc_link = &scheduler;
            makecontext(&f.ctx, entry, 0);
        }
    const uint32_t warps = blocks * threads / 32;
    std::vector<uint32_t> order(warps), stall(blocks, 0);
    for (uint32_t i = 0; i < warps; ++i) order[i] = i;
    for (uint64_t r = 0; r < rounds; ++r) {
        bool moved = false, stalled = false, all = true;
        for (uint32_t& s : stall) {
            if (s) --s;
            else if (blocks > 1 && rng() % 64 == 0) s = (uint32_t)(rng() % 200);
        }
        std::shuffle(order.begin(), order.end(), rng);
        for (uint32_t w : order) {
            if (stall[w / (threads / 32)] || (warps > 1 && rng() % 4 == 0)) {
                stalled = true;
                continue;
            }
            moved |= run_warp(&fibers[(size_t)w * 32]);
        }
        for (uint32_t b = 0; b < blocks; ++b) moved |= release(b * threads, threads, AT_BLOCK_BARRIER);
        for (uint32_t c = 0; cluster_size > 1 && c < blocks; c += cluster_size)
            moved |= release(c * threads, cluster_size * threads, AT_CLUSTER_BARRIER);
        for (auto& f : fibers) all &= f->state == DONE;
        if (all) return true;
        if (!moved && !stalled) fail(STUCK, "threads wait for one another");
    }
    return false;
}
}  // namespace host
