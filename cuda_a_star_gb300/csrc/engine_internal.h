// Internal host-side declarations shared by the engine's translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/gastar.h"
#include "engine_types.h"
#include "team_shape.h"

namespace gastar {

struct DevBuf {
    void* p = nullptr;
    size_t n = 0;
    bool fresh = false;         // set when ensure() reallocated (contents undefined)
    bool pooled = false;        // from a memory pool (BatchMemory)
    bool ensure(size_t bytes);  // grows (contents are not kept)
    void release();
};

// Device memory for batches that a context's later batches use again: mapping
// and unmapping a batch's partitions (11 GB for 512 8-puzzles: 1.3 and 4.9 ms)
// takes longer than searching them (1.9 ms).  What a destroyed batch gives back
// stays in a memory pool of the driver, at most kKeepMax bytes unused, which hands
// it out in exact sizes and takes it back by itself for any cudaMalloc of the
// process that would fail, whoever calls it (20 ms for 8 GB).  Growing a pool
// takes longer than cudaMalloc (0.8 against 0.1 ms per GB, and 0.4 to free), so
// the first batch of a context, and buffers above kKeepMax, go without it.
class BatchMemory {
public:
    static constexpr size_t kKeepMax = (size_t)16 << 30;
    // Allocates `bytes` into `b` (empty) for work on `st`, which is idle.
    bool take(DevBuf& b, size_t bytes, cudaStream_t st);
    // Releases `b`; the work that used it is done.
    void give(DevBuf& b, cudaStream_t st);
    // Whether a batch may take `bytes`, and `beside` more of the device where it
    // is not kept here: what other contexts of the process keep unused counts as
    // free, and is free afterwards where it was needed.
    bool room(size_t bytes, size_t beside);
    // Gives what is kept unused back to the device.
    void trim();
    void close();

private:
    std::mutex mu_;
    cudaMemPool_t pool_ = nullptr;
    bool again_ = false;  // a batch has been destroyed
    uint64_t live_ = 0;   // bytes of the pool that batches hold
};

void set_error(const std::string& s);
bool cuda_ok(cudaError_t e, const char* what);

// The search kernel's instantiations (search_*.cu).
const void* search_kernel_sliding3();
const void* search_kernel_sliding4();
const void* search_kernel_sliding5();
const void* search_kernel_grid();
const void* search_kernel_all();
const void* search_kernel_all16();
const void* search_kernel_for(uint32_t kinds, uint32_t threads);
int launch_search(struct ::gastar_ctx* c, uint32_t kinds, const LaunchParams& P, uint32_t blocks,
                  uint32_t threads, size_t smem, cudaStream_t st);
// Rebuilds the paths of finished instances into `arena` (see path_kernel):
// with `offs` (device, n + 1 prefix offsets) each instance writes its own
// slice in one walk.
int launch_paths(const InstDesc* d_insts, uint32_t n, unsigned long long* arena,
                 unsigned long long arena_words, unsigned long long* used, cudaStream_t st,
                 const unsigned long long* offs = nullptr);
// Largest count of shared-memory heap nodes per warp (>= kHeapSmemNodes) that
// keeps `blocks_per_sm` blocks of this shape resident; *smem = the block's
// dynamic shared memory with it.
uint32_t fit_heap_snodes(gastar_ctx* c, uint32_t kinds, uint32_t warps, uint32_t ew, bool multi, uint32_t threads,
                         int blocks_per_sm, size_t* smem, bool buckets = false);
int occupancy_blocks(struct ::gastar_ctx* c, uint32_t kinds, uint32_t threads, size_t smem);
// Clusters of `size` blocks of this shape that are resident at once (0: the
// size or the shape does not fit).
int occupancy_clusters(uint32_t kinds, uint32_t threads, size_t smem, uint32_t size);
// Whether heavy teams of `size` blocks run as clusters: sizes that every GPC
// can be cut into, up to the largest cluster.
inline bool cluster_team_size(uint32_t size) { return size == 2 || size == 4 || size == 8 || size == 16; }
int device_min_weight(struct ::gastar_ctx* c, const uint8_t* d_w, uint64_t cells, cudaStream_t st,
                      uint32_t* out);
// Places a grid's weights from the caller's host buffer at d_dst and returns
// its least passable weight (255: none); synchronises `st`, so the caller may
// reuse the buffer afterwards.  By the context's upload_mode: staged (host
// threads and a pinned ring), read in place by one kernel that also reduces
// (where the GPU reads pageable host memory through the host's page tables),
// or a copy, then device_min_weight.
int upload_grid(struct ::gastar_ctx* c, uint8_t* d_dst, const uint8_t* h_src, uint64_t cells, cudaStream_t st,
                uint32_t* minw);
// The staged way (upload.cpp): host threads fill pinned chunks and reduce the
// least weight while the previous chunks are sent.
struct HostStager;
int upload_grid_staged(struct ::gastar_ctx* c, uint8_t* d_dst, const uint8_t* h_src, uint64_t cells,
                       cudaStream_t st, uint32_t* minw);
void destroy_stager(HostStager* s);

struct PlainProblem {
    uint32_t kind, n;
    uint64_t start0, start1, goal0, goal1;
    const uint8_t* d_weights;  // grid (device)
    uint32_t W, H, minw, f0;
};
// One instance on a multi-block team (the plain engine); path_keys receives
// the path goal-first (KW words per state) when not null.
int plain_solve(struct ::gastar_ctx* c, const PlainProblem& pp, const gastar_config* user_cfg,
                std::vector<uint64_t>* path_keys, gastar_result* out);

bool valid_board(uint32_t n, const uint8_t* b);
void pack_board(uint32_t n, const uint8_t* b, uint64_t& lo, uint64_t& hi);
void unpack_board(uint32_t n, uint64_t lo, uint64_t hi, uint8_t* b);
uint32_t sliding_h(uint32_t n, const uint8_t* b, const uint8_t* goal, uint32_t heuristic);
bool sliding_solvable(uint32_t n, const uint8_t* s, const uint8_t* g);
uint32_t grid_h(uint32_t x, uint32_t y, uint32_t tx, uint32_t ty, uint32_t minw, uint32_t heuristic);
uint64_t next_pow2(uint64_t v);
// Least non-zero weight of a grid, 255 if none (vectorised scan).
uint8_t min_passable_weight(const uint8_t* weights, size_t cells);

}  // namespace gastar

struct gastar_ctx {
    int device = 0;
    int sms = 0;
    int coop = 0;
    size_t smem_per_sm = 0;  // shared memory of one SM
    size_t smem_optin = 0;   // largest dynamic shared memory one block may ask for
    size_t mem_total = 0;
    char name[256] = {0};
    cudaStream_t stream = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    gastar::DevBuf table, dense, touched, heaps, hdr, stage, path, misc, weights, buckets;
    // Plain engine: descriptor, control block, team control and counters of
    // one solve in one device block, uploaded from a pinned mirror in one copy.
    gastar::DevBuf launch;
    void* h_launch = nullptr;      // pinned
    uint64_t* h_path = nullptr;    // pinned: the path's first words, read back with the control block
    bool can_read_host = false;    // kernels read pageable host memory through the host's
                                   // page tables (ATS over NVLink-C2C on Grace)
    int upload_mode = 2;           // grid uploads: 0 copy, 1 read in place, 2 staged
    gastar::BatchMemory batch_memory;
    gastar::HostStager* stager = nullptr;  // staged uploads (pinned ring, host threads)
    bool table_dirty = true;       // hash table needs a full clear before the next solve
    uint32_t prev_slot_words = 2;  // slot width of the solve that filled the touched list
    uint64_t launches = 0;         // kernels launched by this context
    gastar::InstCtl* h_ctl = nullptr;  // pinned
};
