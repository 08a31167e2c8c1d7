// Every thread of a launch as a fiber on one host thread.  A warp operation
// ends when all 32 lanes have come to the same one; lanes at different ones, or
// past the last, end the program with an error.  Warps run in a random order,
// blocks stall for random times, and a thread gives way at each access by which
// blocks synchronise.
#pragma once

#include "common.h"

#define __shared__

namespace host {
enum Op : int { SHFL, XOR, UP, BALLOT, MIN, MAX, ADD, OR, MATCH, SYNC };
enum Exit : int { LANES_APART = 3, STUCK = 4, BAD_ADDRESS = 5 };
struct Dim {
    uint32_t x;
};
Dim thread_index(), block_index(), block_size();
uint64_t warp_op(Op op, uint64_t v, uint64_t aux);
void block_barrier();
void cluster_barrier();
void give_way();
const void* in_block(const void* p, uint32_t rank);  // the same place of another block of the cluster
char* block_memory(int which);                       // 0: dynamic, 1: static, 2: the domain's context

// Runs `kernel` on blocks x threads; false after `rounds` rounds without an end.
bool launch(uint32_t blocks, uint32_t threads, uint32_t cluster, size_t dynamic, uint64_t seed, uint64_t rounds,
            std::function<void()> kernel);

inline uint64_t globaltimer() {
    static uint64_t t = 0;
    return t += 100;
}
inline void cas128(unsigned long long* a, uint64_t c0, uint64_t c1, uint64_t n0, uint64_t n1, uint64_t& o0,
                   uint64_t& o1) {
    o0 = a[0];
    o1 = a[1];
    if (o0 == c0 && o1 == c1) {
        a[0] = n0;
        a[1] = n1;
    }
}
template <class T> T load(const T* p) {
    give_way();
    return *(const volatile T*)p;
}
template <class T> void store(T* p, T v) {
    give_way();
    *p = v;
}
template <class T> void add(T* p, T v) {
    give_way();
    *p += v;
}
inline void fence() { give_way(); }
inline uint4 load_cluster(const void* p, uint32_t rank) { return *(const uint4*)in_block(p, rank); }
template <class T> T& block_shared() { return *(T*)block_memory(1); }
template <class T> T& block_context() { return *(T*)block_memory(2); }
inline uint4* block_dynamic() { return (uint4*)block_memory(0); }

template <class T> uint64_t bits(T v) {
    uint64_t r = 0;
    std::memcpy(&r, &v, sizeof(T));
    return r;
}
template <class T> T value(uint64_t r) {
    T v;
    std::memcpy(&v, &r, sizeof(T));
    return v;
}
}  // namespace host

#define threadIdx (host::thread_index())
#define blockIdx (host::block_index())
#define blockDim (host::block_size())

template <class T> T __shfl_sync(unsigned, T v, int s) {
    return host::value<T>(host::warp_op(host::SHFL, host::bits(v), (uint64_t)(s & 31)));
}
template <class T> T __shfl_xor_sync(unsigned, T v, int s) {
    return host::value<T>(host::warp_op(host::XOR, host::bits(v), (uint64_t)s));
}
template <class T> T __shfl_up_sync(unsigned, T v, int s) {
    return host::value<T>(host::warp_op(host::UP, host::bits(v), (uint64_t)s));
}
inline uint32_t __ballot_sync(unsigned, bool p) { return (uint32_t)host::warp_op(host::BALLOT, p, 0); }
inline bool __any_sync(unsigned, bool p) { return host::warp_op(host::BALLOT, p, 0) != 0; }
inline bool __all_sync(unsigned, bool p) { return host::warp_op(host::BALLOT, p, 0) == 0xffffffffu; }
inline uint32_t __reduce_min_sync(unsigned, uint32_t v) { return (uint32_t)host::warp_op(host::MIN, v, 0); }
inline uint32_t __reduce_max_sync(unsigned, uint32_t v) { return (uint32_t)host::warp_op(host::MAX, v, 0); }
inline uint32_t __reduce_add_sync(unsigned, uint32_t v) { return (uint32_t)host::warp_op(host::ADD, v, 0); }
inline uint32_t __reduce_or_sync(unsigned, uint32_t v) { return (uint32_t)host::warp_op(host::OR, v, 0); }
inline uint32_t __match_any_sync(unsigned, uint32_t v) { return (uint32_t)host::warp_op(host::MATCH, v, 0); }
inline void __syncwarp() { host::warp_op(host::SYNC, 0, 0); }
inline void __syncthreads() { host::block_barrier(); }
inline void __nanosleep(unsigned) { host::give_way(); }
template <class T> T __ldcg(const T* p) { return *p; }
template <class T> T __ldg(const T* p) { return *p; }
template <class T, class U> void __stcg(T* p, U v) { *p = (T)v; }
inline void __stcg(uint4* p, uint4 v) { *p = v; }
template <class T, class U> T atomicAdd(T* p, U v) {
    const T o = *p;
    *p = o + (T)v;
    return o;
}
template <class T, class U> T atomicMin(T* p, U v) {
    const T o = *p;
    if ((T)v < o) *p = (T)v;
    return o;
}
template <class T, class U> T atomicMax(T* p, U v) {
    const T o = *p;
    if ((T)v > o) *p = (T)v;
    return o;
}
template <class T, class U> T atomicExch(T* p, U v) {
    const T o = *p;
    *p = (T)v;
    return o;
}
template <class T, class U, class V> T atomicCAS(T* p, U c, V v) {
    const T o = *p;
    if (o == (T)c) *p = (T)v;
    return o;
}
