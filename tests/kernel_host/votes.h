// Warp operations as opaque calls.  A vote or reduction whose operand the
// compiler knows after inlining does not compile.
#pragma once

#include "common.h"

#define __shared__ static

struct Dim {
    uint32_t x;
};
extern Dim threadIdx, blockIdx, blockDim;

extern "C" {
uint64_t opaque(uint64_t v, int op);
void vote_on_a_constant(void) __attribute__((error("a vote or reduction of a constant")));
}

#define CHECKED(v, op)                                             \
    (__extension__({                                               \
        auto checked_v = (v);                                      \
        if (__builtin_constant_p(checked_v)) vote_on_a_constant(); \
        opaque((uint64_t)checked_v, op);                           \
    }))
#define __ballot_sync(mask, p) ((uint32_t)CHECKED((bool)(p), 1))
#define __any_sync(mask, p) (CHECKED((bool)(p), 2) != 0)
#define __all_sync(mask, p) (CHECKED((bool)(p), 3) != 0)
#define __reduce_min_sync(mask, v) ((uint32_t)CHECKED(v, 4))
#define __reduce_max_sync(mask, v) ((uint32_t)CHECKED(v, 5))
#define __reduce_add_sync(mask, v) ((uint32_t)CHECKED(v, 6))
#define __reduce_or_sync(mask, v) ((uint32_t)CHECKED(v, 7))
#define __match_any_sync(mask, v) ((uint32_t)CHECKED(v, 8))

template <class T> inline T __shfl_sync(unsigned, T v, int) { return (T)opaque((uint64_t)v, 9); }
template <class T> inline T __shfl_xor_sync(unsigned, T v, int) { return (T)opaque((uint64_t)v, 10); }
template <class T> inline T __shfl_up_sync(unsigned, T v, int) { return (T)opaque((uint64_t)v, 11); }
inline void __syncwarp() { opaque(0, 12); }
inline void __syncthreads() { opaque(0, 13); }
inline void __nanosleep(unsigned) { opaque(0, 14); }

template <class T> T __ldcg(const T* p) { return *(const volatile T*)p; }
inline ulonglong2 __ldcg(const ulonglong2* p) {
    const volatile unsigned long long* q = &p->x;
    return {q[0], q[1]};
}
inline uint4 __ldcg(const uint4* p) {
    const volatile uint32_t* q = &p->x;
    return {q[0], q[1], q[2], q[3]};
}
template <class T> T __ldg(const T* p) { return *(const volatile T*)p; }
template <class T, class U> void __stcg(T* p, U v) { *(volatile T*)p = (T)v; }
inline void __stcg(uint4* p, uint4 v) { *p = v; }

template <class T, class U> T atomicAdd(T* p, U v) { return (T)opaque((uint64_t)p ^ (uint64_t)v, 20); }
template <class T, class U> T atomicMin(T* p, U v) { return (T)opaque((uint64_t)p ^ (uint64_t)v, 21); }
template <class T, class U> T atomicMax(T* p, U v) { return (T)opaque((uint64_t)p ^ (uint64_t)v, 22); }
template <class T, class U> T atomicExch(T* p, U v) { return (T)opaque((uint64_t)p ^ (uint64_t)v, 23); }
template <class T, class U, class V> T atomicCAS(T* p, U c, V v) {
    return (T)opaque((uint64_t)p ^ (uint64_t)c ^ (uint64_t)v, 24);
}

// The headers' inline assembly (see kernel_host.py).
namespace host {
inline uint64_t globaltimer() { return opaque(0, 30); }
inline void cas128(unsigned long long* a, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t& o0, uint64_t& o1) {
    o0 = opaque((uint64_t)a, 31);
    o1 = opaque((uint64_t)a, 32);
}
template <class T> T load(const T* p) { return *(const volatile T*)p; }
template <class T> void store(T* p, T v) { *(volatile T*)p = v; }
template <class T> void add(T* p, T v) { opaque((uint64_t)p ^ v, 33); }
inline void fence() { opaque(0, 34); }
inline void cluster_barrier() { opaque(0, 35); }
inline uint4 load_cluster(const void* p, uint32_t rank) {
    return {(uint32_t)opaque((uint64_t)p, 36), (uint32_t)opaque(rank, 36), (uint32_t)opaque(2, 36), (uint32_t)opaque(3, 36)};
}
template <class T> T& block_shared() {
    static T t;
    return t;
}
template <class T> T& block_context() {
    static T t;
    return t;
}
inline uint4* block_dynamic() { return (uint4*)opaque(0, 37); }
}  // namespace host
