// What the search kernel's headers use of CUDA, for a host compiler: the parts
// that do not depend on what a warp operation does here.
#pragma once

// The library's headers come first: they use names that are macros below.
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <random>
#include <type_traits>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __grid_constant__
#define __launch_bounds__(...)

struct alignas(16) uint4 {
    uint32_t x, y, z, w;
};
struct uint2 {
    uint32_t x, y;
};
struct alignas(16) ulonglong2 {
    unsigned long long x, y;
};
inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return {a, b, c, d}; }
inline uint2 make_uint2(uint32_t a, uint32_t b) { return {a, b}; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __ffsll(long long v) { return __builtin_ffsll(v); }
inline void __threadfence() {}
