// The search kernel's instantiation for 3x3 boards (search.cuh), in a
// translation unit of its own so that the instantiations compile in parallel.
#include "engine_internal.h"
#include "search.cuh"

namespace gastar {
const void* search_kernel_sliding3() { return reinterpret_cast<const void*>(&search_kernel<kind_bit(KIND_SLIDING3)>); }
}  // namespace gastar
