// The search kernel's instantiation for 4x4 boards (search.cuh), in a
// translation unit of its own so that the instantiations compile in parallel.
#include "engine_internal.h"
#include "search.cuh"

namespace gastar {
const void* search_kernel_sliding4() { return reinterpret_cast<const void*>(&search_kernel<kind_bit(KIND_SLIDING4)>); }
}  // namespace gastar
