// The search kernel's instantiation for all kinds, blocks of 9 to 16 warps (search.cuh), in a
// translation unit of its own so that the instantiations compile in parallel.
#include "engine_internal.h"
#include "search.cuh"

namespace gastar {
const void* search_kernel_all16() { return reinterpret_cast<const void*>(&search_kernel<kKindsAll, 512>); }
}  // namespace gastar
