// The search kernel's instantiation for all kinds, blocks of up to 8 warps (batches, server) (search.cuh), in a
// translation unit of its own so that the instantiations compile in parallel.
#include "engine_internal.h"
#include "search.cuh"

namespace gastar {
const void* search_kernel_all() { return reinterpret_cast<const void*>(&search_kernel<kKindsAll>); }
}  // namespace gastar
