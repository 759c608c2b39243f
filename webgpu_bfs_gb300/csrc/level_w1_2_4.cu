// Level-synchronous kernels at 1, 2 and 4 words per vertex.
#include "level_kernels.cuh"

namespace msbfs {
template void fill_level_info<1>(int, uint32_t, LevelKernelInfo*);
template void fill_level_info<2>(int, uint32_t, LevelKernelInfo*);
template void fill_level_info<4>(int, uint32_t, LevelKernelInfo*);
}  // namespace msbfs
