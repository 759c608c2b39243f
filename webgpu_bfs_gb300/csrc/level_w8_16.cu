// Level-synchronous kernels at 8 and 16 words per vertex.
#include "level_kernels.cuh"

namespace msbfs {
template void fill_level_info<8>(int, uint32_t, LevelKernelInfo*);
template void fill_level_info<16>(int, uint32_t, LevelKernelInfo*);
}  // namespace msbfs
