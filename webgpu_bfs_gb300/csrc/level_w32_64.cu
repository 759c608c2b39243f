// Level-synchronous kernels at 32 and 64 words per vertex.
#include "level_kernels.cuh"

namespace msbfs {
template void fill_level_info<32>(int, uint32_t, LevelKernelInfo*);
template void fill_level_info<64>(int, uint32_t, LevelKernelInfo*);
}  // namespace msbfs
