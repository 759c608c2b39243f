// Host side of the level-synchronous kernels (level_kernels.cuh): kernel
// lookup by words per vertex, launches, and the traversed-edge count.
#include "device_common.cuh"

namespace msbfs {

size_t materialize_items(uint32_t V, uint32_t W) {
  const uint32_t tw = W <= 16 ? W : 16;
  const uint32_t tv = MAT_TILE_WORDS / tw;
  return (size_t)((V + tv - 1) / tv) * ((W + tw - 1) / tw);
}

size_t materialize_smem_bytes(uint32_t W, uint32_t NP) {
  const uint32_t tw = W <= 16 ? W : 16;
  const uint32_t tv = MAT_TILE_WORDS / tw;
  const uint32_t np = NP < (uint32_t)MAT_NPMAX ? NP : (uint32_t)MAT_NPMAX;
  return (size_t)(1 + np) * tw * (tv + 2) * sizeof(uint32_t);
}

// Traversed edges of a distance matrix (crates/cli/src/bench.rs:478-491).
__global__ void traversed_edges_kernel(uint32_t V, const uint32_t* __restrict__ off,
                                       const uint32_t* __restrict__ dist, uint32_t S,
                                       unsigned long long* out) {
  unsigned long long acc = 0;
  const size_t total = (size_t)S * V;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    if (dist[i] != 0xffffffffu) {
      const uint32_t v = (uint32_t)(i % V);
      acc += __ldg(off + v + 1) - __ldg(off + v);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// Defined in level_kernels.cuh, instantiated in the level_w*.cu files.
template <int W>
void fill_level_info(int num_sms, uint32_t NP, LevelKernelInfo* k);

bool level_kernel_info(uint32_t W, uint32_t NP, int num_sms, LevelKernelInfo* out) {
  switch (W) {
    case 1: fill_level_info<1>(num_sms, NP, out); return true;
    case 2: fill_level_info<2>(num_sms, NP, out); return true;
    case 4: fill_level_info<4>(num_sms, NP, out); return true;
    case 8: fill_level_info<8>(num_sms, NP, out); return true;
    case 16: fill_level_info<16>(num_sms, NP, out); return true;
    case 32: fill_level_info<32>(num_sms, NP, out); return true;
    case 64: fill_level_info<64>(num_sms, NP, out); return true;
    default: return false;
  }
}

static void launch(void* fn, int grid, int block, size_t smem, const LevelParams& p,
                   cudaStream_t s) {
  void* args[] = {(void*)&p};
  cudaLaunchKernel(fn, dim3(grid), dim3(block), args, smem, s);
}

cudaError_t launch_traverse(const LevelParams& p, const LevelKernelInfo& k, int blocks,
                            bool leave_room, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(k.level_block);
  cfg.stream = s;
  cudaLaunchAttribute attrs[2] = {};
  attrs[0].id = cudaLaunchAttributeCooperative;
  attrs[0].val.cooperative = 1;
  // The part of an SM's L1 that is shared memory stays as it is while blocks are
  // on it, and kernels of other streams start beside these only where it is large
  // enough for them: at 72% (164 KB) all of a served request's kernels did, at
  // 65% and by default none before this one's end. It costs the traversal 1-2%
  // (R-MAT 21 S=512 2.42 -> 2.48 ms, R-MAT 22 S=2,048 14.92 -> 14.96; 86% 3.06 / 16.4).
  attrs[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  attrs[1].val.sharedMemCarveout = 72;
  cfg.attrs = attrs;
  cfg.numAttrs = leave_room ? 2 : 1;
  void* args[] = {(void*)&p};
  return cudaLaunchKernelExC(&cfg, k.traverse, args);
}

void launch_init(const LevelParams& p, const LevelKernelInfo& k, cudaStream_t s) {
  launch(k.init, 1, k.level_block, 0, p, s);
}

void launch_queue(const LevelParams& p, const LevelKernelInfo& k, cudaStream_t s) {
  launch(k.queue, k.level_grids[DIR_PUSH], k.level_block, 0, p, s);
}

void launch_level(const LevelParams& p, const LevelKernelInfo& k, uint32_t dir, bool count,
                  cudaStream_t s) {
  if (dir != DIR_PUSH) launch(k.level[DIR_PULL][count], k.level_grids[DIR_PULL], k.level_block, 0, p, s);
  if (dir == DIR_BOTH) launch_queue(p, k, s);
  if (dir != DIR_PULL) launch(k.level[DIR_PUSH][count], k.level_grids[DIR_PUSH], k.level_block, 0, p, s);
}

void launch_materialize(const LevelParams& p, const LevelKernelInfo& k, bool reduce,
                        cudaStream_t s, uint32_t phase, bool narrow) {
  if (reduce) {
    launch(k.reduce[narrow], k.red_grid[narrow], k.red_block[narrow], 0, p, s);
    return;
  }
  void* args[] = {(void*)&p, &phase};
  cudaLaunchKernel(k.materialize, dim3(k.mat_grid), dim3(k.mat_block), args, k.mat_smem, s);
}

void launch_cleanup(const LevelParams& p, const LevelKernelInfo& k, cudaStream_t s) {
  launch(k.cleanup, 256, 256, 0, p, s);
}

void launch_traversed_edges(uint32_t V, const uint32_t* off, const uint32_t* dist,
                            uint32_t num_sources, unsigned long long* out, cudaStream_t s) {
  cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
  traversed_edges_kernel<<<1024, 256, 0, s>>>(V, off, dist, num_sources, out);
}

}  // namespace msbfs
