// One-CTA-per-source persistent BFS for low-degree, high-diameter graphs
// (road networks, grids, trees).
//
// Semantics follow crates/shaders/src/workgroup_persistent_bfs.wgsl:62-196
// and crates/gpu_bfs/src/dispatch/workgroup_persistent.rs:288-370 of the
// reference: one workgroup runs a whole single-source BFS with its visited
// bitmap in shared memory and synchronises only inside the block, so a
// ~1,000-level traversal needs no grid-wide step. The GB300 form differs:
// the bitmap takes up to ~227 KB of shared memory (vs 14 KB) and, for larger
// graphs, is split over the shared memory of a thread-block cluster (calls of
// few sources) or moves to an L2-resident global slab per block instead of
// giving up the path; the frontier queues live in one L2-resident global slab of V
// words per resident block (no overflow fallback), distances are exact u32
// written into the caller's row, and the grid is persistent: each resident
// block pulls the next source from an atomic cursor until all sources are
// done. No block ever waits on another.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "../../include/msbfs.h"
#include "cta_expand.cuh"
#include "cta_grid.h"
#include "device_common.cuh"

namespace cg = cooperative_groups;

namespace msbfs {

constexpr uint32_t CTA_DIST_MAX = 0xffffffffu;
// Block forms of cta_bfs_kernel: threads, resident blocks per SM it is built
// for, lanes per frontier vertex. One block walks a whole level between two
// barriers, so a call of few sources wants every frontier vertex in one
// sweep of the block, a call of many wants many blocks per SM. The form is
// chosen by the blocks an SM will hold (the call's sources per SM, at most
// what the bitmaps leave room for). ms a pass, three calls in flight:
//   one block per SM    road 339x338 S=1 / road 1000x1000 S=250 / grid 64x64
//     CTA_WIDE          S=64: 1,024 threads x 4 lanes 0.197 / 5.62 / 0.031,
//     CTA_SMALL         512 x 4 0.233 / 7.68 / 0.028, 256 x 4 0.38 / - /
//                       0.030, 1,024 x 2 0.240 / - / 0.038 (a small graph's
//                       frontier fits 128 vertices, and its barrier is cheaper)
//   two or three        road 339x338 S=256: 512 x 2 0.445, 512 x 4 0.498,
//     CTA_MID           256 x 2 0.445 (alone 0.99 against 0.89), 1,024 x 4 0.60
//   four or more        road 339x338 S=2,048: 256 threads x 2 lanes x 8 blocks
//     CTA_TPUT          2.84, 192 x 2 x 9 2.80, 256 x 1 x 7 3.07, 256 x 2 x 7
//                       2.90, 256 x 4 x 7 3.11, 128 x 2 x 14 3.60
// Global-bitmap mode (graphs whose bitmap does not fit shared memory, with
// wider frontiers) always uses CTA_MID: road 1448x1448 S=512 42 ms, CTA_WIDE 44,
// CTA_TPUT 73.
#ifndef MSBFS_CTA_TPUT_THREADS
#define MSBFS_CTA_TPUT_THREADS 256
#endif
#ifndef MSBFS_CTA_TPUT_MINB
#define MSBFS_CTA_TPUT_MINB 8
#endif
enum : int { CTA_WIDE = 0, CTA_SMALL = 1, CTA_MID = 2, CTA_TPUT = 3 };
template <int FORM>
struct CtaForm {
  static constexpr int THREADS = FORM == CTA_WIDE ? 1024 : FORM == CTA_TPUT ? MSBFS_CTA_TPUT_THREADS : 512;
  static constexpr int MINB = FORM == CTA_WIDE ? 1 : FORM == CTA_TPUT ? MSBFS_CTA_TPUT_MINB : 3;
  static constexpr int LPV = FORM <= CTA_SMALL ? 4 : 2;
};
// Vertices from which one block per SM is the wide one: where frontiers (of the
// order of the square root) exceed the small one's sweep. us of a statistics call,
// wide / small, grids S=1, S=64, roads S=1, S=64: 8,100 vertices 89 / 89, 126 / 125,
// 104 / 101, 178 / 165; 16,384 114 / 128, 174 / 163, 166 / 164, 237 / 223; 25,600
// 161 / 178, 212 / 225, 211 / 237, 326 / 311; 32,761 198 / 224, 248 / 275, 238 /
// 265, 324 / 323; 65,536 324 / 383, 360 / 423, 362 / 447, 445 / 508.
constexpr size_t CTA_WIDE_VERTICES = 32768;
constexpr size_t CTA_MID_BLOCKS = 3;  // most blocks per SM of the middle form
// Global-bitmap mode keeps its per-block scratch (queue slab + bitmap) within
// this many bytes by shrinking the grid.
constexpr size_t CTA_GLOBAL_SCRATCH_BYTES = 4ull << 30;
// Frontier entries per shared-memory queue half (16 KB).
constexpr uint32_t CTA_SMEM_QUEUE = 4096;
// Cluster form: threads of rank 0 (which walks every frontier) and lanes per
// frontier vertex. Road 1448 x 1448, S=64, ms a pass: 1 lane 6.79, 2 lanes
// 6.99, 4 lanes 7.32 (one edge at a time, with a visited test before each
// atomic 9.09). 512 threads were a quarter slower than 1,024.
#ifndef MSBFS_CTA_CLUSTER_THREADS
#define MSBFS_CTA_CLUSTER_THREADS 1024
#endif
constexpr int CTA_CLUSTER_THREADS = MSBFS_CTA_CLUSTER_THREADS;
constexpr int CTA_CLUSTER_LPV = 1;

// GB: the visited bitmap lives in an L2-resident global slab per block (for
// graphs whose bitmap does not fit shared memory) instead of shared memory.
//
// Counters: level L appends through s_cnt[L % 3]; thread 0 clears
// s_cnt[(L+1) % 3] during level L (last read right after the barrier of
// level L-2), so a level needs one block barrier. The per-source statistics
// follow from the frontier sizes, which every thread knows.
template <bool GB, int ER, int FORM>
__global__ void __launch_bounds__(CtaForm<FORM>::THREADS, CtaForm<FORM>::MINB)
    cta_bfs_kernel(CtaParams p) {
  constexpr int THREADS = CtaForm<FORM>::THREADS, LPV = CtaForm<FORM>::LPV;
  extern __shared__ __align__(16) uint32_t smem_dyn[];
  __shared__ uint32_t s_src_idx;
  __shared__ uint32_t s_cnt[5];  // frontier sizes of three levels, pieces of two
  const uint32_t V = p.V;
  const uint32_t words = (V + 31) / 32;
  uint32_t* bits = GB ? p.gbits + (size_t)blockIdx.x * words : smem_dyn;
  // queue halves after the bitmap
  const uint32_t sbits = smem_addr(smem_dyn), scnt = smem_addr(s_cnt);
  const CtaQueue<ER> q{sbits + (GB ? 0 : (words + 1) / 2 * 8),
                       p.gqueue + (size_t)blockIdx.x * V, p.qh, V, p.off};

  for (;;) {
    if (threadIdx.x == 0) {
      s_src_idx = atomicAdd(p.work, 1u);
      for (int k = 0; k < 5; ++k) s_cnt[k] = 0;
    }
    for (uint32_t i = threadIdx.x; i < words; i += THREADS) bits[i] = 0;
    __syncthreads();
    const uint32_t si = s_src_idx;
    if (si >= p.num_sources) break;
    const uint32_t src = p.sources[si];
    uint32_t* row = p.dist ? p.dist + (size_t)si * V : nullptr;
    if (threadIdx.x == 0) {
      bits[src >> 5] = 1u << (src & 31);
      if (row) row[src] = 0;
      q.put_source(src);
    }
    uint32_t n_in = 1, level = 0, reached = 0, slot = 0;  // slot: 4 * (level % 3)
    unsigned long long sum = 0;
    __syncthreads();
    while (n_in) {
      reached += n_in;
      sum += (unsigned long long)level * n_in;
      const uint32_t nslot = slot == 8 ? 0 : slot + 4;
      if (threadIdx.x == 0) sts32(scnt + nslot, 0);
      cta_level<ER, THREADS, LPV>(
          p.erec, p.idx, q, level, n_in, scnt + slot, row,
          [&](uint32_t v, uint32_t bit) {
            return GB ? atomicOr(&bits[v >> 5], bit) : atoms_or(sbits + (v >> 5) * 4, bit);
          },
          p.big ? q.sq + 8 * p.qh : 0u, scnt + 12);
      n_in = lds32(scnt + slot);
      slot = nslot;
      ++level;
    }
    if (row) {
      // Unreached vertices: coalesced sweep of the row guided by the bitmap
      // (read from L2 in global mode: the bits were set by atomics).
      if (reached < V)
        for (uint32_t v = threadIdx.x; v < V; v += THREADS) {
          const uint32_t w = GB ? __ldcg(bits + (v >> 5)) : bits[v >> 5];
          if (!((w >> (v & 31)) & 1u)) row[v] = CTA_DIST_MAX;
        }
    }
    if (p.stats && threadIdx.x == 0) {
      p.stats[si].sum = sum;
      p.stats[si].reached = reached;
      p.stats[si].ecc = level - 1;
    }
    __syncthreads();
  }
}

// Cluster form, for graphs whose visited bitmap does not fit one block's
// shared memory. A cluster of CL blocks serves one source at a time: block
// rank r keeps bitmap words [r*wpb, (r+1)*wpb) in its shared memory, and
// rank 0 runs the traversal exactly as cta_bfs_kernel does, setting visited
// bits of the other ranks' words with atomicOr through distributed shared
// memory (one hop inside the GPC instead of an L2 round trip). The other
// ranks zero their slice before a traversal and fill the unreached vertices
// of their slice after it. Two cluster barriers per source: (1) the source
// index is in every block and every slice is zero, (2) the traversal is done.
// The queue (shared-memory halves in rank 0, then one global slab of V words
// per cluster) and the edge records work as in cta_bfs_kernel.
template <int CL, int ER>
__global__ void __launch_bounds__(CTA_CLUSTER_THREADS, 1) cta_cluster_kernel(CtaParams p) {
  extern __shared__ __align__(16) uint32_t smem_dyn[];
  __shared__ uint32_t s_src_idx;  // written into every block by rank 0
  __shared__ uint32_t s_cnt[3];
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = cluster.block_rank();
  const uint32_t V = p.V;
  const uint32_t words = (V + 31) / 32;
  const uint32_t wpb = (words + CL - 1) / CL;  // bitmap words per block
  const uint32_t w0 = min(words, rank * wpb);
  const uint32_t w1 = min(words, w0 + wpb);
  uint32_t* bits = smem_dyn;  // this block's slice: words [w0, w1)
  const uint32_t sbits = smem_addr(smem_dyn), scnt = smem_addr(s_cnt);
  const CtaQueue<ER> q{sbits + (wpb + 1) / 2 * 8, p.gqueue + (size_t)(blockIdx.x / CL) * V,
                       p.qh, V, p.off};
  // Sets v's bit and returns the bitmap word as it was: in rank 0's own slice
  // or in another block's, reached through distributed shared memory.
  auto mark = [&](uint32_t v, uint32_t bit) -> uint32_t {
    const uint32_t w = v >> 5;
    uint32_t o = 0, base = 0;
#pragma unroll
    for (int r = 1; r < CL; ++r)
      if (w >= r * wpb) {
        o = r;
        base = r * wpb;
      }
    uint32_t at, old;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(at)
                 : "r"(sbits + (w - base) * 4), "r"(o));
    asm volatile("atom.shared::cluster.or.b32 %0, [%1], %2;"
                 : "=r"(old)
                 : "r"(at), "r"(bit)
                 : "memory");
    return old;
  };

  for (;;) {
    if (rank == 0 && threadIdx.x == 0) {
      const uint32_t si = atomicAdd(p.work, 1u);
      for (int r = 0; r < CL; ++r) *cluster.map_shared_rank(&s_src_idx, r) = si;
      s_cnt[0] = s_cnt[1] = s_cnt[2] = 0;
    }
    for (uint32_t i = threadIdx.x; i < w1 - w0; i += blockDim.x) bits[i] = 0;
    cluster.sync();  // (1)
    const uint32_t si = s_src_idx;
    if (si >= p.num_sources) break;  // the same value in every block
    const uint32_t src = p.sources[si];
    uint32_t* row = p.dist ? p.dist + (size_t)si * V : nullptr;
    if (rank == 0) {
      if (threadIdx.x == 0) {
        mark(src, 1u << (src & 31));
        if (row) row[src] = 0;
        q.put_source(src);
      }
      uint32_t n_in = 1, level = 0, reached = 0, slot = 0;  // slot: 4 * (level % 3)
      unsigned long long sum = 0;
      __syncthreads();
      while (n_in) {
        reached += n_in;
        sum += (unsigned long long)level * n_in;
        const uint32_t nslot = slot == 8 ? 0 : slot + 4;
        if (threadIdx.x == 0) sts32(scnt + nslot, 0);
        cta_expand<ER, CTA_CLUSTER_THREADS, CTA_CLUSTER_LPV, 4 / CTA_CLUSTER_LPV>(
            p.erec, p.idx, q, level, n_in, scnt + slot, row, mark);
        __syncthreads();
        n_in = lds32(scnt + slot);
        slot = nslot;
        ++level;
      }
      if (p.stats && threadIdx.x == 0) {
        p.stats[si].sum = sum;
        p.stats[si].reached = reached;
        p.stats[si].ecc = level - 1;
      }
    }
    cluster.sync();  // (2)
    if (row) {
      // Unreached vertices of this block's slice.
      const uint32_t vb = w0 * 32, ve = min(V, w1 * 32);
      for (uint32_t v = vb + threadIdx.x; v < ve; v += blockDim.x)
        if (!((bits[(v >> 5) - w0] >> (v & 31)) & 1u)) row[v] = CTA_DIST_MAX;
    }
    __syncthreads();  // the slice is read above and zeroed at the top
  }
}

// Edge records of a road-like graph: for every edge e = (u, v), {v, off[v] <<
// 4 | out-degree of v}, or, wide, {v | out-degree of v << 28, off[v]}. One thread
// per vertex u.
__global__ void edge_records_kernel(uint32_t V, const uint32_t* __restrict__ off,
                                    const uint32_t* __restrict__ idx, uint2* __restrict__ erec,
                                    bool wide) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < V; u += gridDim.x * blockDim.x) {
    for (uint32_t e = off[u]; e < off[u + 1]; ++e) {
      const uint32_t v = idx[e];
      const uint32_t b = off[v], n = off[v + 1] - b;
      erec[e] = wide ? make_uint2(n * (ER_WIDE_ID + 1) | v, b) : make_uint2(v, b << 4 | n);
    }
  }
}

int edge_record_kind(size_t V, size_t E) {
  if (E < (size_t(1) << 28)) return ER_PACKED;
  return V <= (size_t)ER_WIDE_ID + 1 ? ER_WIDE : ER_NONE;
}

void launch_edge_records(uint32_t V, const uint32_t* off, const uint32_t* idx, uint2* erec,
                         int kind, cudaStream_t s) {
  edge_records_kernel<<<1024, 256, 0, s>>>(V, off, idx, erec, kind == ER_WIDE);
}

constexpr size_t CTA_SMEM_RESERVE = 1024;  // static shared variables and slack

size_t cta_max_vertices(int device) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (optin <= (int)CTA_SMEM_RESERVE) return 0;
  return ((size_t)optin - CTA_SMEM_RESERVE) * 8;
}

// Lets launches of the kernel take all the dynamic shared memory a block can
// have. The limit belongs to the kernel, which calls of other sizes launch from
// other threads: set to each call's size, one call could lower it under another.
static cudaError_t allow_smem(void* fn, int optin) {
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)CTA_SMEM_RESERVE);
}

template <bool GB, int ER>
static void* cta_fn(int form) {
  if constexpr (!GB) {
    if (form == CTA_TPUT) return (void*)cta_bfs_kernel<GB, ER, CTA_TPUT>;
    if (form == CTA_WIDE) return (void*)cta_bfs_kernel<GB, ER, CTA_WIDE>;
    if (form == CTA_SMALL) return (void*)cta_bfs_kernel<GB, ER, CTA_SMALL>;
  }
  return (void*)cta_bfs_kernel<GB, ER, CTA_MID>;
}

static void* cta_kernel(const CtaShape& sh) {
  if (sh.global_bits)  // (the only mode of graphs with wide records: they have 2^26 vertices)
    return sh.edge_records == ER_WIDE     ? cta_fn<true, ER_WIDE>(sh.form)
           : sh.edge_records == ER_PACKED ? cta_fn<true, ER_PACKED>(sh.form)
                                          : cta_fn<true, ER_NONE>(sh.form);
  return sh.edge_records ? cta_fn<false, ER_PACKED>(sh.form) : cta_fn<false, ER_NONE>(sh.form);
}

template <int CL, int ER>
static void* cta_cluster_fn() {
  return (void*)cta_cluster_kernel<CL, ER>;
}

static void* cluster_kernel(int cl, bool er) {
  switch (cl) {
    case 2: return er ? cta_cluster_fn<2, ER_PACKED>() : cta_cluster_fn<2, ER_NONE>();
    case 4: return er ? cta_cluster_fn<4, ER_PACKED>() : cta_cluster_fn<4, ER_NONE>();
    case 8: return er ? cta_cluster_fn<8, ER_PACKED>() : cta_cluster_fn<8, ER_NONE>();
    default: return nullptr;
  }
}

// Clusters that can be resident at once for a cluster launch of `cl` blocks
// with `smem` bytes of dynamic shared memory each (0 if it cannot launch).
static int cluster_capacity(int cl, bool er, size_t smem, int block, int optin) {
  void* fn = cluster_kernel(cl, er);
  if (!fn) return 0;
  if (allow_smem(fn, optin) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(cl);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cl;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

// Cluster mode for a call of few sources: the smallest cluster whose slices
// hold the bitmap next to rank 0's queue halves. MSBFS_CTA_CLUSTER=0 turns
// it off, =1 uses it whatever the number of sources.
static bool cta_cluster_shape(uint32_t V, int optin, int edge_records, size_t num_sources,
                              uint32_t sm_share, CtaShape* out) {
  const char* env = getenv("MSBFS_CTA_CLUSTER");
  const int mode = env ? atoi(env) : -1;
  if (mode == 0) return false;
  const size_t words = ((size_t)V + 31) / 32;
  const size_t entry = sizeof(uint32_t);  // a vertex id or a packed edge range
  const size_t slack = 2048;
  for (int cl : {2, 4, 8}) {
    const size_t wpb = (words + cl - 1) / cl;
    const size_t slice = (wpb + 1) / 2 * 2 * sizeof(uint32_t);
    if (slice + 2 * 1024 * entry + slack > (size_t)optin) continue;
    const size_t room = (size_t)optin - slack - slice;
    CtaShape sh{};
    sh.block = CTA_CLUSTER_THREADS;
    sh.edge_records = edge_records;
    sh.cluster = cl;
    sh.qh = (uint32_t)std::min<size_t>(CTA_SMEM_QUEUE, room / (2 * entry) / 32 * 32);
    sh.smem = slice + 2 * (size_t)sh.qh * entry;
    const int n = cluster_capacity(cl, edge_records, sh.smem, sh.block, optin);
    if (n < 1) continue;
    // A cluster traverses a source faster than a global-bitmap block, but a
    // global-bitmap launch keeps several blocks per SM busy: clusters pay
    // off while every source has a cluster of its own (road 1448 x 1448:
    // S=64 10.7 vs 18.8 ms; S=152, two sources per cluster, 21.2 vs 22.1;
    // S=256 46.3 vs 28.0 with a 512-thread rank 0).
    if (mode != 1 && num_sources > (size_t)n) return false;
    sh.grid = std::max(1, (int)((uint64_t)n * sm_share / 100)) * cl;
    *out = sh;
    return true;
  }
  return false;
}

bool cta_launch_shape(uint32_t V, int device, bool allow_global, int edge_records,
                      size_t num_sources, uint32_t sm_share, CtaShape* out) {
  int sms = 0, optin = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
  const size_t words = ((size_t)V + 31) / 32;
  const size_t entry = sizeof(uint32_t);  // a vertex id or a packed edge range
  const bool shared_bits = (size_t)V <= cta_max_vertices(device);
  if (!shared_bits && !allow_global) return false;
  if (!shared_bits && cta_cluster_shape(V, optin, edge_records, num_sources, sm_share, out))
    return true;
  CtaShape sh{};
  sh.edge_records = edge_records;
  sh.global_bits = !shared_bits;
  const size_t bitmap = shared_bits ? (words + 1) / 2 * 2 * sizeof(uint32_t) : 0;
  const size_t slack = 2048;  // static shared variables + the driver's per-block reserve
  const size_t fit = std::max<size_t>(1, (size_t)per_sm / (bitmap + slack));
  const size_t per = std::min(fit, (num_sources + sms - 1) / std::max(sms, 1));
  if (shared_bits && per > CTA_MID_BLOCKS) {
    sh.form = CTA_TPUT;
    sh.block = CtaForm<CTA_TPUT>::THREADS;
    sh.minb = CtaForm<CTA_TPUT>::MINB;
  } else if (per > 1 || !shared_bits) {
    sh.form = CTA_MID;
    sh.block = CtaForm<CTA_MID>::THREADS;
    sh.minb = CtaForm<CTA_MID>::MINB;
  } else {
    sh.form = V >= CTA_WIDE_VERTICES ? CTA_WIDE : CTA_SMALL;
    sh.block = V >= CTA_WIDE_VERTICES ? CtaForm<CTA_WIDE>::THREADS : CtaForm<CTA_SMALL>::THREADS;
    sh.minb = 1;
  }
  // The queue halves get the shared memory left once the bitmaps of minb
  // resident blocks have theirs, so the queue never costs a resident block.
  // A frontier beyond the halves continues in the global slab.
  const size_t blocks = std::min<size_t>((size_t)sh.minb, fit);
  const size_t budget = std::min<size_t>((size_t)per_sm / blocks, (size_t)optin) - slack;
  size_t room = budget > bitmap ? budget - bitmap : 0;
  // Without edge records, room for long lists' pieces if some is left for the
  // queue (ms: star of 100,000 leaves 15.3 -> 0.4, R-MAT 16 S=1 2.63 -> 1.39).
  sh.big = !edge_records && room >= BIG_BYTES + 4096;
  if (sh.big) room -= BIG_BYTES;
  sh.qh = (uint32_t)std::min<size_t>(CTA_SMEM_QUEUE, room / (2 * entry) / 32 * 32);
  sh.smem = bitmap + 2 * (size_t)sh.qh * entry + (sh.big ? BIG_BYTES : 0);
  void* fn = cta_kernel(sh);
  int occ = 0;
  if (allow_smem(fn, optin) != cudaSuccess) cudaGetLastError();
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, sh.block, sh.smem);
  if (occ < 1) return false;
  sh.grid = std::max(1, (int)((uint64_t)sms * occ * sm_share / 100));
  if (!shared_bits) {
    // Two thirds of the L2 for bitmaps, but not fewer than one per SM.
    int l2 = 0;
    cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, device);
    const size_t in_l2 = (size_t)l2 / 3 * 2 / (words * sizeof(uint32_t)) / sms * sms;
    sh.grid = (int)global_bitmap_grid(sh.grid, std::max<size_t>(in_l2, sms), num_sources);
    const size_t per_block = ((size_t)V + words) * sizeof(uint32_t);
    sh.grid = (int)std::max<size_t>(
        1, std::min<size_t>((size_t)sh.grid, CTA_GLOBAL_SCRATCH_BYTES / per_block));
  }
  *out = sh;
  return true;
}

void launch_cta(const CtaParams& params, const CtaShape& sh, int grid, cudaStream_t s) {
  CtaParams p = params;
  p.qh = sh.qh;  // the dynamic shared memory holds exactly these queue halves
  p.big = sh.big;
  if (!sh.edge_records) p.erec = nullptr;
  if (sh.cluster > 1) {
    // grid: blocks, a multiple of the cluster size (checked by the caller)
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(sh.block);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = sh.cluster;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    void* args[] = {&p};
    cudaLaunchKernelExC(&cfg, cluster_kernel(sh.cluster, sh.edge_records), args);
    return;
  }
  void* args[] = {&p};
  cudaLaunchKernel(cta_kernel(sh), dim3(grid), dim3(sh.block), args, sh.smem, s);
}

// ---------------------------------------------------------------------------
// Allocation-free form of the CTA-per-source launch.
//
// Its scratch -- a copy of the sources, the source cursor and one frontier
// queue slab (V words) per resident block -- lives in this fixed array
// instead of engine-owned cudaMalloc memory, so the entry point below never
// allocates. Every GPU that loads the library holds the array until exit.
// Layout in u32 words: [0] source cursor, [NOALLOC_SRC_OFF, +NOALLOC_SRC_CAP)
// sources of the current chunk, [NOALLOC_Q_OFF, end) queue slabs.
constexpr size_t NOALLOC_WORDS = MSBFS_NOALLOC_SCRATCH_BYTES / sizeof(uint32_t);
constexpr size_t NOALLOC_SRC_OFF = 64;
constexpr size_t NOALLOC_SRC_CAP = 65536;
constexpr size_t NOALLOC_Q_OFF = NOALLOC_SRC_OFF + NOALLOC_SRC_CAP;
static __device__ __align__(256) uint32_t g_noalloc_scratch[NOALLOC_WORDS];

namespace {
std::mutex g_noalloc_mu;
uint32_t* g_noalloc_addr[64];  // device address of the array, per device
}  // namespace

}  // namespace msbfs

namespace {

// Restores the calling thread's current device when the entry point returns.
struct DeviceRestore {
  int prev = -1;
  DeviceRestore() {
    if (cudaGetDevice(&prev) != cudaSuccess) {
      cudaGetLastError();
      prev = -1;
    }
  }
  ~DeviceRestore() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

}  // namespace

extern "C" int msbfs_run_cta_noalloc(int device, size_t num_vertices,
                                     const uint32_t* row_offsets_device,
                                     const uint32_t* col_indices_device,
                                     const uint32_t* sources, size_t num_sources,
                                     uint32_t* dist_device, void* cuda_stream) {
  using namespace msbfs;
  if (num_sources == 0) return MSBFS_OK;
  if (device < 0 || device >= 64) return MSBFS_ERR_NO_DEVICE;
  if (!row_offsets_device || !col_indices_device || !sources || !dist_device)
    return MSBFS_ERR_INVALID_ARGUMENT;
  if (num_vertices == 0) return MSBFS_ERR_EMPTY_GRAPH;
  for (size_t i = 0; i < num_sources; ++i)
    if ((size_t)sources[i] >= num_vertices) return MSBFS_ERR_SOURCE_OOB;
  // Size limits, checked before touching the device: the visited bitmap must
  // fit shared memory and at least one queue slab must fit the scratch array.
  if (num_vertices > MSBFS_NOALLOC_MAX_VERTICES ||
      NOALLOC_Q_OFF + num_vertices > NOALLOC_WORDS)
    return MSBFS_ERR_SCRATCH_TOO_SMALL;
  const DeviceRestore restore;
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return MSBFS_ERR_NO_DEVICE;
  }
  // Once per device, with that device current: the array's device address
  // (in host code the symbol itself is only a host-side stand-in).
  uint32_t* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[device]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return MSBFS_ERR_CUDA;
      }
      g_noalloc_addr[device] = static_cast<uint32_t*>(p);
    }
    base = g_noalloc_addr[device];
  }
  const uint32_t V = (uint32_t)num_vertices;
  CtaShape sh{};
  if (!cta_launch_shape(V, device, /*allow_global=*/false, /*edge_records=*/ER_NONE, num_sources,
                        /*sm_share=*/100, &sh))
    return MSBFS_ERR_SCRATCH_TOO_SMALL;
  const size_t slabs = (NOALLOC_WORDS - NOALLOC_Q_OFF) / (size_t)V;
  const cudaStream_t s = static_cast<cudaStream_t>(cuda_stream);
  // A non-sticky error left on this thread by earlier work would otherwise
  // be reported as this call's launch failure below.
  cudaGetLastError();
  for (size_t s0 = 0; s0 < num_sources; s0 += NOALLOC_SRC_CAP) {
    const size_t n = std::min(NOALLOC_SRC_CAP, num_sources - s0);
    // The cursor must start at zero; queue slabs need no clearing. Chunks
    // follow one another in stream order, so a chunk's copy of its sources
    // cannot overwrite those of the chunk before it while that one runs.
    if (cudaMemsetAsync(base, 0, sizeof(uint32_t), s) != cudaSuccess ||
        cudaMemcpyAsync(base + NOALLOC_SRC_OFF, sources + s0, n * sizeof(uint32_t),
                        cudaMemcpyHostToDevice, s) != cudaSuccess) {
      cudaGetLastError();
      return MSBFS_ERR_CUDA;
    }
    CtaParams cp{};
    cp.V = V;
    cp.off = row_offsets_device;
    cp.idx = col_indices_device;
    cp.sources = base + NOALLOC_SRC_OFF;
    cp.num_sources = (uint32_t)n;
    cp.dist = dist_device + s0 * num_vertices;
    cp.gqueue = base + NOALLOC_Q_OFF;
    cp.work = base;
    const int blocks = (int)std::min<size_t>({(size_t)sh.grid, n, slabs});
    launch_cta(cp, sh, blocks, s);
    if (cudaGetLastError() != cudaSuccess) return MSBFS_ERR_CUDA;
  }
  return MSBFS_OK;
}
