// Engine: the C ABI of include/msbfs.h over the sm_103a kernels.
//
// Mirrors crates/gpu_bfs/src/engine.rs of the reference (GpuBfsEngine: method
// enum, Auto router, per-call source validation, pooled device buffers behind
// a mutex) with a CUDA runtime underneath instead of wgpu:
//  * graphs are uploaded once and stay resident (CSR + CSC, aliased when the
//    graph is symmetric, like PushPullGraphBuffers in buffer.rs:108-221);
//  * a level-synchronous pass is one cooperative launch that runs the source
//    init and every level (the last block of a level decides the next one, so
//    no host round trip per level or per batch of levels, replacing
//    multi_word_bp.rs:730-814's speculative 4..64-hop submits and
//    indirect_sparse_push.rs:1462-1578's macro batches), and the distance
//    materialisation;
//  * the CTA-per-source path is one persistent launch per call.
#include <cuda_runtime.h>

#include <algorithm>
#include <condition_variable>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "../../include/msbfs.h"
#include "device_common.cuh"
#include "host_graph.h"
#include "host_pool.h"

using namespace msbfs;

#ifndef MSBFS_PUSH_SEG
#define MSBFS_PUSH_SEG 64
#endif
#ifndef MSBFS_PUSH_SEG0
#define MSBFS_PUSH_SEG0 8  // out-edges per entry of the sources' queue
#endif

namespace {

struct Workspace;

}  // namespace

struct msbfs_graph {
  msbfs_engine* eng = nullptr;
  std::vector<msbfs_engine*> users;  // other engines of the device that may run on it
  uint64_t id = 0;  // unique in the process: keys every engine's workspaces
  size_t V = 0, E = 0;
  bool sym = false;
  uint32_t max_deg = 0;
  uint32_t* off = nullptr;   // CSR
  uint32_t* idx = nullptr;
  uint32_t* coff = nullptr;  // CSC (== CSR when symmetric)
  uint32_t* cidx = nullptr;
  // Bottom-up steps: in-edge lists of `heavy` and more are scanned by whole
  // warps, in slices of at most `split`.
  uint32_t split = 0, heavy = 0;  // as asked for (the tables may use shorter slices; heavy 0: by the rule)
  uint32_t scan_degree = 0;       // `heavy` in use
  uint32_t n_heavy = 0;   // vertices of several slices
  uint32_t n_slices = 0;
  void* tables = nullptr;  // the allocation that holds the following three
  uint4* slices = nullptr;
  uint32_t* hslices = nullptr;
  // Bottom-up work order: vertices with 0 < in-degree < heavy, ascending ids.
  uint32_t n_order = 0;
  uint4* order = nullptr;  // {vertex, in-edge begin, in-edge end, 0}
  uint2* erec = nullptr;  // edge records of road-like graphs (CTA path)
  int erec_kind = 0;
  std::vector<uint32_t> h_coff;  // host CSC offsets (V + 1): rebuilds the tables above
};

namespace {

struct Workspace {
  uint64_t graph_id = 0;
  uint32_t W = 0;
  uint64_t wide_bytes = 0;  // state_bytes of its graph and width
  uint32_t mode = 0;
  bool count = false;  // level kernels keep the profiling counters
  LevelParams p{};
  LevelKernelInfo k{};
  LevelCtl* d_ctl = nullptr;
  LevelRec* d_log = nullptr;
  std::vector<void*> allocs;
  // Set when a pass stopped part-way (an error after work was queued): its
  // buffers may hold that pass's bits, so the next call builds a fresh
  // workspace instead of reusing this one.
  bool dirty = false;
  uint32_t next_epoch = 1;  // stamps of later passes start here (0: never enqueued)
  ~Workspace() {
    for (void* a : allocs) cudaFree(a);
  }
};

uint32_t bit_length_u64(uint64_t x) {
  uint32_t n = 0;
  while (x) {
    ++n;
    x >>= 1;
  }
  return n;
}

uint32_t method_path(int m) {
  switch (m) {
    case MSBFS_METHOD_WORKGROUP_PERSISTENT_BFS:
      return MSBFS_PATH_CTA;
    case MSBFS_METHOD_MULTI_WORD_BIT_PARALLEL:
    case MSBFS_METHOD_BIT_PARALLEL_64_PULL:
    case MSBFS_METHOD_INDIRECT_MACRO_BATCH:
      return MSBFS_PATH_PULL;
    case MSBFS_METHOD_BIT_PARALLEL_32:
    case MSBFS_METHOD_BIT_PARALLEL_64:
    case MSBFS_METHOD_SPARSE_BIT_PARALLEL_64:
    case MSBFS_METHOD_MULTI_WORD_BIT_PARALLEL_PUSH:
    case MSBFS_METHOD_BOOLEAN_REACHABILITY:
      return MSBFS_PATH_PUSH;
    default:
      return MSBFS_PATH_HYBRID;
  }
}

uint32_t path_mode(uint32_t path) {
  return path == MSBFS_PATH_PUSH ? MODE_PUSH : path == MSBFS_PATH_PULL ? MODE_PULL : MODE_HYBRID;
}

}  // namespace

struct msbfs_engine {
  int device = 0;
  int method = MSBFS_METHOD_AUTO;
  int num_sms = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t ev_start = nullptr, ev_stop = nullptr, ev_pass = nullptr, ev_copies = nullptr;
  std::mutex mu;
  std::string last_error;
  uint32_t max_words = 0;   // words per vertex of a pass at most (0: choose_words)
  size_t total_mem = 0;     // device memory, once a call wanted a wide pass
  uint32_t alpha = 14;
  uint32_t beta = 24;
  uint32_t seg = MSBFS_PUSH_SEG;  // out-edges per top-down queue entry
#ifndef MSBFS_HEAVY
#define MSBFS_HEAVY 0
#endif
  // In-degree from which a whole warp scans a vertex (0: warp_scan_degree).
  uint32_t heavy = MSBFS_HEAVY;
#ifndef MSBFS_SPLIT
// ms of a traversal with slices of at most 512 / 1,024 / 2,048 (in-degree 64
// on): R-MAT 22 S=512 4.94 / 4.81 / 4.77, S=64 1.70 / 1.57 / 1.55; R-MAT 21 S=64
// statistics 0.981 / 0.889 / 0.895. Smaller graphs get shorter ones.
#define MSBFS_SPLIT 1024
#endif
  uint32_t split = MSBFS_SPLIT;  // in-edge slice length of bottom-up steps
  uint32_t bits_div = 64;
  uint32_t sm_share = 100;  // percent of the resident grid the persistent kernels use
  // Served form: most of it for the next traversals, and reductions in blocks
  // that find room beside another stream's traversal.
  uint32_t traverse_cap = 100;
  bool narrow_reduce = false;
#ifndef MSBFS_MAT_WAVES
// R-MAT scale 22, S=512, materialisation ms: 1 wave (persistent) 1.82, 2
// 1.81, 4 1.69, 8 1.65, one block per tile 1.59. Blocks of a long
// grid-stride loop drift apart and spread their row writes over more DRAM
// pages; a write-only kernel with the same 256-byte row segments reaches
// 6.5 TB/s persistent at 5 blocks per SM and 7.4 TB/s in short blocks.
#define MSBFS_MAT_WAVES 0
#endif
  // Materialisation grid in waves of its resident blocks (0: one block per
  // tile); a smaller SM share keeps it persistent at that share.
  uint32_t mat_waves = MSBFS_MAT_WAVES;
  uint32_t level_cap = 0;   // levels per pass before MSBFS_ERR_TIMEOUT (0: V + 2)
  bool host_loop = false;
  uint32_t traverse_blocks = 0;  // grid of the traversal (MSBFS_TRAVERSE_BLOCKS; 0: get_workspace)
  // Polls of a grid barrier before the traversal gives up (tens of seconds;
  // MSBFS_BARRIER_SPINS), and the word that it then sets (page-locked).
  uint32_t barrier_spins = 1u << 26;
  uint32_t* h_stuck = nullptr;  // (comes with the first level-path call)
  bool zero_copy = true;  // MSBFS_ZERO_COPY=0 stages host output in HBM instead
  bool narrow = true;     // MSBFS_NARROW=0 keeps host-bound rows u32 over the link
  int profiling = 0;
  std::vector<msbfs_level_record> log;       // records of the last call
  LevelRec* h_log = nullptr;                 // pinned, LOG_CAP per pass
  size_t h_log_passes = 0;
  std::vector<cudaEvent_t> lvl_events;       // profiling levels 2 and 3
  std::vector<std::vector<float>> pass_event_ms;
  std::map<std::tuple<uint64_t, uint32_t, uint32_t>, std::unique_ptr<Workspace>> ws;
  // call scratch
  uint32_t* d_sources = nullptr;
  size_t d_sources_cap = 0;
  uint32_t* d_dist = nullptr;
  size_t d_dist_cap = 0;  // u32 elements
  uint8_t* d_dist8 = nullptr;  // byte rows of host-bound calls
  size_t d_dist8_cap = 0;
  uint8_t* h_dist8 = nullptr;  // page-locked landing buffer of the byte rows
  size_t h_dist8_cap = 0;
  std::vector<cudaEvent_t> chunk_events;  // one per landed chunk of byte rows
  HostPool pool;              // host-side output work of the running call
  // Page-locked output: share of a pass's rows written as u32 over the link
  // (MSBFS_SPLIT_ROWS; R-MAT 22, S=512: 1.0 50.5 ms per call, 0.8 47.0,
  // 0.7 45.8, 0.6 44.0, 0.5 ~45).
  double split_frac = 0.6;
  bool last_split = false;   // the last call split its materialisation
  std::vector<uint32_t> split_rows;         // per pass: first byte row
  std::vector<cudaEvent_t> split_events;    // per pass: its byte rows are done
  uint32_t* d_reach = nullptr;
  size_t d_reach_cap = 0;
  uint32_t* d_cta_queue = nullptr;
  size_t d_cta_queue_cap = 0;
  uint32_t* d_cta_bits = nullptr;  // global-bitmap mode of the CTA path
  size_t d_cta_bits_cap = 0;
  uint32_t* d_work = nullptr;
  unsigned long long* d_counter = nullptr;
  SourceStats* d_sstats = nullptr;  // per-source reductions of host-output calls
  size_t d_sstats_cap = 0;
  LevelCtl* h_ctl = nullptr;  // one per pass of the last call, in h_stuck's allocation
  size_t h_ctl_cap = 0;
  // last call
  msbfs_stats last{};
  size_t last_passes = 0;
  bool last_level_path = false;
};

namespace {

int set_err(msbfs_engine* e, int code, const std::string& msg) {
  if (e) e->last_error = msg;
  return code;
}

int cuda_fail(msbfs_engine* e, cudaError_t err, const char* what) {
  cudaGetLastError();  // clear sticky-free errors
  std::string m = std::string(what) + ": " + cudaGetErrorString(err);
  return set_err(e, err == cudaErrorMemoryAllocation ? MSBFS_ERR_OOM : MSBFS_ERR_CUDA, m);
}

#define CK(call)                                            \
  do {                                                      \
    cudaError_t _e = (call);                                \
    if (_e != cudaSuccess) return cuda_fail(eng, _e, #call); \
  } while (0)

// cudaMalloc that gives the engine's pooled workspaces back when the device is
// out of memory, and tries once more.
cudaError_t device_alloc(msbfs_engine* eng, void** ptr, size_t bytes) {
  cudaError_t err = cudaMalloc(ptr, bytes);
  if (err != cudaErrorMemoryAllocation || eng->ws.empty()) return err;
  cudaGetLastError();
  // Earlier asynchronous calls may still run on them.
  if ((err = cudaStreamSynchronize(eng->stream)) != cudaSuccess ||
      (err = cudaStreamSynchronize(eng->copy_stream)) != cudaSuccess)
    return err;
  eng->ws.clear();
  return cudaMalloc(ptr, bytes);
}

template <typename T>
int grow(msbfs_engine* eng, T** ptr, size_t* cap, size_t need) {
  if (need <= *cap && *ptr) return MSBFS_OK;
  if (*ptr) {
    // Earlier asynchronous calls may still read the old buffer.
    CK(cudaStreamSynchronize(eng->stream));
    CK(cudaStreamSynchronize(eng->copy_stream));
    cudaFree(*ptr);
  }
  *ptr = nullptr;
  *cap = 0;
  size_t n = std::max(need, (size_t)1);
  CK(device_alloc(eng, (void**)ptr, n * sizeof(T)));
  *cap = n;
  return MSBFS_OK;
}

int dev_alloc(msbfs_engine* eng, Workspace* w, void** ptr, size_t bytes) {
  if (bytes == 0) bytes = 16;
  CK(device_alloc(eng, ptr, bytes));
  w->allocs.push_back(*ptr);
  CK(cudaMemsetAsync(*ptr, 0, bytes, eng->stream));
  return MSBFS_OK;
}

uint32_t level_planes(const msbfs_graph* g) {
  return std::min<uint32_t>(bit_length_u64(g->V > 1 ? g->V - 1 : 1), 8);
}

// Traversal state of a pass of W words a vertex (the parts that grow with W).
uint64_t state_bytes(const msbfs_graph* g, uint32_t W) {
  return (uint64_t)g->V * W * 4 * (5 + level_planes(g));
}

// Passes above this width are taken for speed only, where memory allows.
constexpr uint32_t PLAIN_WORDS = 16;

// The default width above PLAIN_WORDS keeps the state of an engine's wide passes
// within an eighth of the device memory, and takes at most half of what is free.
bool wide_pass_fits(msbfs_engine* eng, const msbfs_graph* g, uint32_t W, uint32_t mode) {
  const auto it = eng->ws.find(std::make_tuple(g->id, W, mode));
  if (it != eng->ws.end() && !it->second->dirty) return true;
  const uint64_t need = state_bytes(g, W);
  if (eng->total_mem && need > eng->total_mem / 8) return false;
  size_t free_mem = 0;
  if (cudaMemGetInfo(&free_mem, &eng->total_mem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return need <= eng->total_mem / 8 && need <= free_mem / 2;
}

// Blocks of a traversal. Blocks that a small graph cannot feed only make the
// grid barriers of its levels longer: a block per 1,024 lane loads (visited
// pieces and edges).
int traversal_blocks(const msbfs_engine* eng, const msbfs_graph* g, uint32_t W, int resident) {
  const uint64_t loads = (uint64_t)g->V * std::max(1u, W / 4) + g->E;
  const uint64_t blocks = std::min<uint64_t>(resident, std::max<uint64_t>(64, loads / 1024));
  return std::max(1, (int)(blocks * eng->sm_share / 100));
}

int get_workspace(msbfs_engine* eng, const msbfs_graph* g, uint32_t W, uint32_t mode,
                  Workspace** out) {
  auto key = std::make_tuple(g->id, W, mode);
  auto it = eng->ws.find(key);
  if (it != eng->ws.end()) {
    if (!it->second->dirty) {
      *out = it->second.get();
      return MSBFS_OK;
    }
    CK(cudaStreamSynchronize(eng->stream));
    CK(cudaStreamSynchronize(eng->copy_stream));
    eng->ws.erase(it);
  }
  // Workspaces stay pooled until memory runs short (device_alloc); those of wide
  // passes only while they fit the engine's share together.
  if (W > PLAIN_WORDS && !eng->max_words) {
    uint64_t wide = state_bytes(g, W);
    for (auto& kv : eng->ws)
      if (kv.second->W > PLAIN_WORDS) wide += kv.second->wide_bytes;
    if (wide > eng->total_mem / 8) {
      CK(cudaStreamSynchronize(eng->stream));
      CK(cudaStreamSynchronize(eng->copy_stream));
      for (auto o = eng->ws.begin(); o != eng->ws.end();)
        o = o->second->W > PLAIN_WORDS ? eng->ws.erase(o) : std::next(o);
    }
  }
  auto w = std::make_unique<Workspace>();
  w->graph_id = g->id;
  w->W = W;
  w->wide_bytes = state_bytes(g, W);
  w->mode = mode;
  const uint32_t NP = level_planes(g);
  if (!level_kernel_info(W, NP, eng->num_sms, &w->k))
    return set_err(eng, MSBFS_ERR_INVALID_ARGUMENT, "unsupported words per vertex");
  // Work is claimed dynamically, so a smaller grid is only slower, never wrong.
  w->count = eng->profiling == 1 || eng->profiling == 2;
  for (int d = 0; d < 2; ++d)
    w->k.level_grids[d] = std::max(1, (int)((uint64_t)w->k.level_grids[d] * eng->sm_share / 100));
  if (eng->sm_share < 100) {
    w->k.mat_grid = std::max(1, (int)((uint64_t)w->k.mat_grid * eng->sm_share / 100));
  } else {
    const size_t items = materialize_items((uint32_t)g->V, W);
    const size_t want = eng->mat_waves ? (size_t)w->k.mat_grid * eng->mat_waves : items;
    w->k.mat_grid = (int)std::max<size_t>(1, std::min(want, items));
  }
  for (int& grid : w->k.red_grid) grid = std::max(1, (int)((uint64_t)grid * eng->sm_share / 100));
  w->k.traverse_grid = traversal_blocks(eng, g, W, w->k.traverse_resident);
  if (eng->traverse_blocks) w->k.traverse_grid = (int)eng->traverse_blocks;
  LevelParams& p = w->p;
  p.V = (uint32_t)g->V;
  p.W = W;
  p.E = g->E;
  p.out_off = g->off;
  p.out_idx = g->idx;
  p.in_off = g->coff;
  p.in_idx = g->cidx;
  const size_t VW = g->V * (size_t)W;
  p.NP = NP;
  // A level's queue holds each vertex once (the stamp), so V + E/seg
  // entries bound it; the sources' queue (slot 0 at level 0) uses seg0.
  p.qcap = (uint32_t)std::min<uint64_t>(g->V + g->E / eng->seg + 1, 0xFFFFFFFFull);
  const uint64_t qcap0 = std::min<uint64_t>(g->V + g->E / MSBFS_PUSH_SEG0 + 1, 0xFFFFFFFFull);
  p.qcap0 = (uint32_t)qcap0;
  p.mode = mode;
  p.alpha = eng->alpha;
  p.beta = eng->beta;
  p.seg = eng->seg;
  p.seg0 = std::min<uint32_t>(MSBFS_PUSH_SEG0, eng->seg);
  p.bits_div = eng->bits_div;
  p.max_levels = (uint32_t)std::min<uint64_t>(g->V + 2, 0xFFFFFFF0ull);
  if (eng->level_cap) p.max_levels = std::min(p.max_levels, eng->level_cap);
  p.n_slices = g->n_slices;
  p.slices = g->slices;
  p.hslices = g->hslices;
  p.n_order = g->n_order;
  p.order = g->order;
  int rc;
  void* ptr;
  if ((rc = dev_alloc(eng, w.get(), &ptr, VW * 4))) return rc;
  p.vis = (uint32_t*)ptr;
  for (int i = 0; i < 3; ++i) {
    if ((rc = dev_alloc(eng, w.get(), &ptr, VW * 4))) return rc;
    p.F[i] = (uint32_t*)ptr;
  }
  if ((rc = dev_alloc(eng, w.get(), &ptr, VW * 4 * (size_t)p.NP))) return rc;
  p.planes = (uint32_t*)ptr;
  if ((rc = dev_alloc(eng, w.get(), &ptr, VW * 4))) return rc;
  p.ovf = (uint32_t*)ptr;
  for (int i = 0; i < 3; ++i) {
    if ((rc = dev_alloc(eng, w.get(), &ptr, (size_t)(i == 0 ? qcap0 : p.qcap) * 8))) return rc;
    p.Q[i] = (unsigned long long*)ptr;
  }
  if ((rc = dev_alloc(eng, w.get(), &ptr, g->V * 4))) return rc;
  p.stamp = (uint32_t*)ptr;
  const size_t fwords = (g->V + 31) / 32;
  if ((rc = dev_alloc(eng, w.get(), &ptr, 3 * fwords * 4))) return rc;
  for (int i = 0; i < 3; ++i) p.fbits[i] = (uint32_t*)ptr + i * fwords;
  if ((rc = dev_alloc(eng, w.get(), &ptr, sizeof(LevelCtl)))) return rc;
  w->d_ctl = (LevelCtl*)ptr;
  p.ctl = w->d_ctl;
  if ((rc = dev_alloc(eng, w.get(), &ptr, sizeof(GridSync)))) return rc;
  p.sync = (GridSync*)ptr;
  p.spins = eng->barrier_spins;
  if ((rc = dev_alloc(eng, w.get(), &ptr, sizeof(LevelRec) * LOG_CAP))) return rc;
  w->d_log = (LevelRec*)ptr;
  p.log = w->d_log;
  if ((rc = dev_alloc(eng, w.get(), &ptr, (size_t)g->n_heavy * W * 4))) return rc;
  p.hcand = (uint32_t*)ptr;
  if ((rc = dev_alloc(eng, w.get(), &ptr, (size_t)g->n_heavy * 4))) return rc;
  p.hcount = (uint32_t*)ptr;
  p.hlive_words = (g->n_slices + 31) / 32;
  if ((rc = dev_alloc(eng, w.get(), &ptr, (size_t)std::max(p.hlive_words, 1u) * 4))) return rc;
  p.hlive = (uint32_t*)ptr;
  if (p.hlive_words)
    CK(cudaMemsetAsync(p.hlive, 0xFF, p.hlive_words * sizeof(uint32_t), eng->stream));
  *out = w.get();
  eng->ws[key] = std::move(w);
  return MSBFS_OK;
}

// Reserves the stamps of one pass: level L of the pass stamps epoch + L.
int next_epoch(msbfs_engine* eng, Workspace* w) {
  const uint64_t span = (uint64_t)w->p.max_levels + 2;
  if (w->next_epoch + span > 0xFFFFFFFFull) {
    CK(cudaMemsetAsync(w->p.stamp, 0, w->p.V * sizeof(uint32_t), eng->stream));
    w->next_epoch = 1;
  }
  w->p.epoch = w->next_epoch;
  w->next_epoch += (uint32_t)span;
  return MSBFS_OK;
}

int ensure_events(msbfs_engine* eng, size_t n) {
  while (eng->lvl_events.size() < n) {
    cudaEvent_t e;
    CK(cudaEventCreate(&e));
    eng->lvl_events.push_back(e);
  }
  return MSBFS_OK;
}

// Profiling form of the host-driven loop: one level kernel at a time with a
// CUDA event on each side, then the materialisation likewise. The last entry
// of the returned vector is the materialisation.
int run_pass_profiled(msbfs_engine* eng, Workspace* w, bool reduce, std::vector<float>* ms) {
  int rc;
  CK(cudaMemsetAsync(w->d_ctl, 0, sizeof(LevelCtl), eng->stream));
  launch_init(w->p, w->k, eng->stream);
  LevelCtl probe{};
  CK(cudaMemcpyAsync(&probe, w->d_ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost, eng->stream));
  CK(cudaStreamSynchronize(eng->stream));
  ms->clear();
  for (uint32_t L = 0;; ++L) {
    if ((rc = ensure_events(eng, 2))) return rc;
    CK(cudaEventRecord(eng->lvl_events[0], eng->stream));
    if (probe.build_queue) launch_queue(w->p, w->k, eng->stream);
    launch_level(w->p, w->k, probe.dir, w->count, eng->stream);
    CK(cudaEventRecord(eng->lvl_events[1], eng->stream));
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&probe, w->d_ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost, eng->stream));
    CK(cudaStreamSynchronize(eng->stream));
    float t = 0.f;
    cudaEventElapsedTime(&t, eng->lvl_events[0], eng->lvl_events[1]);
    ms->push_back(t);
    if (probe.terminated) break;
    if (L > w->p.max_levels) {
      w->dirty = true;
      return set_err(eng, MSBFS_ERR_TIMEOUT, "level loop did not terminate");
    }
  }
  CK(cudaEventRecord(eng->lvl_events[0], eng->stream));
  launch_materialize(w->p, w->k, reduce, eng->stream);
  CK(cudaEventRecord(eng->lvl_events[1], eng->stream));
  launch_cleanup(w->p, w->k, eng->stream);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(eng->stream));
  float t = 0.f;
  cudaEventElapsedTime(&t, eng->lvl_events[0], eng->lvl_events[1]);
  ms->push_back(t);
  return MSBFS_OK;
}

// Host-driven loop: launches level kernels in speculative batches of 8 and
// reads the control block between batches (extra launches after the last
// level return immediately).
int run_pass_host_loop(msbfs_engine* eng, Workspace* w, bool reduce) {
  CK(cudaMemsetAsync(w->d_ctl, 0, sizeof(LevelCtl), eng->stream));
  launch_init(w->p, w->k, eng->stream);
  LevelCtl probe{};
  for (uint64_t launched = 0;;) {
    const uint32_t dirs = w->mode == MODE_PUSH ? DIR_PUSH : w->mode == MODE_PULL ? DIR_PULL
                                                                                  : DIR_BOTH;
    for (int i = 0; i < 8; ++i) launch_level(w->p, w->k, dirs, w->count, eng->stream);
    launched += 8;
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&probe, w->d_ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost, eng->stream));
    CK(cudaStreamSynchronize(eng->stream));
    if (probe.terminated) break;
    if (launched > (uint64_t)w->p.max_levels + 16) {
      w->dirty = true;
      return set_err(eng, MSBFS_ERR_TIMEOUT, "level loop did not terminate");
    }
  }
  launch_materialize(w->p, w->k, reduce, eng->stream);
  launch_cleanup(w->p, w->k, eng->stream);
  CK(cudaGetLastError());
  return MSBFS_OK;
}

// Words per vertex of a call's passes: up to 64 by default. A pass costs far
// less than twice one of half its width (the levels' latency and fixed parts
// are shared, and a gathered row of 128 bytes costs little more than one of
// 64). ms of a call at up to 16 / 32 / 64 words: Erdos-Renyi 100,000 x 16,
// S=700 0.525 / 0.421 / -, S=2,048 1.125 / 0.893 / 0.705; R-MAT 20, S=513
// 2.00 / 2.05 / -, S=2,048 5.99 / 4.92 / 4.38.
uint32_t choose_words(msbfs_engine* eng, const msbfs_graph* g, size_t S, uint32_t mode) {
  const uint32_t most = eng->max_words ? eng->max_words : 64;
  const uint32_t need = (uint32_t)((std::min<size_t>(S, (size_t)most * 32) + 31) / 32);
  uint32_t W = 1;
  while (W < need) W <<= 1;
  if (!eng->max_words)
    while (W > PLAIN_WORDS && !wide_pass_fits(eng, g, W, mode)) W >>= 1;
  return W;
}

int validate_call(msbfs_engine* eng, const msbfs_graph* g, const uint32_t* sources, size_t S) {
  if (!eng) return MSBFS_ERR_INVALID_ARGUMENT;
  if (!g) return set_err(eng, MSBFS_ERR_INVALID_ARGUMENT, "graph is null");
  if (g->eng != eng && std::find(g->users.begin(), g->users.end(), eng) == g->users.end())
    return set_err(eng, MSBFS_ERR_INVALID_ARGUMENT, "graph belongs to another engine");
  if (S == 0) return MSBFS_OK;
  if (!sources) return set_err(eng, MSBFS_ERR_INVALID_ARGUMENT, "sources is null");
  char buf[160];
  if (g->V == 0) {
    snprintf(buf, sizeof buf, "Source vertex %u at index 0 exceeds graph vertex count 0", sources[0]);
    return set_err(eng, MSBFS_ERR_EMPTY_GRAPH, buf);
  }
  for (size_t i = 0; i < S; ++i)
    if ((size_t)sources[i] >= g->V) {
      snprintf(buf, sizeof buf, "Source vertex %u at index %zu exceeds graph vertex count %zu",
               sources[i], i, g->V);
      return set_err(eng, MSBFS_ERR_SOURCE_OOB, buf);
    }
  return MSBFS_OK;
}

// The router's road test (engine.rs:157-198): low degree, sparse.
bool is_road_like(const msbfs_graph* g) { return g->max_deg <= 8 && g->E <= 4 * g->V; }

int resolve_method(const msbfs_graph* g, int method, size_t S) {
  if (method == MSBFS_METHOD_AUTO) {
    if (g->V == 0 || S == 0) return MSBFS_METHOD_NAIVE_SEQUENTIAL;
    if (is_road_like(g)) return MSBFS_METHOD_WORKGROUP_PERSISTENT_BFS;
    if (g->max_deg >= 128) return MSBFS_METHOD_INDIRECT_SPARSE_QUEUE_PUSH;
    if (S >= 64) return MSBFS_METHOD_MULTI_WORD_BIT_PARALLEL;
    if (S >= 32) return MSBFS_METHOD_BIT_PARALLEL_64;
    if (S > 1) return MSBFS_METHOD_BIT_PARALLEL_32;
    return MSBFS_METHOD_SPARSE_QUEUE;
  }
  return method;
}

// Queues a whole call on eng->stream. dist_dev: S*V output (device) or null
// in reachability mode; reach_dev: V*ceil(S/32) words (device) or null.
// host_out / host_reach: when non-null, rows are copied back per pass on the
// copy stream while later passes run.
int enqueue_call(msbfs_engine* eng, int method, const msbfs_graph* g, const uint32_t* sources,
                 size_t S, uint32_t* dist_dev, uint32_t* reach_dev, uint32_t* host_out,
                 uint32_t* host_reach, SourceStats* stats_dev = nullptr,
                 uint8_t* dist8_dev = nullptr, double split_frac = 0.0) {
  int rc;
  if (stats_dev) CK(cudaMemsetAsync(stats_dev, 0, S * sizeof(SourceStats), eng->stream));
  const int m = resolve_method(g, method, S);
  uint32_t path = method_path(m);
  if (reach_dev && path == MSBFS_PATH_CTA) path = MSBFS_PATH_HYBRID;
  CtaShape cta{};
  if (path == MSBFS_PATH_CTA &&
      !cta_launch_shape((uint32_t)g->V, eng->device, true, g->erec_kind, S, eng->sm_share, &cta))
    path = MSBFS_PATH_HYBRID;
  if (!g->sym && path != MSBFS_PATH_CTA && !g->coff)
    return set_err(eng, MSBFS_ERR_INVALID_GRAPH, "missing transpose");

  eng->last = msbfs_stats{};
  eng->last.method = (uint32_t)m;
  eng->last.path = path;
  eng->last_level_path = path != MSBFS_PATH_CTA;
  if ((rc = grow(eng, &eng->d_sources, &eng->d_sources_cap, S))) return rc;
  CK(cudaEventRecord(eng->ev_start, eng->stream));
  CK(cudaMemcpyAsync(eng->d_sources, sources, S * sizeof(uint32_t), cudaMemcpyHostToDevice,
                     eng->stream));
  const size_t V = g->V;

  if (path == MSBFS_PATH_CTA) {
    // Cluster mode: `blocks` stays a multiple of the cluster size, one
    // queue slab per cluster.
    const int cl = std::max(1, cta.cluster);
    const int blocks = std::max(cl, std::min<int>(cta.grid, (int)std::min<size_t>(S * cl, 1u << 30)) / cl * cl);
    if (V > cta.qh &&  // else every frontier fits the shared-memory halves
        (rc = grow(eng, &eng->d_cta_queue, &eng->d_cta_queue_cap, (size_t)(blocks / cl) * V)))
      return rc;
    if (cta.global_bits &&
        (rc = grow(eng, &eng->d_cta_bits, &eng->d_cta_bits_cap, (size_t)blocks * ((V + 31) / 32))))
      return rc;
    CK(cudaMemsetAsync(eng->d_work, 0, sizeof(uint32_t), eng->stream));
    CtaParams cp{};
    cp.V = (uint32_t)V;
    cp.off = g->off;
    cp.idx = g->idx;
    cp.sources = eng->d_sources;
    cp.num_sources = (uint32_t)S;
    cp.dist = dist_dev;
    cp.gqueue = eng->d_cta_queue;
    cp.work = eng->d_work;
    cp.stats = stats_dev;
    cp.gbits = cta.global_bits ? eng->d_cta_bits : nullptr;
    cp.erec = g->erec;
    launch_cta(cp, cta, blocks, eng->stream);
    CK(cudaGetLastError());
    eng->last.passes = 1;
    eng->last.cta_cluster = cta.cluster > 1 ? (uint32_t)cta.cluster : 0u;
    eng->last_passes = 0;
    if (host_out) {
      CK(cudaMemcpyAsync(host_out, dist_dev, S * V * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                         eng->stream));
    }
    CK(cudaEventRecord(eng->ev_stop, eng->stream));
    return MSBFS_OK;
  }

  const uint32_t mode = path_mode(path);
  uint32_t W = choose_words(eng, g, S, mode);
  Workspace* w = nullptr;
  rc = get_workspace(eng, g, W, mode, &w);
  while (rc == MSBFS_ERR_OOM && W > PLAIN_WORDS && !eng->max_words)
    rc = get_workspace(eng, g, W >>= 1, mode, &w);
  if (rc) return rc;
  const size_t PW = (size_t)W * 32;
  const size_t passes = (S + PW - 1) / PW;
  const bool reduce = stats_dev != nullptr;
  // Split materialisation (one-launch traversal only): the u32 rows follow
  // the byte rows in a second launch, while the host widens the bytes.
  const bool one_launch = !eng->host_loop && eng->profiling == 0;
  const bool split = split_frac > 0.0 && dist8_dev && dist_dev && !reduce && !reach_dev && one_launch;
  eng->last_split = split;
  eng->split_rows.assign(passes, 0);
  while (split && eng->split_events.size() < passes) {
    cudaEvent_t e;
    CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    eng->split_events.push_back(e);
  }
  if (passes > eng->h_ctl_cap) {
    CK(cudaStreamSynchronize(eng->stream));
    const uint32_t stuck = eng->h_stuck ? *eng->h_stuck : 0u;
    if (eng->h_stuck) cudaFreeHost(eng->h_stuck);
    eng->h_stuck = nullptr;
    eng->h_ctl = nullptr;
    eng->h_ctl_cap = 0;
    char* at = nullptr;
    CK(cudaMallocHost((void**)&at, alignof(LevelCtl) + passes * sizeof(LevelCtl)));
    eng->h_stuck = reinterpret_cast<uint32_t*>(at);
    *eng->h_stuck = stuck;
    eng->h_ctl = reinterpret_cast<LevelCtl*>(at + alignof(LevelCtl));
    eng->h_ctl_cap = passes;
  }
  eng->last.passes = (uint32_t)passes;
  eng->last.words_per_vertex = W;
  eng->last_passes = passes;
  if (eng->profiling) {
    if (passes > eng->h_log_passes) {
      CK(cudaStreamSynchronize(eng->stream));
      if (eng->h_log) cudaFreeHost(eng->h_log);
      eng->h_log = nullptr;
      eng->h_log_passes = 0;
      CK(cudaMallocHost((void**)&eng->h_log, passes * LOG_CAP * sizeof(LevelRec)));
      eng->h_log_passes = passes;
    }
    eng->pass_event_ms.assign(passes, {});
  }
  const size_t wpv = (S + 31) / 32;
  // Any early return below leaves passes half-queued: the workspace is
  // retired unless the loop completes.
  w->dirty = true;
  for (size_t ps = 0; ps < passes; ++ps) {
    const size_t s0 = ps * PW;
    const size_t np = std::min(PW, S - s0);
    PassDesc d{};
    d.sources = eng->d_sources + s0;
    d.dist = dist_dev ? dist_dev + s0 * V : nullptr;
    d.reach = reach_dev;
    d.stats = stats_dev ? stats_dev + s0 : nullptr;
    d.dist8 = dist8_dev ? dist8_dev + s0 * V : nullptr;
    d.num_sources = (uint32_t)np;
    d.reach_wpv = (uint32_t)wpv;
    d.reach_col = (uint32_t)(ps * W);
    d.row_split = split ? (uint32_t)(split_frac * (double)np) / 32u * 32u : 0u;
    eng->split_rows[ps] = d.row_split;
    w->p.d = d;
    w->p.h_stuck = eng->h_stuck;
    if ((rc = next_epoch(eng, w))) return rc;
    if (eng->profiling >= 2) {
      if ((rc = run_pass_profiled(eng, w, reduce, &eng->pass_event_ms[ps]))) return rc;
    } else if (!one_launch) {
      if ((rc = run_pass_host_loop(eng, w, reduce))) return rc;
    } else {
      int blocks = w->k.traverse_grid;
      if (eng->traverse_cap < 100)
        blocks = std::min(blocks, std::max(1, (int)((uint64_t)w->k.traverse_resident * eng->traverse_cap / 100)));
      const cudaError_t launched = launch_traverse(
          w->p, w->k, blocks, eng->sm_share < 100 || eng->traverse_cap < 100, eng->stream);
      const bool refused = launched == cudaErrorCooperativeLaunchTooLarge ||
                           launched == cudaErrorLaunchOutOfResources ||
                           launched == cudaErrorNotSupported;
      if (refused) {
        // Its blocks cannot all be resident (a process may be given a part of
        // the device only): the host drives this engine's levels from now on.
        // One materialisation then writes the pass, all its rows in one form.
        cudaGetLastError();
        eng->host_loop = true;
        w->p.d.row_split = eng->split_rows[ps] = 0;
        if ((rc = run_pass_host_loop(eng, w, reduce))) return rc;
      } else {
        CK(launched);
        if (split) launch_materialize(w->p, w->k, false, eng->stream, MAT_BYTES);
      }
      if (split) {
        CK(cudaMemcpyAsync(&eng->h_ctl[ps], w->d_ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost,
                           eng->stream));
        CK(cudaEventRecord(eng->split_events[ps], eng->stream));
      }
      if (!refused)
        launch_materialize(w->p, w->k, reduce, eng->stream, split ? MAT_WIDE : MAT_ALL,
                           eng->narrow_reduce);
      CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(&eng->h_ctl[ps], w->d_ctl, sizeof(LevelCtl), cudaMemcpyDeviceToHost,
                       eng->stream));
    if (eng->profiling)
      CK(cudaMemcpyAsync(eng->h_log + ps * LOG_CAP, w->d_log, LOG_CAP * sizeof(LevelRec),
                         cudaMemcpyDeviceToHost, eng->stream));
    if (host_out) {
      CK(cudaEventRecord(eng->ev_pass, eng->stream));
      CK(cudaStreamWaitEvent(eng->copy_stream, eng->ev_pass, 0));
      CK(cudaMemcpyAsync(host_out + s0 * V, dist_dev + s0 * V, np * V * sizeof(uint32_t),
                         cudaMemcpyDeviceToHost, eng->copy_stream));
    }
  }
  w->dirty = false;
  if (host_reach) {
    CK(cudaMemcpyAsync(host_reach, reach_dev, V * wpv * sizeof(uint32_t),
                       cudaMemcpyDeviceToHost, eng->stream));
  }
  if (host_out) {
    CK(cudaEventRecord(eng->ev_copies, eng->copy_stream));
    CK(cudaStreamWaitEvent(eng->stream, eng->ev_copies, 0));
  }
  CK(cudaEventRecord(eng->ev_stop, eng->stream));
  return MSBFS_OK;
}

int finish_call(msbfs_engine* eng, msbfs_stats* stats) {
  CK(cudaEventSynchronize(eng->ev_stop));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, eng->ev_start, eng->ev_stop);
  eng->last.gpu_ms = ms;
  uint32_t status = 0, check_site = 0;
  for (size_t i = 0; i < eng->last_passes; ++i) {
    const LevelCtl& c = eng->h_ctl[i];
    if (!check_site) check_site = c.check_site;
    eng->last.levels = std::max(eng->last.levels, c.level + 1);
    eng->last.push_levels += c.push_levels;
    eng->last.pull_levels += c.pull_levels;
    eng->last.reached_pairs += c.pairs;
    status |= c.status;
  }
  eng->log.clear();
  if (eng->profiling && eng->h_log) {
    for (size_t ps = 0; ps < eng->last_passes; ++ps) {
      const LevelCtl& c = eng->h_ctl[ps];
      const uint32_t nlev = std::min<uint32_t>(c.level + 1, LOG_CAP);
      const std::vector<float>* ev =
          ps < eng->pass_event_ms.size() ? &eng->pass_event_ms[ps] : nullptr;
      for (uint32_t L = 0; L < nlev; ++L) {
        const LevelRec& r = eng->h_log[ps * LOG_CAP + L];
        msbfs_level_record o{};
        o.pass = (uint32_t)ps;
        o.level = r.level;
        o.dir = r.dir;
        o.frontier_vertices = r.frontier_vertices;
        o.frontier_entries = r.frontier_entries;
        o.active = r.active;
        o.edges = r.edges;
        o.new_vertices = r.new_vertices;
        o.new_pairs = r.new_pairs;
        o.rows = r.rows;
        o.device_ms = r.t_end > r.t_start ? (double)(r.t_end - r.t_start) * 1e-6 : 0.0;
        o.event_ms = (ev && L < ev->size() && !ev->empty()) ? (*ev)[L] : 0.0;
        eng->log.push_back(o);
      }
      if (ev && !ev->empty()) {
        msbfs_level_record m{};
        m.pass = (uint32_t)ps;
        m.level = c.level;
        m.dir = MSBFS_DIR_MATERIALIZE;
        m.event_ms = ev->back();
        eng->log.push_back(m);
      }
    }
  }
  if (stats) *stats = eng->last;
  if (status & STATUS_CHECK)
    return set_err(eng, MSBFS_ERR_CUDA,
                   "bounds check failed at site " + std::to_string(check_site));
  // Also when it was an earlier asynchronous call that got stuck: its rows are
  // void, and the calls queued behind it on the same workspace did nothing.
  if ((status & STATUS_STUCK) || (eng->h_stuck && *(volatile uint32_t*)eng->h_stuck)) {
    CK(cudaStreamSynchronize(eng->stream));
    eng->ws.clear();  // the pass left its traversal state as it was
    *eng->h_stuck = 0;
    return set_err(eng, MSBFS_ERR_TIMEOUT, "a level's grid barrier ran out of time");
  }
  if (status & STATUS_LEVEL_CAP) return set_err(eng, MSBFS_ERR_TIMEOUT, "level cap reached");
  if (status & STATUS_BAD_SOURCE) return set_err(eng, MSBFS_ERR_SOURCE_OOB, "source out of range");
  return MSBFS_OK;
}

// From which in-degree a whole warp scans a vertex: 64 on graphs with at least
// 3 vertices of in-degree 32-63 per resident warp, else 32. Such a list fills
// one or two rounds of a warp, each as long as the latency of its dependent
// loads; vertices side by side in a tile share that latency, but a tile lasts
// as long as its longest list, which only evens out over many. ms of a
// traversal with 32 / 64 (vertices per warp): Erdos-Renyi of degree 40, 1 M
// vertices, S=512 (125) 3.80 / 2.32, S=64 2.18 / 1.17; of degree 32, 400 K, S=64
// (29) 0.650 / 0.469; of degree 24, 400 K, S=512 (3.7) 0.824 / 0.774; R-MAT 20 S=1
// (10) 0.277 / 0.244, R-MAT 20 of edge factor 32, S=512 (3.7) 1.63 / 1.59; below
// the line R-MAT 18 S=512 (1.9) 0.515 / 0.553, R-MAT 20 of edge factor 8, S=64
// (1.7) 0.421 / 0.467, R-MAT 13 S=200 (0.03) 0.110 / 0.133. Against 64, 128 is
// 1-2% slower on R-MAT 21 and 22; 16 loses to 32 on R-MAT 20 and larger.
uint32_t warp_scan_degree(const msbfs_engine* eng, const std::vector<uint32_t>& coff) {
  constexpr size_t LEVEL_WARPS_PER_SM = 48;  // resident: 6 blocks of 8 (level_kernels.cuh)
  size_t mid = 0;
  for (size_t v = 0; v + 1 < coff.size(); ++v) mid += coff[v + 1] - coff[v] - 32 < 32;
  return mid >= 3 * LEVEL_WARPS_PER_SM * (size_t)eng->num_sms ? 64 : 32;
}

// Slice table of the vertices of in-degree >= heavy and the bottom-up work
// list of the other vertices with in-edges, from the graph's host CSC
// offsets. Rebuilt when the autotuner changes the slice length or the
// in-degree; the caller drops the workspaces that point at the old tables
// first.
int build_bottom_up_tables(msbfs_engine* eng, msbfs_graph* g, uint32_t split, uint32_t heavy) {
  const size_t V = g->V;
  const std::vector<uint32_t>& coff = g->h_coff;
  g->heavy = heavy;
  if (!heavy) heavy = warp_scan_degree(eng, coff);
  g->scan_degree = heavy;
  cudaFree(g->tables);
  g->tables = nullptr;
  g->slices = nullptr;
  g->hslices = nullptr;
  g->order = nullptr;
  g->split = split;
  g->n_heavy = 0;
  // A slice is one warp's serial work. With less than a full slice of edges
  // per warp slot of the device (64 an SM), shorter ones: a level of a small graph lasts as long
  // as its longest slice (directed R-MAT 18, S=333: bottom-up levels of 220 us
  // behind warps that scanned up to 16 vertices of <= 512 in-edges). Not below
  // 256: a list's slices meet in its candidate words, two fences and an atomic
  // each. us of a traversal with at least 64 / 128 / 256 / 512: directed R-MAT
  // 18 S=333 359 / 343 / 334 / 355, R-MAT 16 S=100 231 / 200 / 198 / 220, R-MAT
  // 14 S=64 147 / 136 / 134 / 124, R-MAT 10 S=300 109 / 118 / 122 / 121.
  uint32_t len = split;
  const uint64_t warps = (uint64_t)eng->num_sms * 64;
  while (len > 256 && (uint64_t)len * warps > g->E) len /= 2;
  // Heavy vertices by in-degree, descending (a counting sort; those beyond
  // its range keep their order in front).
  uint32_t max_in = 0;
  for (size_t v = 0; v < V; ++v) max_in = std::max(max_in, coff[v + 1] - coff[v]);
  const uint32_t TOP = std::min(max_in + 2, 1u << 16);
  std::vector<uint32_t> at(TOP + 1, 0), by_degree;
  auto degree_rank = [&](size_t v) { return TOP - 1 - std::min(coff[v + 1] - coff[v], TOP - 1); };
  heavy = std::max(heavy, 1u);
  for (size_t v = 0; v < V; ++v)
    if (coff[v + 1] - coff[v] >= heavy) at[degree_rank(v) + 1]++;
  for (uint32_t i = 0; i < TOP; ++i) at[i + 1] += at[i];
  by_degree.resize(at[TOP]);
  for (size_t v = 0; v < V; ++v)
    if (coff[v + 1] - coff[v] >= heavy) by_degree[at[degree_rank(v)]++] = (uint32_t)v;
  std::vector<uint32_t> per_vertex;  // slices of each vertex of several
  std::vector<uint32_t> h(by_degree.size());
  size_t many = 0;  // the vertices of several slices come first
  for (size_t i = 0; i < by_degree.size(); ++i) {
    const uint32_t v = by_degree[i], d = coff[v + 1] - coff[v];
    h[i] = d > len ? g->n_heavy++ : SLICE_H;
    if (d > len) {
      per_vertex.push_back((d + len - 1) / len);
      many = i + 1;
    }
  }
  // First slices first: by the time a vertex's later slices run, the lanes
  // its first ones found are published, and they can stop at once.
  std::vector<uint4> table;  // slices, then the work order, then the slice counts
  for (uint32_t j = 0;; ++j) {
    const size_t before = table.size();
    for (size_t i = 0; i < (j ? many : by_degree.size()); ++i) {
      const uint32_t v = by_degree[i], d = coff[v + 1] - coff[v];
      const uint64_t first = (uint64_t)j * len;
      if (first >= d) {
        if (d < TOP - 1) break;  // shorter lists follow
        continue;
      }
      const uint32_t sb = coff[v] + (uint32_t)first;
      const uint32_t se = d - first > len ? sb + len : coff[v + 1];
      table.push_back(make_uint4(v, sb, se, h[i] | (j ? 0u : SLICE_FIRST)));
    }
    if (table.size() == before) break;
  }
  g->n_slices = (uint32_t)table.size();
  // Bottom-up work list: the other vertices with in-edges, ascending ids
  // (neighbouring vertices share cache lines of the visited and frontier
  // rows; sorting them by in-degree within windows of 256 or 1,024 entries,
  // for groups of similar length, cost 8 and 10% on R-MAT scale 22, S=512).
  // Each entry carries the vertex and its in-edge range, so a bottom-up
  // step starts a vertex's scan one dependent load earlier.
  table.reserve(table.size() + V + per_vertex.size() / 4 + 1);
  for (size_t v = 0; v < V; ++v) {
    const uint32_t b = coff[v], e = coff[v + 1];
    if (e > b && e - b < heavy) table.push_back(make_uint4((uint32_t)v, b, e, 0u));
  }
  const size_t counts = table.size();
  g->n_order = (uint32_t)(counts - g->n_slices);
  for (size_t i = 0; i < per_vertex.size(); i += 4) {
    uint32_t c[4] = {};
    for (size_t k = i; k < std::min(i + 4, per_vertex.size()); ++k) c[k - i] = per_vertex[k];
    table.push_back(make_uint4(c[0], c[1], c[2], c[3]));
  }
  const size_t bytes = table.size() * sizeof(uint4);
  CK(device_alloc(eng, &g->tables, std::max<size_t>(bytes, 16)));
  if (bytes) CK(cudaMemcpy(g->tables, table.data(), bytes, cudaMemcpyHostToDevice));
  g->slices = static_cast<uint4*>(g->tables);
  g->order = g->slices + g->n_slices;
  g->hslices = reinterpret_cast<uint32_t*>(g->slices + counts);
  return MSBFS_OK;
}

int upload_graph(msbfs_engine* eng, size_t V, size_t E, const uint32_t* off, const uint32_t* idx,
                 msbfs_graph** out) {
  if (!eng || !out) return MSBFS_ERR_INVALID_ARGUMENT;
  if (V >= 0xFFFFFFFFull || E > 0xFFFFFFFFull)
    return set_err(eng, MSBFS_ERR_INVALID_GRAPH, "graph exceeds u32 indices");
  std::string why = msbfs::validate(V, E, off, idx, E);
  if (!why.empty()) return set_err(eng, MSBFS_ERR_INVALID_GRAPH, why);
  auto g = std::make_unique<msbfs_graph>();
  g->eng = eng;
  static std::atomic<uint64_t> next_graph_id{1};
  g->id = next_graph_id++;
  g->V = V;
  g->E = E;
  g->max_deg = msbfs::max_degree(V, off);
  msbfs::HostCsr t = msbfs::transpose(V, E, off, idx);
  g->sym = std::equal(t.off.begin(), t.off.end(), off) &&
           (E == 0 || std::memcmp(t.idx.data(), idx, E * 4) == 0);
  CK(cudaSetDevice(eng->device));
  CK(device_alloc(eng, (void**)&g->off, (V + 1) * 4));
  CK(device_alloc(eng, (void**)&g->idx, std::max<size_t>(E, 1) * 4));
  CK(cudaMemcpy(g->off, off, (V + 1) * 4, cudaMemcpyHostToDevice));
  if (E) CK(cudaMemcpy(g->idx, idx, E * 4, cudaMemcpyHostToDevice));
  if (g->sym) {
    g->coff = g->off;
    g->cidx = g->idx;
  } else {
    CK(device_alloc(eng, (void**)&g->coff, (V + 1) * 4));
    CK(device_alloc(eng, (void**)&g->cidx, std::max<size_t>(E, 1) * 4));
    CK(cudaMemcpy(g->coff, t.off.data(), (V + 1) * 4, cudaMemcpyHostToDevice));
    if (E) CK(cudaMemcpy(g->cidx, t.idx.data(), E * 4, cudaMemcpyHostToDevice));
  }
  g->h_coff = std::move(t.off);
  int rc = build_bottom_up_tables(eng, g.get(), eng->split, eng->heavy);
  if (rc) return rc;
  // Road-like graphs (the ones the router sends to the CTA path) get edge
  // records, 8 bytes per edge, so a CTA-path level costs one dependent L2
  // round trip instead of three.
  if (is_road_like(g.get()) && E > 0 && (g->erec_kind = edge_record_kind(V, E))) {
    CK(device_alloc(eng, (void**)&g->erec, E * sizeof(uint2)));
    launch_edge_records((uint32_t)V, g->off, g->idx, g->erec, g->erec_kind, eng->stream);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(eng->stream));
  }
  *out = g.release();
  return MSBFS_OK;
}

void free_graph(msbfs_graph* g) {
  if (!g) return;
  std::vector<msbfs_engine*> engines = g->users;
  engines.push_back(g->eng);
  for (msbfs_engine* eng : engines) {
    if (!eng) continue;
    std::lock_guard<std::mutex> lk(eng->mu);
    cudaSetDevice(eng->device);
    cudaStreamSynchronize(eng->stream);
    for (auto it = eng->ws.begin(); it != eng->ws.end();)
      if (std::get<0>(it->first) == g->id)
        it = eng->ws.erase(it);
      else
        ++it;
  }
  if (!g->sym) {
    cudaFree(g->coff);
    cudaFree(g->cidx);
  }
  cudaFree(g->off);
  cudaFree(g->idx);
  cudaFree(g->tables);
  cudaFree(g->erec);
  delete g;
}

// Copies n byte distances from the device to the host through a ring of
// page-locked chunk slots (one event per slot on the copy stream) while the
// engine's host threads widen each chunk, once it has landed, into u32
// (0xFF -> 0xFFFFFFFF) at `out`: the host link carries a quarter of the
// bytes, and the host's cores, which write memory faster than the link
// delivers it, do the widening. The calling thread issues the copies; a
// slot is refilled only after all workers have widened its previous chunk,
// and a worker waits for its chunk's copy to be issued before it waits on
// the slot's event.
int widen_to_host(msbfs_engine* eng, const uint8_t* src, uint32_t* out, size_t n) {
  if (n == 0) return MSBFS_OK;
  constexpr size_t SLOTS = 16, CHUNK_MAX = 32u << 20;
  // Chunks of an eighth of the rows (1 MB at least), so that small calls
  // overlap their copies with the widening too.
  const size_t CHUNK = std::min(CHUNK_MAX, std::max<size_t>(1u << 20, (n / 8 + 4095) / 4096 * 4096));
  const size_t stage = std::min(n, CHUNK * SLOTS);
  if (stage > eng->h_dist8_cap) {
    if (eng->h_dist8) cudaFreeHost(eng->h_dist8);
    eng->h_dist8 = nullptr;
    eng->h_dist8_cap = 0;
    CK(cudaHostAlloc((void**)&eng->h_dist8, stage, cudaHostAllocDefault));
    eng->h_dist8_cap = stage;
  }
  while (eng->chunk_events.size() < SLOTS) {
    cudaEvent_t e;
    CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    eng->chunk_events.push_back(e);
  }
  const size_t nchunks = (n + CHUNK - 1) / CHUNK;
  // A worker per 256 KB (us into fresh memory with 4 / 16 workers: 1 MB of
  // distances, R-MAT 14 S=64, 289 / 381; 17 MB, R-MAT 17 S=129, 2,114 / 1,616).
  const unsigned T = eng->pool.reserve(
      (unsigned)std::min<size_t>(HostPool::max_workers(), std::max<size_t>(n >> 18, 1)));
  if (!T) return set_err(eng, MSBFS_ERR_OOM, "no thread to widen the byte rows with");
  std::mutex mu;
  std::condition_variable cv;
  size_t issued = 0, widened = 0;  // chunks issued / widened by every worker (in order)
  unsigned slot_done[SLOTS] = {};
  bool failed = false;
  const uint8_t* ring = eng->h_dist8;
  eng->pool.start(T, [&](unsigned k) {
    cudaSetDevice(eng->device);
    for (size_t c = 0; c < nchunks; ++c) {
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return issued > c || failed; });
        if (failed) return;
      }
      const size_t slot = c % SLOTS;
      if (cudaEventSynchronize(eng->chunk_events[slot]) != cudaSuccess) {
        std::lock_guard<std::mutex> lk(mu);
        failed = true;
        cv.notify_all();
        return;
      }
      const size_t b = c * CHUNK, len = std::min(CHUNK, n - b);
      const size_t lo = len * k / T, hi = len * (k + 1) / T;
      const uint8_t* in = ring + slot * CHUNK;
      uint32_t* o = out + b;
      for (size_t i = lo; i < hi; ++i) {
        const uint32_t d = in[i];
        o[i] = d == 0xFFu ? 0xFFFFFFFFu : d;
      }
      std::lock_guard<std::mutex> lk(mu);
      if (++slot_done[slot] == T) {
        slot_done[slot] = 0;
        ++widened;
        cv.notify_all();
      }
    }
  });
  cudaError_t err = cudaSuccess;
  for (size_t c = 0; c < nchunks && err == cudaSuccess; ++c) {
    const size_t slot = c % SLOTS, b = c * CHUNK, len = std::min(CHUNK, n - b);
    {
      std::unique_lock<std::mutex> lk(mu);
      cv.wait(lk, [&] { return c < SLOTS || widened + SLOTS > c || failed; });
      if (failed) break;
    }
    err = cudaMemcpyAsync(eng->h_dist8 + slot * CHUNK, src + b, len, cudaMemcpyDeviceToHost,
                          eng->copy_stream);
    if (err == cudaSuccess) err = cudaEventRecord(eng->chunk_events[slot], eng->copy_stream);
    std::lock_guard<std::mutex> lk(mu);
    if (err == cudaSuccess)
      issued = c + 1;
    else
      failed = true;
    cv.notify_all();
  }
  eng->pool.wait();
  if (failed || err != cudaSuccess) {
    cudaGetLastError();
    return set_err(eng, MSBFS_ERR_CUDA, "byte-row copy failed");
  }
  return MSBFS_OK;
}

// Whether p is ordinary host memory (not page-locked, managed or device).
bool is_pageable(const void* p) {
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return attr.type == cudaMemoryTypeUnregistered;
}

// Waits for the engine's host workers when the scope ends, on every path: the
// caller may free the buffer they work on once the call has returned.
struct PoolScope {
  HostPool& pool;
  ~PoolScope() { pool.wait(); }
};

// Blocking run into caller-owned host memory.
int run_host(msbfs_engine* eng, int method, const msbfs_graph* g, const uint32_t* sources,
             size_t S, uint32_t* out, msbfs_stats* stats) {
  int rc = validate_call(eng, g, sources, S);
  if (rc) return rc;
  if (stats) *stats = msbfs_stats{};
  if (S == 0) return MSBFS_OK;
  if (!out) return set_err(eng, MSBFS_ERR_INVALID_ARGUMENT, "out is null");
  CK(cudaSetDevice(eng->device));
  // Page-locked host output (cudaHostAlloc / cudaHostRegister) is written by
  // the materialise kernel directly over the host link, in 512-byte row
  // segments, instead of being staged in HBM and copied afterwards. The
  // CTA-per-source path stores 4-byte distances as it discovers them, which
  // the host link serves ~9x slower than a staged copy, so it keeps staging.
  const bool cta = method_path(resolve_method(g, method, S)) == MSBFS_PATH_CTA;
  const size_t V = g->V;
  const PoolScope scope{eng->pool};
  uint32_t* zc = nullptr;  // device address of page-locked `out`
  if (eng->zero_copy && !cta) {
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, out) == cudaSuccess &&
        attr.type == cudaMemoryTypeHost && attr.devicePointer)
      zc = (uint32_t*)attr.devicePointer;
    else
      cudaGetLastError();
  }
  // Byte rows (decided on the device for each pass: all its distances fit a
  // byte) widened by the host's cores. Pageable output: a byte pass's rows
  // all travel as bytes; a deeper pass writes u32 rows to HBM staging,
  // copied afterwards. Page-locked output: the link alone is about as fast
  // as link + widening, which share the host's memory bandwidth, so a pass
  // splits its rows -- the first split_frac written as u32 straight over the
  // link while the host widens the rest, which travel as bytes. Without room
  // for the byte rows the call keeps u32 rows throughout.
  const bool use_bytes = eng->narrow && !cta && (!zc || eng->split_frac < 1.0);
  // u32 rows copied into pageable memory: fresh pages are made present while
  // the traversal runs (byte rows' widening faults them in by itself). Road
  // 339x338 into fresh memory: S=256 (117 MB) 5.27 -> 4.43 ms, S=16 (7 MB)
  // 0.68 -> 0.70.
  constexpr size_t PREFAULT_FROM = size_t(32) << 20;
  const size_t out_bytes = S * V * sizeof(uint32_t);
  if (!use_bytes && !zc && out_bytes >= PREFAULT_FROM && is_pageable(out))
    prefault(eng->pool, out, out_bytes);
  if (use_bytes && grow(eng, &eng->d_dist8, &eng->d_dist8_cap, S * V) == MSBFS_OK) {
    uint32_t* wide = zc;
    if (!wide) {
      if ((rc = grow(eng, &eng->d_dist, &eng->d_dist_cap, S * V))) return rc;
      wide = eng->d_dist;
    }
    if ((rc = enqueue_call(eng, method, g, sources, S, wide, nullptr, nullptr, nullptr, nullptr,
                           eng->d_dist8, zc ? eng->split_frac : 0.0)))
      return rc;
    const size_t PW = (size_t)eng->last.words_per_vertex * 32;
    if (eng->last_split) {
      // Each pass's bytes are widened as soon as they exist, while the GPU
      // writes its u32 rows and runs later passes.
      for (size_t ps = 0; ps < eng->last_passes; ++ps) {
        CK(cudaEventSynchronize(eng->split_events[ps]));
        if (!eng->h_ctl[ps].narrow) continue;
        const size_t s0 = ps * PW, np = std::min(PW, S - s0), r0 = eng->split_rows[ps];
        if ((rc = widen_to_host(eng, eng->d_dist8 + (s0 + r0) * V, out + (s0 + r0) * V,
                                (np - r0) * V)))
          return rc;
      }
      return finish_call(eng, stats);
    }
    if ((rc = finish_call(eng, stats))) return rc;
    for (size_t ps = 0; ps < eng->last_passes; ++ps) {
      const size_t s0 = ps * PW, np = std::min(PW, S - s0);
      if (eng->h_ctl[ps].narrow) {
        if ((rc = widen_to_host(eng, eng->d_dist8 + s0 * V, out + s0 * V, np * V))) return rc;
      } else if (!zc) {
        CK(cudaMemcpy(out + s0 * V, eng->d_dist + s0 * V, np * V * sizeof(uint32_t),
                      cudaMemcpyDeviceToHost));
      }
    }
    return MSBFS_OK;
  }
  if (zc) {
    if ((rc = enqueue_call(eng, method, g, sources, S, zc, nullptr, nullptr, nullptr)))
      return rc;
    return finish_call(eng, stats);
  }
  const size_t total = S * V;
  if ((rc = grow(eng, &eng->d_dist, &eng->d_dist_cap, total))) return rc;
  if ((rc = enqueue_call(eng, method, g, sources, S, eng->d_dist, nullptr, out, nullptr)))
    return rc;
  return finish_call(eng, stats);
}

}  // namespace

// ===================================================================== C ABI

extern "C" {

int msbfs_engine_create(int device, int method, msbfs_engine** out) {
  if (!out) return MSBFS_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (method < 0 || method > MSBFS_METHOD_AUTO) return MSBFS_ERR_INVALID_ARGUMENT;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    return MSBFS_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= n) return MSBFS_ERR_NO_DEVICE;
  auto eng = std::make_unique<msbfs_engine>();
  eng->device = device;
  eng->method = method;
  msbfs_engine* e = eng.get();
  if (cudaSetDevice(device) != cudaSuccess) return MSBFS_ERR_CUDA;
  cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (cudaStreamCreateWithFlags(&e->own_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&e->copy_stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&e->ev_start) != cudaSuccess || cudaEventCreate(&e->ev_stop) != cudaSuccess ||
      cudaEventCreateWithFlags(&e->ev_pass, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&e->ev_copies, cudaEventDisableTiming) != cudaSuccess ||
      cudaMalloc((void**)&e->d_work, sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc((void**)&e->d_counter, sizeof(unsigned long long)) != cudaSuccess)
    return MSBFS_ERR_CUDA;
  e->stream = e->own_stream;
  const char* hl = getenv("MSBFS_HOST_LOOP");
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  e->host_loop = !coop || (hl && hl[0] == '1');
  const char* tb = getenv("MSBFS_TRAVERSE_BLOCKS");
  if (tb) e->traverse_blocks = (uint32_t)std::max(0, atoi(tb));
  const char* bs = getenv("MSBFS_BARRIER_SPINS");
  if (bs) e->barrier_spins = (uint32_t)std::max(1, atoi(bs));
  const char* zc = getenv("MSBFS_ZERO_COPY");
  e->zero_copy = !(zc && zc[0] == '0');
  const char* nr = getenv("MSBFS_NARROW");
  e->narrow = !(nr && nr[0] == '0');
  const char* mw = getenv("MSBFS_MAT_WAVES");
  if (mw) e->mat_waves = (uint32_t)std::max(0, atoi(mw));
  const char* sr = getenv("MSBFS_SPLIT_ROWS");
  if (sr) e->split_frac = std::min(1.0, std::max(0.0, atof(sr)));
  *out = eng.release();
  return MSBFS_OK;
}

void msbfs_engine_destroy(msbfs_engine* e) {
  if (!e) return;
  cudaSetDevice(e->device);
  cudaStreamSynchronize(e->stream);
  cudaStreamSynchronize(e->copy_stream);
  e->ws.clear();
  cudaFree(e->d_sources);
  cudaFree(e->d_dist);
  cudaFree(e->d_dist8);
  if (e->h_dist8) cudaFreeHost(e->h_dist8);
  for (cudaEvent_t ev : e->chunk_events) cudaEventDestroy(ev);
  for (cudaEvent_t ev : e->split_events) cudaEventDestroy(ev);
  cudaFree(e->d_reach);
  cudaFree(e->d_cta_queue);
  cudaFree(e->d_cta_bits);
  cudaFree(e->d_work);
  cudaFree(e->d_counter);
  cudaFree(e->d_sstats);
  if (e->h_log) cudaFreeHost(e->h_log);
  if (e->h_stuck) cudaFreeHost(e->h_stuck);
  for (cudaEvent_t ev : e->lvl_events) cudaEventDestroy(ev);
  cudaEventDestroy(e->ev_start);
  cudaEventDestroy(e->ev_stop);
  cudaEventDestroy(e->ev_pass);
  cudaEventDestroy(e->ev_copies);
  cudaStreamDestroy(e->own_stream);
  cudaStreamDestroy(e->copy_stream);
  delete e;
}

int msbfs_engine_method(const msbfs_engine* e) { return e ? e->method : -1; }

const char* msbfs_engine_last_error(const msbfs_engine* e) {
  return e ? e->last_error.c_str() : "null engine";
}

int msbfs_engine_set_stream(msbfs_engine* e, void* s) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  e->stream = s ? (cudaStream_t)s : e->own_stream;
  return MSBFS_OK;
}

int msbfs_engine_set_tuning(msbfs_engine* e, uint32_t max_words, uint32_t alpha, uint32_t beta) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  if (max_words) {
    if (max_words > 64 || (max_words & (max_words - 1)))
      return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "max_words_per_pass must be a power of two <= 64");
    e->max_words = max_words;
  }
  if (alpha) e->alpha = alpha;
  if (beta) e->beta = beta;
  cudaSetDevice(e->device);
  cudaStreamSynchronize(e->stream);
  e->ws.clear();  // thresholds are baked into the workspaces
  return MSBFS_OK;
}

int msbfs_engine_set_sm_share(msbfs_engine* e, uint32_t percent) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  if (percent < 1 || percent > 100)
    return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "sm share must be 1..100 percent");
  std::lock_guard<std::mutex> lk(e->mu);
  e->sm_share = percent;
  cudaSetDevice(e->device);
  cudaStreamSynchronize(e->stream);
  e->ws.clear();  // grid sizes are baked into the workspaces
  return MSBFS_OK;
}

int msbfs_engine_set_level_cap(msbfs_engine* e, uint32_t max_levels) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  e->level_cap = max_levels;
  cudaSetDevice(e->device);
  cudaStreamSynchronize(e->stream);
  e->ws.clear();  // the cap is baked into the workspaces
  return MSBFS_OK;
}

int msbfs_engine_set_profiling(msbfs_engine* e, int level) {
  if (!e || level < 0 || level > 3) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  auto counting = [](int l) { return l == 1 || l == 2; };
  if (counting(e->profiling) != counting(level)) {
    // The workspaces hold the counting or the production level kernels.
    cudaSetDevice(e->device);
    cudaStreamSynchronize(e->stream);
    e->ws.clear();
  }
  e->profiling = level;
  return MSBFS_OK;
}

int msbfs_engine_level_log(const msbfs_engine* e, msbfs_level_record* out, size_t cap,
                           size_t* count) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  const size_t n = e->log.size();
  if (count) *count = n;
  if (out) std::memcpy(out, e->log.data(), std::min(cap, n) * sizeof(msbfs_level_record));
  return MSBFS_OK;
}

int msbfs_select_auto_method(size_t V, size_t E, const uint32_t* off, size_t S) {
  msbfs_graph g;
  g.V = V;
  g.E = E;
  g.max_deg = (V && off) ? msbfs::max_degree(V, off) : 0;
  return resolve_method(&g, MSBFS_METHOD_AUTO, S);
}

int msbfs_graph_create(msbfs_engine* e, size_t V, size_t E, const uint32_t* off,
                       const uint32_t* idx, msbfs_graph** out) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  return upload_graph(e, V, E, off, idx, out);
}

void msbfs_graph_destroy(msbfs_graph* g) { free_graph(g); }

}  // extern "C"

// Lets another engine of the same device run on `g` without a second upload
// (the served form's slots share one resident graph). Not part of the C ABI:
// destroying `g` drops the workspaces of every engine attached to it, so `g`
// must be destroyed before any of them.
int msbfs_graph_attach(msbfs_graph* g, msbfs_engine* e) {
  if (!g || !e || !g->eng) return MSBFS_ERR_INVALID_ARGUMENT;
  if (e->device != g->eng->device)
    return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "graph lives on another device");
  if (e != g->eng && std::find(g->users.begin(), g->users.end(), e) == g->users.end())
    g->users.push_back(e);
  return MSBFS_OK;
}

// The part of the device that a level-path traversal of S sources takes, in
// percent of the blocks resident on all of it; 0 when the engine's method sends
// the call to the CTA path. Not part of the C ABI.
uint32_t msbfs_engine_traversal_share(msbfs_engine* e, const msbfs_graph* g, size_t S) {
  std::lock_guard<std::mutex> lk(e->mu);
  if (method_path(resolve_method(g, e->method, S)) == MSBFS_PATH_CTA) return 0;
  uint32_t W = 1;
  while (W < 64 && (size_t)W * 32 < S) W <<= 1;
  LevelKernelInfo k{};
  if (!level_kernel_info(W, level_planes(g), e->num_sms, &k)) return 100;
  const int blocks = traversal_blocks(e, g, W, k.traverse_resident);
  return (uint32_t)((100ull * blocks + k.traverse_resident - 1) / k.traverse_resident);
}

// The served form's cap on the blocks of the engine's next traversals, in
// percent of those resident on the whole device, and whether its calls may have
// to find room beside other traversals. Not part of the C ABI.
void msbfs_engine_cap_traversal(msbfs_engine* e, uint32_t percent, bool beside) {
  std::lock_guard<std::mutex> lk(e->mu);
  e->traverse_cap = percent;
  e->narrow_reduce = beside;
}

extern "C" {

int msbfs_graph_info(const msbfs_graph* g, size_t* V, size_t* E, uint32_t* max_deg, int* sym) {
  if (!g) return MSBFS_ERR_INVALID_ARGUMENT;
  if (V) *V = g->V;
  if (E) *E = g->E;
  if (max_deg) *max_deg = g->max_deg;
  if (sym) *sym = g->sym ? 1 : 0;
  return MSBFS_OK;
}

int msbfs_run_ms_bfs(msbfs_engine* e, const msbfs_graph* g, const uint32_t* sources, size_t S,
                     uint32_t* out, msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  return run_host(e, e->method, g, sources, S, out, stats);
}

int msbfs_run_ms_bfs_with_method(msbfs_engine* e, int method, const msbfs_graph* g,
                                 const uint32_t* sources, size_t S, uint32_t* out,
                                 msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  if (method < 0 || method > MSBFS_METHOD_AUTO)
    return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "unknown method");
  std::lock_guard<std::mutex> lk(e->mu);
  return run_host(e, method, g, sources, S, out, stats);
}

int msbfs_run_ms_bfs_csr(msbfs_engine* e, size_t V, size_t E, const uint32_t* off,
                         const uint32_t* idx, const uint32_t* sources, size_t S, uint32_t* out,
                         msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  if (S == 0) {
    if (stats) *stats = msbfs_stats{};
    return MSBFS_OK;
  }
  msbfs_graph* g = nullptr;
  int rc;
  {
    std::lock_guard<std::mutex> lk(e->mu);
    rc = upload_graph(e, V, E, off, idx, &g);
    if (rc == MSBFS_OK) rc = run_host(e, e->method, g, sources, S, out, stats);
  }
  free_graph(g);
  return rc;
}

int msbfs_run_ms_bfs_device(msbfs_engine* e, int method, const msbfs_graph* g,
                            const uint32_t* sources, size_t S, uint32_t* out_device) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  if (method < 0 || method > MSBFS_METHOD_AUTO)
    return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "unknown method");
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  int rc = validate_call(e, g, sources, S);
  if (rc) return rc;
  e->last = msbfs_stats{};
  e->last_passes = 0;
  if (S == 0) {
    CK(cudaEventRecord(e->ev_start, e->stream));
    CK(cudaEventRecord(e->ev_stop, e->stream));
    return MSBFS_OK;
  }
  if (!out_device) return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "out is null");
  CK(cudaSetDevice(e->device));
  return enqueue_call(e, method, g, sources, S, out_device, nullptr, nullptr, nullptr);
}

static_assert(sizeof(SourceStats) == sizeof(msbfs_source_stats), "stats layout");

int msbfs_run_ms_bfs_stats_device(msbfs_engine* e, int method, const msbfs_graph* g,
                                  const uint32_t* sources, size_t S,
                                  msbfs_source_stats* stats_device) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  if (method < 0 || method > MSBFS_METHOD_AUTO)
    return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "unknown method");
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  int rc = validate_call(e, g, sources, S);
  if (rc) return rc;
  e->last = msbfs_stats{};
  e->last_passes = 0;
  if (S == 0) {
    CK(cudaEventRecord(e->ev_start, e->stream));
    CK(cudaEventRecord(e->ev_stop, e->stream));
    return MSBFS_OK;
  }
  if (!stats_device) return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "stats is null");
  CK(cudaSetDevice(e->device));
  return enqueue_call(e, method, g, sources, S, nullptr, nullptr, nullptr, nullptr,
                      reinterpret_cast<SourceStats*>(stats_device));
}

int msbfs_run_ms_bfs_stats(msbfs_engine* e, const msbfs_graph* g, const uint32_t* sources,
                           size_t S, msbfs_source_stats* out, msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  int rc = validate_call(e, g, sources, S);
  if (rc) return rc;
  if (stats) *stats = msbfs_stats{};
  if (S == 0) return MSBFS_OK;
  if (!out) return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "out is null");
  CK(cudaSetDevice(e->device));
  if ((rc = grow(e, &e->d_sstats, &e->d_sstats_cap, S))) return rc;
  if ((rc = enqueue_call(e, e->method, g, sources, S, nullptr, nullptr, nullptr, nullptr,
                         e->d_sstats)))
    return rc;
  CK(cudaMemcpyAsync(out, e->d_sstats, S * sizeof(SourceStats), cudaMemcpyDeviceToHost,
                     e->stream));
  CK(cudaEventRecord(e->ev_stop, e->stream));
  return finish_call(e, stats);
}

int msbfs_engine_synchronize(msbfs_engine* e, msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  return finish_call(e, stats);
}

int msbfs_run_reachability(msbfs_engine* e, const msbfs_graph* g, const uint32_t* sources,
                           size_t S, uint32_t* words, msbfs_stats* stats) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  int rc = validate_call(e, g, sources, S);
  if (rc) return rc;
  if (stats) *stats = msbfs_stats{};
  if (S == 0 || g->V == 0) return MSBFS_OK;
  if (!words) return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "words is null");
  CK(cudaSetDevice(e->device));
  const size_t wpv = (S + 31) / 32;
  if ((rc = grow(e, &e->d_reach, &e->d_reach_cap, g->V * wpv))) return rc;
  int method = e->method;
  if (resolve_method(g, method, S) == MSBFS_METHOD_WORKGROUP_PERSISTENT_BFS)
    method = MSBFS_METHOD_PUSH_PULL_ADAPTIVE;
  if ((rc = enqueue_call(e, method, g, sources, S, nullptr, e->d_reach, nullptr, words)))
    return rc;
  return finish_call(e, stats);
}

int msbfs_traversed_edges_device(msbfs_engine* e, const msbfs_graph* g, const uint32_t* dist,
                                 size_t S, uint64_t* out_edges) {
  if (!e || !g || !out_edges) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  *out_edges = 0;
  if (S == 0 || g->V == 0) return MSBFS_OK;
  CK(cudaSetDevice(e->device));
  launch_traversed_edges((uint32_t)g->V, g->off, dist, (uint32_t)S, e->d_counter, e->stream);
  CK(cudaGetLastError());
  unsigned long long h = 0;
  CK(cudaMemcpyAsync(&h, e->d_counter, sizeof h, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  *out_edges = h;
  return MSBFS_OK;
}

}  // extern "C"

// ============================================================ level autotuner

namespace {

// Settings of the level-synchronous path that the autotuner varies. Words and
// heavy are 0 where the default rules stand: these depend on the graph, and
// the words (like alpha, beta and bits_div) apply to every graph of the engine.
struct LevelSettings {
  uint32_t words, alpha, beta, split, bits_div, heavy;
  uint32_t& at(int i) {
    return i == 0 ? words : i == 1 ? alpha : i == 2 ? beta : i == 3 ? split : i == 4 ? bits_div
                                                                                  : heavy;
  }
  bool operator==(const LevelSettings& o) const {
    return words == o.words && alpha == o.alpha && beta == o.beta && split == o.split &&
           bits_div == o.bits_div && heavy == o.heavy;
  }
};

// The thresholds are baked into an engine's workspaces, so they
// are dropped; a new slice length rebuilds the graph's bottom-up
// tables (done only when no other engine runs on the graph).
int apply_settings(msbfs_engine* eng, msbfs_graph* g, const LevelSettings& s) {
  CK(cudaStreamSynchronize(eng->stream));
  CK(cudaStreamSynchronize(eng->copy_stream));
  eng->ws.clear();
  eng->max_words = s.words;
  eng->alpha = s.alpha;
  eng->beta = s.beta;
  eng->bits_div = s.bits_div;
  if (s.split != g->split || s.heavy != g->heavy)
    return build_bottom_up_tables(eng, g, s.split, s.heavy);
  return MSBFS_OK;
}

// Device time (CUDA events) of one per-source-statistics call: the smaller
// of two after a call that builds the workspace.
int time_stats_call(msbfs_engine* eng, msbfs_graph* g, const uint32_t* src, size_t S, int method,
                    double* ms) {
  int rc;
  if ((rc = grow(eng, &eng->d_sstats, &eng->d_sstats_cap, S))) return rc;
  double best = 1e30;
  for (int k = 0; k < 3; ++k) {
    if ((rc = enqueue_call(eng, method, g, src, S, nullptr, nullptr, nullptr, nullptr,
                           eng->d_sstats)))
      return rc;
    msbfs_stats st{};
    if ((rc = finish_call(eng, &st))) return rc;
    if (k > 0) best = std::min(best, st.gpu_ms);
  }
  *ms = best;
  return MSBFS_OK;
}

}  // namespace

extern "C" int msbfs_engine_autotune(msbfs_engine* e, msbfs_graph* g, const uint32_t* sources,
                                     size_t S, const char* cache_path, msbfs_tuning* out) {
  if (!e) return MSBFS_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(e->mu);
  msbfs_engine* eng = e;
  int rc = validate_call(e, g, sources, S);
  if (rc) return rc;
  if (S == 0 || g->V == 0) return set_err(e, MSBFS_ERR_INVALID_ARGUMENT, "autotune needs sources");
  CK(cudaSetDevice(e->device));
  size_t bucket = 1;
  while (bucket < S) bucket <<= 1;
  const std::string key =
      msbfs::graph_class(g->V, g->E, g->max_deg) + "/s" + std::to_string(bucket);
  msbfs_tuning t{};
  std::strncpy(t.class_name, key.c_str(), sizeof t.class_name - 1);
  LevelSettings best{e->max_words, e->alpha, e->beta, g->split, e->bits_div, g->heavy};
  const int method = resolve_method(g, e->method, S);
  const uint32_t mode = path_mode(method_path(method));
  // What the words and the in-degree of a setting come to for this call (a cap
  // above the words that the sources need makes no difference).
  uint32_t wmax = 1;
  while (wmax < (S + 31) / 32 && wmax < 64) wmax <<= 1;
  auto words_of = [&](const LevelSettings& s) {
    return s.words ? std::min(s.words, wmax) : choose_words(e, g, S, mode);
  };
  auto heavy_of = [&](const LevelSettings& s) {
    return s.heavy ? s.heavy : warp_scan_degree(e, g->h_coff);
  };
  auto report = [&](const LevelSettings& s) {
    t.max_words_per_pass = words_of(s);
    t.alpha = s.alpha;
    t.beta = s.beta;
    t.hub_split = s.split;
    t.bitmap_div = s.bits_div;
    t.warp_scan_degree = g->scan_degree;
    if (out) *out = t;
    return MSBFS_OK;
  };
  if (method_path(method) == MSBFS_PATH_CTA) return report(best);
  t.level_path = 1;
  const bool shared = !g->users.empty() || g->eng != e;  // other engines hold its tables
  // Cache: one line per class,
  // "class words alpha beta split bitmap_div warp_scan_degree ms".
  if (cache_path) {
    std::ifstream in(cache_path);
    std::string k;
    LevelSettings s{};
    double ms = 0;
    while (in >> k >> s.words >> s.alpha >> s.beta >> s.split >> s.bits_div >> s.heavy >> ms) {
      if (k != key) continue;
      if (shared) {
        s.split = g->split;
        s.heavy = g->heavy;
      }
      if ((rc = apply_settings(e, g, s))) return rc;
      t.from_cache = 1;
      t.ms = ms;
      return report(s);
    }
  }
  double best_ms = 0;
  if ((rc = time_stats_call(e, g, sources, S, method, &best_ms))) return rc;
  t.default_ms = best_ms;
  t.trials = 1;
  const std::vector<std::vector<uint32_t>> cands = {
      {std::max(1u, wmax / 4), std::max(1u, wmax / 2), wmax},  // words per vertex
      {4, 8, 14, 28, 56},                                      // alpha
      {6, 12, 24, 64, 256},                                    // beta
      {256, 512, 1024},                                        // slice length
      {16, 64, 256},                                           // bitmap divisor
      {8, 16, 32, 64}};                                        // warp-scan in-degree
  const uint32_t start_words = words_of(best);  // (while the engine holds these settings)
  // One setting at a time, each from the best found so far; a change is
  // kept only when it is at least 2% faster (timing noise).
  for (int i = 0; i < 6; ++i) {
    if ((i == 3 || i == 5) && shared) continue;
    const LevelSettings base = best;
    for (uint32_t c : cands[i]) {
      LevelSettings s = base;
      s.at(i) = c;
      if (s == base || (i == 0 && c == start_words) || (i == 5 && c == heavy_of(base))) continue;
      if ((rc = apply_settings(e, g, s))) return rc;
      double ms = 0;
      if ((rc = time_stats_call(e, g, sources, S, method, &ms))) return rc;
      ++t.trials;
      if (ms < best_ms * 0.98) {
        best_ms = ms;
        best = s;
      }
    }
  }
  if ((rc = apply_settings(e, g, best))) return rc;
  t.ms = best_ms;
  if (cache_path) {
    std::ofstream o(cache_path, std::ios::app);
    o << key << ' ' << best.words << ' ' << best.alpha << ' ' << best.beta << ' ' << best.split
      << ' ' << best.bits_div << ' ' << best.heavy << ' ' << best_ms << '\n';
  }
  return report(best);
}
