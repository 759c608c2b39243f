// One level of a block's single-source BFS: frontier queue and expansion,
// shared by the CTA-per-source kernels and the batched form.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

namespace msbfs {

constexpr uint32_t CTA_FULL = 0xffffffffu;
enum : int { ER_NONE = 0, ER_PACKED = 1, ER_WIDE = 2 };
constexpr uint32_t ER_WIDE_ID = 0x0fffffffu;  // the target's bits of a wide record

// Frontier entries. ER_PACKED: the graph carries edge records, 8 bytes per edge
// {target, target's edge range packed as begin << 4 | count} (built once per
// road-like graph: at most 8 out-edges, fewer than 2^28 edges), and a queue
// entry is the packed edge range of a frontier vertex instead of its id.
// Expanding a vertex then costs one dependent L2 round trip per level (its
// edge records) instead of three (queue entry, offsets, adjacency): on a
// ~4,000-level road graph the per-level latency chain is what a traversal's
// time is made of.
// ER_WIDE, for 2^28 edges and more (and at most 2^28 vertices): the records are
// {target | its count << 28, target's edge begin}, and a queue entry is the
// position of the record by which a vertex was found, which its expansion reads
// again (from the L1, as a rule); the source, without one, is an id. 8200 x 8200
// grid, S=1 / 32, ms: ids 576 / 1,731, these records 489 / 1,465.
//
// Queue: the first `qh` entries of a level's frontier sit in shared memory
// (two halves, by level parity), the rest in one global slab of V words per
// block. The frontiers of consecutive levels are disjoint vertex sets, so
// |F_L| + |F_L+1| <= V: in the slab even levels sit at the front and odd
// levels at the back.
// Shared-memory accesses by 32-bit address: through generic pointers (a queue
// entry may also sit in the slab) each would pay the generic path's latency.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t r;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(a) : "memory");
  return r;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t x) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ uint32_t atoms_or(uint32_t a, uint32_t x) {
  uint32_t r;
  asm volatile("atom.shared.or.b32 %0, [%1], %2;" : "=r"(r) : "r"(a), "r"(x) : "memory");
  return r;
}
__device__ __forceinline__ uint32_t atoms_add(uint32_t a, uint32_t x) {
  uint32_t r;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(r) : "r"(a), "r"(x) : "memory");
  return r;
}

template <int ER>
struct CtaQueue {
  uint32_t sq;     // shared-memory address of the halves
  uint32_t* slab;  // global memory
  uint32_t qh, V;
  const uint32_t* off;
  __device__ __forceinline__ uint32_t* slab_at(uint32_t lv, uint32_t i) const {
    return (lv & 1) ? slab + (V - 1 - i) : slab + i;
  }
  __device__ __forceinline__ uint32_t half(uint32_t lv) const {
    return sq + ((lv & 1) ? 4 * qh : 0);
  }
  // The frontier of level 0 (the halves may hold nothing: qh == 0).
  __device__ __forceinline__ void put_source(uint32_t u) const {
    uint32_t x = u;
    if constexpr (ER == ER_PACKED) {
      const uint32_t b = __ldg(off + u);
      x = b << 4 | (__ldg(off + u + 1) - b);
    }
    if (qh)
      sts32(sq, x);
    else
      slab[0] = x;
  }
};

// Marks the targets v[k] (where fresh[k]) of one batch of edges per lane and
// appends the new ones, entries nx[k], to the frontier of level `nd`.
// `mark(v, bit)` sets v's visited bit and returns the bitmap word as it was
// (testing the bit first only adds a step: road 339x338 S=2,048 3.25 -> 3.08
// ms without it). New vertices get their places with one shared-memory
// atomicAdd per warp (ballot prefix sums).
template <int ER, int BATCH, typename Mark>
__device__ __forceinline__ void cta_discover(const CtaQueue<ER>& q, uint32_t nd, uint32_t cnt,
                                             uint32_t* row, const uint32_t* v, const uint32_t* nx,
                                             bool* fresh, Mark&& mark) {
  uint32_t was[BATCH];
#pragma unroll
  for (int k = 0; k < BATCH; ++k) {
    was[k] = 0;
    if (fresh[k]) was[k] = mark(v[k], __funnelshift_l(0u, 1u, v[k]));
  }
  uint32_t total, before;  // of the warp, of the lower lanes
  uint32_t lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
#pragma unroll
  for (int k = 0; k < BATCH; ++k)
    fresh[k] = fresh[k] && !(was[k] & __funnelshift_l(0u, 1u, v[k]));
  if constexpr (BATCH == 1) {
    const uint32_t b0 = __ballot_sync(CTA_FULL, fresh[0]);
    total = __popc(b0);
    before = __popc(b0 & lt);
  } else {
    static_assert(BATCH <= 7, "counts of three bits");
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < BATCH; ++k) c += fresh[k] ? 1u : 0u;
    const uint32_t b0 = __ballot_sync(CTA_FULL, c & 1u), b1 = __ballot_sync(CTA_FULL, c & 2u);
    total = __popc(b0) + 2 * __popc(b1);
    before = __popc(b0 & lt) + 2 * __popc(b1 & lt);
    if constexpr (BATCH >= 4) {
      const uint32_t b2 = __ballot_sync(CTA_FULL, c & 4u);
      total += 4 * __popc(b2);
      before += 4 * __popc(b2 & lt);
    }
  }
  if (total) {
    const uint32_t hout = q.half(nd);
    uint32_t pos = 0;
    if ((threadIdx.x & 31) == 0) pos = atoms_add(cnt, total);
    pos = __shfl_sync(CTA_FULL, pos, 0) + before;
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      if (!fresh[k]) continue;
      if (row) row[v[k]] = nd;
      if (pos < q.qh)
        sts32(hout + 4 * pos, nx[k]);
      else
        *q.slab_at(nd, pos) = nx[k];
      ++pos;
    }
  }
}

// No vertex is set aside.
struct CtaNoBig {
  __device__ __forceinline__ bool operator()(uint32_t, uint32_t) const { return false; }
};

// Expands the n_in frontier entries of `level`: LPV lanes take one vertex,
// each BATCH of its edges per round. Each step of a round -- edge records,
// bitmap atomics, queue places -- is issued for all edges before the next
// step needs a result, so a level is one pass through that latency chain, not
// one pass per edge. A level with few vertices is bound by the length of this
// instruction sequence (about 6 cycles an instruction with one warp per
// scheduler), hence the straight-line common case: queue entries read without
// a per-lane branch while the frontier fits the shared-memory half (its length
// is a multiple of 32, so a warp's entries past n_in are still inside it).
// `big(e, n)` may take a vertex's edges [e, e + n) over (called by its first
// lane): they are then left out here.
template <int ER, int THREADS, int LPV, int BATCH, typename Mark, typename Big = CtaNoBig>
__device__ __forceinline__ void cta_expand(const uint2* erec, const uint32_t* idx,
                                           const CtaQueue<ER>& q, uint32_t level, uint32_t n_in,
                                           uint32_t cnt, uint32_t* row, Mark&& mark,
                                           Big&& big = Big{}) {
  constexpr bool HAS_BIG = !std::is_same<std::remove_reference_t<Big>, CtaNoBig>::value;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t sub = lane % LPV;
  const uint32_t nd = level + 1;
  const uint32_t hin = q.half(level);
  for (uint32_t base = (threadIdx.x - lane) / LPV; base < n_in; base += THREADS / LPV) {
    const uint32_t i = base + lane / LPV;
    uint32_t x = 0, e = 0, n = 0;
    if (n_in <= q.qh) {
      x = lds32(hin + 4 * i);
    } else if (i < n_in) {
      if (i < q.qh)
        x = lds32(hin + 4 * i);
      else
        x = *q.slab_at(level, i);
    }
    if constexpr (ER == ER_PACKED) {
      e = x >> 4;
      n = i < n_in ? x & 15u : 0u;
    } else if (i < n_in) {
      if (ER == ER_WIDE && level) {
        const uint2 r = __ldg(erec + x);
        e = r.y;
        n = r.x / (ER_WIDE_ID + 1);
      } else {
        e = __ldg(q.off + x);
        n = __ldg(q.off + x + 1) - e;
      }
    }
    if constexpr (HAS_BIG) {
      bool taken = false;
      if (sub == 0) taken = big(e, n);
      if (__shfl_sync(CTA_FULL, taken, lane - sub)) n = 0;
    }
    for (;;) {
      uint32_t v[BATCH], nx[BATCH];
      bool fresh[BATCH];
#pragma unroll
      for (int k = 0; k < BATCH; ++k) {
        v[k] = nx[k] = 0;
        fresh[k] = sub + k * LPV < n;
        if (fresh[k]) {
          if constexpr (ER == ER_PACKED) {
            const uint2 r = __ldg(erec + e + sub + k * LPV);
            v[k] = r.x;
            nx[k] = r.y;
          } else if constexpr (ER == ER_WIDE) {
            nx[k] = e + sub + k * LPV;
            v[k] = __ldg(erec + nx[k]).x & ER_WIDE_ID;
          } else {
            v[k] = nx[k] = __ldg(idx + e + sub + k * LPV);
          }
        }
      }
      cta_discover<ER, BATCH>(q, nd, cnt, row, v, nx, fresh, mark);
      if (!__any_sync(CTA_FULL, n > LPV * BATCH)) break;
      e += LPV * BATCH;
      n -= min(n, (uint32_t)(LPV * BATCH));
    }
  }
}

// Long edge lists of a level, set aside in pieces for whole warps, so that no
// few lanes walk a hub's edges alone.
constexpr uint32_t BIG_DEGREE = 128, BIG_PIECE = 1024, BIG_PIECES = 1024;
constexpr size_t BIG_BYTES = BIG_PIECES * 2 * sizeof(uint32_t);

// One level of a block's traversal, up to the barrier after which the next
// frontier's size, counted at shared address `cnt`, can be read. Graphs without
// edge records keep lists of more than BIG_DEGREE edges for a second sweep
// (sbig: shared address of BIG_BYTES, 0 for none; spieces: of two counters, by
// level parity, both 0 before level 0).
template <int ER, int THREADS, int LPV, typename Mark>
__device__ __forceinline__ void cta_level(const uint2* erec, const uint32_t* idx,
                                          const CtaQueue<ER>& q, uint32_t level, uint32_t n_in,
                                          uint32_t cnt, uint32_t* row, Mark&& mark, uint32_t sbig,
                                          uint32_t spieces) {
  if constexpr (ER != ER_NONE) {
    cta_expand<ER, THREADS, LPV, 4 / LPV>(erec, idx, q, level, n_in, cnt, row, mark);
    __syncthreads();
  } else {
    const uint32_t snbig = spieces + (level & 1) * 4;
    // The other parity's counter was last read before this level began.
    if (threadIdx.x == 0) sts32(spieces + (~level & 1) * 4, 0);
    cta_expand<ER, THREADS, LPV, 4 / LPV>(
        erec, idx, q, level, n_in, cnt, row, mark, [&](uint32_t e, uint32_t d) {
          if (d <= BIG_DEGREE || !sbig) return false;
          const uint32_t pieces = (d + BIG_PIECE - 1) / BIG_PIECE;
          const uint32_t at = atoms_add(snbig, pieces);
          const bool fits = at + pieces <= BIG_PIECES;
          for (uint32_t k = 0; k < pieces && at + k < BIG_PIECES; ++k) {
            sts32(sbig + 8 * (at + k), e + k * BIG_PIECE);
            sts32(sbig + 8 * (at + k) + 4, fits ? min(BIG_PIECE, d - k * BIG_PIECE) : 0u);
          }
          return fits;
        });
    __syncthreads();
    const uint32_t nbig = min(lds32(snbig), BIG_PIECES);
    if (nbig) {
      for (uint32_t b = threadIdx.x / 32; b < nbig; b += THREADS / 32) {
        const uint32_t e = lds32(sbig + 8 * b), len = lds32(sbig + 8 * b + 4);
        for (uint32_t j0 = 0; j0 < len; j0 += 128) {
          const uint32_t j = j0 + (threadIdx.x & 31);
          uint32_t v[4];
          bool fresh[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            fresh[k] = j + 32 * k < len;
            v[k] = fresh[k] ? __ldg(idx + e + j + 32 * k) : 0u;
          }
          cta_discover<ER, 4>(q, level + 1, cnt, row, v, v, fresh, mark);
        }
      }
      __syncthreads();
    }
  }
}

}  // namespace msbfs
