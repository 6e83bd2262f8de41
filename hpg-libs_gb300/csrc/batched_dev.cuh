// batched_dev.cuh -- device helpers shared by the batched search kernels
// (batched.cu: fused, split and lockstep forms; wave.cu: the warp-cooperative
// form): change-point encoding, order keys, chunked result slots.
#pragma once

#include <cooperative_groups.h>

#include "batched.cuh"
#include "chunk_slots.hpp"
#include "search_core.cuh"

namespace hpgbwt {
namespace bdev {

namespace cg = cooperative_groups;

// Change-point entry types.
enum : uint32_t { kCpBwd = 0, kCpFwd = 1, kBlk1 = 2, kBlkN = 3 };
// Sub-operations of an entry: 0 deletion, then per base b: 1+3b aux step,
// 2+3b insertion, 3+3b mismatch; 13 = finished.
constexpr uint32_t kSubEnd = 13;

// Order keys: section << 28 | t << 8 | slot, following the helper's emission
// order: exact hit, j=1 block, backward j ascending, j=n-1 block, forward j descending.
__device__ __forceinline__ uint32_t order_key(uint32_t section, uint32_t t, uint32_t slot) {
  return (section << 28) | (t << 8) | slot;
}

// Pool slots are reserved per lane in chunks (chunk_slots.hpp), so an emission normally
// waits on no atomic: the per-list arrival count is a fire-and-forget reduction and
// the list position is assigned later by the scatter kernel.

// sa1: of a one-row hit whose SA value is known, that value plus one.
__device__ __forceinline__ void write_hit(const BatchedParams& p, unsigned slot, uint32_t rs, uint32_t key,
                                          uint32_t k, uint32_t l, uint32_t meta, uint32_t sa1 = 0) {
  atomicAdd(&p.rs_count[rs], 1u);  // result unused: compiles to a reduction
  if (slot < p.res_cap) {
    PendingHit h;
    h.rs = rs;
    h.key = key;
    h.k = k;
    h.l = l;
    h.meta = meta;
    h.sa1 = sa1;
    p.res[slot] = h;
  } else {
    atomicOr(p.status, kStatusResFull);
  }
}

__device__ __forceinline__ void emit_hit(const BatchedParams& p, uint32_t rs, uint32_t key, uint32_t k, uint32_t l,
                                         uint32_t meta) {
  cg::coalesced_group g = cg::coalesced_threads();
  unsigned base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(p.res_total, (unsigned)g.size());
  base = g.shfl(base, 0) + g.thread_rank();
  write_hit(p, base, rs, key, k, l, meta);
}

__device__ __forceinline__ unsigned claim(unsigned int* ctr, unsigned n) {
  cg::coalesced_group g = cg::coalesced_threads();
  unsigned base = 0;
  if (g.thread_rank() == 0) base = atomicAdd(ctr, (unsigned)g.size() * n);
  return g.shfl(base, 0) + g.thread_rank() * n;
}

// Chunked slot of the result pool for the calling lane (c_res: its chunk), and the end of
// the lane's last chunk.
__device__ __forceinline__ unsigned res_slot(const BatchedParams& p, uint32_t& c_res) {
  return pool_slot(
      p.res_cap, c_res, [&](unsigned n) { return claim(p.res_total, n); },
      [&](uint32_t i) { p.res[i].rs = 0xFFFFFFFFu; });
}

__device__ __forceinline__ void res_leave(const BatchedParams& p, uint32_t c_res) {
  chunk_leave(p.res_cap, c_res, [&](uint32_t i) { p.res[i].rs = 0xFFFFFFFFu; });
}

// The same of the queue of change points.
__device__ __forceinline__ unsigned spill_slot(const BatchedParams& p, uint32_t& c_spill) {
  return pool_slot(
      p.spill_cap, c_spill, [&](unsigned n) { return claim(p.spill_tail, n); },
      [&](uint32_t i) { p.spill[i].rs = 0xFFFFFFFFu; });
}

__device__ __forceinline__ void spill_leave(const BatchedParams& p, uint32_t c_spill) {
  chunk_leave(p.spill_cap, c_spill, [&](uint32_t i) { p.spill[i].rs = 0xFFFFFFFFu; });
}

// Lane modes.
enum : uint32_t { kNone = 0, kChain = 1, kCont = 2, kSingle = 3, kKmer = 4 };

// Cold lane state lives in shared memory (one word per lane and field), so
// that the registers hold only what every step touches.
//   meta: J (16 bits) | entry type << 16 | sub-operation << 18 | block err_pos << 22 | in entry << 24
//   misc: stack depth (4 bits) | chains left in the claimed chunk << 4
__device__ __forceinline__ uint32_t meta_j(uint32_t m) { return m & 0xFFFFu; }
__device__ __forceinline__ uint32_t meta_type(uint32_t m) { return (m >> 16) & 3u; }
__device__ __forceinline__ uint32_t meta_sub(uint32_t m) { return (m >> 18) & 15u; }
__device__ __forceinline__ uint32_t meta_bpos(uint32_t m) { return (m >> 22) & 3u; }
__device__ __forceinline__ bool meta_in(uint32_t m) { return (m >> 24) & 1u; }
__device__ __forceinline__ uint32_t make_meta(uint32_t j, uint32_t type, uint32_t sub, uint32_t bpos, bool in) {
  return j | (type << 16) | (sub << 18) | (bpos << 22) | ((in ? 1u : 0u) << 24);
}


}  // namespace bdev
}  // namespace hpgbwt
