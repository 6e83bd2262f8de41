// chunk_slots.hpp -- slots of a shared array that lanes reserve a chunk at a time, so
// that an append normally waits on no atomic.  A lane's state is one word: its next
// slot | slots left << 28.  `claim(n)` advances the array's counter by n and returns
// where it stood; `empty(slot)` marks a slot that is counted but holds nothing.  A reader
// that takes the slots below min(counter, capacity) finds each one written or marked:
// whatever a claim counted and no lane writes is marked here.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define HPG_HD __host__ __device__ __forceinline__
#else
#define HPG_HD inline
#endif

namespace hpgbwt {

constexpr unsigned kResChunk = 8;                 // slots a claim reserves
constexpr uint32_t kChunkSlotMask = 0x0FFFFFFFu;  // of the state: the next slot

// The next slot of a bounded queue of cap < 2^28 entries, or cap where no whole chunk is
// left: the part of the refused chunk that lies below cap is marked.
template <typename Claim, typename Empty>
HPG_HD unsigned chunk_slot(uint32_t cap, uint32_t& state, Claim claim, Empty empty) {
  if ((state >> 28) == 0) {
    const unsigned c = claim(kResChunk);
    if (c + kResChunk > cap) {
      for (unsigned s = c; s < cap; ++s) empty(s);  // (fewer than a chunk)
      state = 0;
      return cap;
    }
    state = c | (kResChunk << 28);
  }
  const unsigned slot = state & kChunkSlotMask;
  state = (slot + 1) | (((state >> 28) - 1) << 28);
  return slot;
}

// The next slot of a pool of any size, which may be at or past cap (the caller's
// overflow).  A chunk that ends past what the state's word holds gives its first slot only.
template <typename Claim, typename Empty>
HPG_HD unsigned pool_slot(uint32_t cap, uint32_t& state, Claim claim, Empty empty) {
  if ((state >> 28) == 0) {
    const unsigned c = claim(kResChunk);
    if (c > kChunkSlotMask - kResChunk) {
      for (unsigned s = c + 1; s < c + kResChunk && s < cap; ++s) empty(s);
      state = 0;
      return c;
    }
    state = c | (kResChunk << 28);
  }
  const unsigned slot = state & kChunkSlotMask;
  state = (slot + 1) | (((state >> 28) - 1) << 28);
  return slot;
}

// Marks what is left of a lane's last chunk.
template <typename Empty>
HPG_HD void chunk_leave(uint32_t cap, uint32_t state, Empty empty) {
  const uint32_t slot = state & kChunkSlotMask, left = state >> 28;
  for (uint32_t i = 0; i < left; ++i)
    if (slot + i < cap) empty(slot + i);
}

}  // namespace hpgbwt
