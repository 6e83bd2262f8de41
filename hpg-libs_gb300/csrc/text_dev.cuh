// text_dev.cuh -- comparing reads with the packed text: the device helpers of the
// kernels that finish one-row searches without rank steps (text_search.cu,
// block_search.cu).  A chain's symbols are counted in search order: symbol i is
// W[i] of a forward search, W[len-1-i] of a backward one, complemented on the '-' strand.
#pragma once

#include "fm_device.cuh"

namespace hpgbwt {

// 32 symbols of a 2-bit stream from symbol i on (i may be -31 or reach past the
// end by as much: the streams are padded), symbol i in the low bits.
__device__ __forceinline__ uint64_t load32(const uint64_t* s, int64_t i) {
  const uint64_t* w = s + (i >> 5);
  const uint32_t sh = ((uint32_t)i & 31u) << 1;
  return (__ldg(w) >> sh) | ((__ldg(w + 1) << 1) << (63u - sh));
}

// The 32 symbols in reverse order.
__device__ __forceinline__ uint64_t rev32(uint64_t x) {
  const uint64_t r = __brevll(x);
  return ((r & 0x5555555555555555ull) << 1) | ((r >> 1) & 0x5555555555555555ull);
}

__device__ __forceinline__ uint64_t comp_word(const DevIndex& X, uint32_t strand) {
  return strand ? 0x5555555555555555ull * X.comp_xor : 0ull;
}

// (the words below are selected, not branched on, so that a warp's strands and
// directions stay together)

// Symbols i .. i+31 of a chain (past the read's end: whatever the stream holds), symbol i in the low bits.
__device__ __forceinline__ uint64_t query32(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len,
                                            bool fwd, uint32_t strand, int i) {
  const uint64_t x = load32(packed, (int64_t)b0 + (fwd ? i : len - 32 - i));
  const uint64_t r = rev32(x);
  return (fwd ? x : r) ^ comp_word(X, strand);
}

// The text read leftwards from position P of physical direction d, from its m-th symbol on:
// T_d[P-1-m], T_d[P-2-m], ... (past the text's ends: padding).
__device__ __forceinline__ uint64_t text32(const DevIndex& X, uint32_t d, uint32_t P, int m) {
  const uint64_t x = load32(X.text, d ? (int64_t)X.top - P + m : (int64_t)P - 32 - m);
  const uint64_t r = rev32(x);
  return d ? x : r;
}

// How many of the symbols i .. i+want-1 of a chain agree with the text read
// leftwards from position P of physical direction d; want <= P.
__device__ __forceinline__ int agree(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len, bool fwd,
                                     uint32_t strand, uint32_t d, int i, uint32_t P, int want) {
  for (int m = 0; m < want; m += 32) {
    const uint64_t x = text32(X, d, P, m) ^ query32(X, packed, b0, len, fwd, strand, i + m);
    if (x) return min(want, m + ((__ffsll((long long)x) - 1) >> 1));
  }
  return want;
}

}  // namespace hpgbwt
