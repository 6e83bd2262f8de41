// search_core.cuh -- per-thread forms of the reference search loops, used by
// the plain kernels (one thread per read and strand).
//
//   exact_bwd / exact_fwd ....... BWExactSearchBackward/Forward (search/search.h:9-65)
//   vector_run .................. BWExactSearchVectorBackward/Forward (search/search.c:1407-1489)
//   search1_helper .............. BWSearch1VectorHelper (search/search.c:1491-1709)
//
// The helper keeps one mutable result cursor and appends copies of it, as the
// reference does, so the error fields of every hit (including the
// base/position quirk of search.c:1556) and the emission order match.
#pragma once

#include "fm_device.cuh"
#include "text_dev.cuh"

namespace hpgbwt {

// Packed hit metadata: dir | nm<<1 | kind<<2 | base<<4 | (uint16)err_pos<<16.
__host__ __device__ __forceinline__ uint32_t pack_meta(uint32_t dir, uint32_t nm, uint32_t kind, uint32_t base,
                                                       int32_t err_pos) {
  return (dir & 1u) | ((nm & 1u) << 1) | ((kind & 3u) << 2) | ((base & 0xFFu) << 4) |
         ((uint32_t)(uint16_t)(int16_t)err_pos << 16);
}

struct Cursor {
  uint32_t dir, nm, kind, base;
  int32_t err_pos;
  uint32_t k, l;
  __device__ __forceinline__ uint32_t meta() const {
    return nm ? pack_meta(dir, 1, kind, base, err_pos) : pack_meta(dir, 0, 0, 0, 0);
  }
};

#ifdef __CUDACC__

// Where the read's packed bases are, for searches that finish with the text on the
// device; packed null: rank steps only.
struct TextRead {
  const uint64_t* packed;
  uint64_t b0;
  int len;
  uint32_t strand;
};

// How far a one-row search at row k agrees with the text over `want` symbols from symbol i of
// its direction on (search order), and the row it has then.
__device__ __forceinline__ int text_run(const DevIndex& X, View v, const TextRead& r, bool fwd, int i, int want,
                                        uint32_t k, uint32_t& row) {
  const uint32_t P = load_row_word((v.d ? X.dir[1].sa : X.dir[0].sa) + k);
  const int m = agree(X, r.packed, r.b0, r.len, fwd, r.strand, v.d, i, P, (int)min((uint32_t)want, P));
  row = load_row_word((v.d ? X.dir[1].isa : X.dir[0].isa) + P - (uint32_t)m);
  return m;
}

// Continue a search over `want` bases from W[pos] on (dir -1 or +1); true if the interval
// survives.  One row that has matched on ends by the text.
__device__ __forceinline__ bool exact_run(const DevIndex& X, View v, const TextRead& r, const uint8_t* W, int pos, int dir,
                                          int want, uint32_t& k, uint32_t& l, uint32_t& sectors) {
  for (; want > 0; --want, pos += dir) {
    const bool one = k == l;
    sectors += ((k >> 6) == (l >> 6)) ? 1u : 2u;
    bw_step(X, v, W[pos], k, l);
    if (k > l) return false;
    if (one && want > 1 && r.packed) {
      const int i = dir > 0 ? pos + 1 : r.len - pos;
      uint32_t row;
      if (text_run(X, v, r, dir > 0, i, want - 1, k, row) != want - 1) return false;
      k = l = row;
      return true;
    }
  }
  return k <= l;
}

// Continue a backward search over W[pos..start]; true if the interval survives.
__device__ __forceinline__ bool exact_bwd(const DevIndex& X, View v, const TextRead& r, const uint8_t* W, int pos,
                                          int start, uint32_t& k, uint32_t& l, uint32_t& sectors) {
  return exact_run(X, v, r, W, pos, -1, pos - start + 1, k, l, sectors);
}

__device__ __forceinline__ bool exact_fwd(const DevIndex& X, View v, const TextRead& r, const uint8_t* W, int pos, int end,
                                          uint32_t& k, uint32_t& l, uint32_t& sectors) {
  return exact_run(X, v, r, W, pos, 1, end - pos + 1, k, l, sectors);
}

__device__ __forceinline__ int64_t isize(uint2 v) { return (int64_t)v.y - (int64_t)v.x; }

// A vector search: the interval of each step t (t + 1 symbols), of which the helper reads
// those of positions n/2 .. 0 of the backward search and n/2 - 1 .. n of the forward one
// (n = len - 1), an interval only where its size differs from the next one's.  So only that
// half is kept in memory, and no element after the search has failed (their size is -1
// always) nor, but for the last, of a run of one row that the text matched.
// Plain search of 262,144 reads of 100 bp, 100 Mbp: 1217 us a call with all elements of that
// half written and read, the kernel bound by them (1.9 GB); 909 so.
struct SearchVector {
  uint2* at;      // the element of read position j at at[j * stride]
  size_t stride;
  int len;
  bool fwd;
  int one_from;   // steps after it and before `last` have one row each
  int last;       // the last step before the search failed
  __device__ __forceinline__ uint2 operator[](int j) const {
    const int t = fwd ? j : len - 1 - j;
    if (t > last) return make_uint2(1, 0);
    if (t > one_from && t < last) return make_uint2(0, 0);
    return at[(size_t)j * stride];
  }
};

__device__ __forceinline__ SearchVector vector_run(const DevIndex& X, View v, const TextRead& r, const uint8_t* W,
                                                   int len, bool fwd, uint2* vec, size_t stride, uint32_t& sectors) {
  uint32_t k = 0, l = X.top;
  const int dir = fwd ? 1 : -1;
  const int half = (len - 1) / 2, keep = fwd ? half - 1 : len - 1 - half;  // first step whose element is kept
  int i = fwd ? 0 : len - 1, t = 0;
  const int L = r.packed ? (int)X.tmer_len : 0;
  if (L && len >= 2 * L + 2) {
    const uint64_t q = query32(X, r.packed, r.b0, len, fwd, r.strand, 0);
    const uint32_t c = __brev((uint32_t)q) >> (32 - 2 * L);
    const uint2 s = load_row_pair((v.d ? X.tmer[1] : X.tmer[0]) + (((c & 0x55555555u) << 1) | ((c >> 1) & 0x55555555u)));
    k = s.x;
    l = s.y;
    t = L;
    i += dir * L;
    if (L > keep) vec[(size_t)(i - dir) * stride] = s;  // (the shortest such read's forward search)
  }
  SearchVector out{vec, stride, len, fwd, len, 0};
  for (; t < len && k <= l; ++t, i += dir) {
    const bool one = k == l;
    sectors += ((k >> 6) == (l >> 6)) ? 1u : 2u;
    bw_step(X, v, W[i], k, l);
    if (k > l) break;
    if (t >= keep) vec[(size_t)i * stride] = make_uint2(k, l);
    if (one && t + 1 < len && r.packed) {
      uint32_t row;
      const int m = text_run(X, v, r, fwd, t + 1, len - t - 1, k, row);
      out.one_from = t;
      out.last = t + m;
      if (m && out.last >= keep) vec[(size_t)(i + dir * m) * stride] = make_uint2(row, row);
      return out;
    }
  }
  out.last = t - 1;
  return out;
}

// The helper for one strand.  `emit(cursor)` appends a hit and returns false
// when the list is full, which ends the helper (search/results.h:100-101).
// Returns true on overflow.
template <typename Emit>
__device__ bool search1_helper(const DevIndex& X, const TextRead& r, const uint8_t* W, int len, const SearchVector& vk,
                               const SearchVector& vki, View B, View F, Emit& emit, uint32_t& sectors) {
  const int start = 0, end = len - 1;
  const int n = end - start;
  int half = n / 2;
  Cursor c;
  c.dir = 0;
  c.nm = 0;
  c.kind = 0;
  c.base = 0;
  c.err_pos = 0;

  const uint2 v0 = vk[0];
  if (v0.x <= v0.y) {
    c.k = v0.x;
    c.l = v0.y;
    if (!emit(c)) return true;
  }
  c.nm = 1;
  c.kind = 0;
  c.base = 0xFF;
  c.err_pos = start;

  int64_t res = isize(v0), res_last;
  uint2 v = vk[1];
  res_last = res;
  res = isize(v);
  if (res != res_last) {
    c.k = v.x;
    c.l = v.y;
    c.kind = 1;  // DELETION
    c.base = 0xFF;
    c.err_pos = start;
    if (!emit(c)) return true;
    const uint32_t bw = W[start];
    for (uint32_t b = 0; b < 4; ++b) {
      uint32_t ka = v.x, la = v.y;
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, B, b, ka, la);
      if (ka > la) continue;
      if (b != bw) {
        c.k = ka;
        c.l = la;
        c.kind = 2;  // MISMATCH, err_pos kept
        c.base = b;
        if (!emit(c)) return true;
      }
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, B, bw, ka, la);
      if (ka <= la) {
        c.k = ka;
        c.l = la;
        c.kind = 3;  // stored as (kind 3, base INSERTION, position b) by search.c:1556
        c.base = 3;
        c.err_pos = (int32_t)b;
        if (!emit(c)) return true;
      }
    }
  }

  for (int i = start + 2, j = 2; j <= half; ++i, ++j) {
    res_last = res;
    v = vk[j];
    res = isize(v);
    if (res == res_last) continue;
    c.kind = 1;
    c.base = 0xFF;
    c.err_pos = i - 1;
    {
      uint32_t k = v.x, l = v.y;
      if (exact_bwd(X, B, r, W, i - 2, start, k, l, sectors)) {
        c.k = k;
        c.l = l;
        if (!emit(c)) return true;
      }
    }
    const uint32_t wi = W[i - 1];
    for (uint32_t b = 0; b < 4; ++b) {
      uint32_t ka = v.x, la = v.y;
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, B, b, ka, la);
      if (ka > la) continue;
      c.kind = 3;  // INSERTION, err_pos kept
      c.base = b;
      {
        uint32_t k = ka, l = la;
        if (exact_bwd(X, B, r, W, i - 1, start, k, l, sectors)) {
          c.k = k;
          c.l = l;
          if (!emit(c)) return true;
        }
      }
      if (b != wi) {
        c.kind = 2;  // MISMATCH
        uint32_t k = ka, l = la;
        if (exact_bwd(X, B, r, W, i - 2, start, k, l, sectors)) {
          c.k = k;
          c.l = l;
          if (!emit(c)) return true;
        }
      }
    }
  }

  half--;
  c.dir = 1;
  v = vki[n];
  res = isize(v);
  res_last = res;
  v = vki[n - 1];
  res = isize(v);
  if (res != res_last) {
    c.k = v.x;
    c.l = v.y;
    c.kind = 1;
    c.base = 0xFF;
    c.err_pos = end;
    if (!emit(c)) return true;
    const uint32_t bw = W[end];
    for (uint32_t b = 0; b < 4; ++b) {
      uint32_t ka = v.x, la = v.y;
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, F, b, ka, la);
      if (ka > la) continue;
      if (b != bw) {
        c.k = ka;
        c.l = la;
        c.kind = 2;
        c.base = b;
        if (!emit(c)) return true;
      }
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, F, bw, ka, la);
      if (ka <= la) {
        c.k = ka;
        c.l = la;
        c.kind = 3;
        c.base = b;
        if (!emit(c)) return true;
      }
    }
  }

  for (int i = end - 2, j = n - 2; j >= half; --i, --j) {
    res_last = res;
    v = vki[j];
    res = isize(v);
    if (res == res_last) continue;
    c.kind = 1;
    c.base = 0xFF;
    c.err_pos = i + 1;
    {
      uint32_t k = v.x, l = v.y;
      if (exact_fwd(X, F, r, W, i + 2, end, k, l, sectors)) {
        c.k = k;
        c.l = l;
        if (!emit(c)) return true;
      }
    }
    const uint32_t wi = W[i + 1];
    for (uint32_t b = 0; b < 4; ++b) {
      uint32_t ka = v.x, la = v.y;
      sectors += ((ka >> 6) == (la >> 6)) ? 1u : 2u;
      bw_step(X, F, b, ka, la);
      if (ka > la) continue;
      c.kind = 3;
      c.base = b;
      {
        uint32_t k = ka, l = la;
        if (exact_fwd(X, F, r, W, i + 1, end, k, l, sectors)) {
          c.k = k;
          c.l = l;
          if (!emit(c)) return true;
        }
      }
      if (b != wi) {
        c.kind = 2;
        uint32_t k = ka, l = la;
        if (exact_fwd(X, F, r, W, i + 2, end, k, l, sectors)) {
          c.k = k;
          c.l = l;
          if (!emit(c)) return true;
        }
      }
    }
  }
  return false;
}

#endif  // __CUDACC__

}  // namespace hpgbwt
