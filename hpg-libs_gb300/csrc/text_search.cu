// text_search.cu -- the batched BWSearch1 search (the vector searches of
// bwt.c:1940-1950 and the 1-error helper's branches, search/search.c:1491-1709)
// with the text, the suffix array and its inverse on the device (full_rows.cu).
//
// A vector search ("chain") of a read that occurs in the text narrows to one
// row after about log4(n) steps (13 to 16) and stays there for the rest of the
// read.  Rank steps from there on are dependent random sectors, one a base;
// the same facts are in the text: the row's SA value says where the match
// lies, the read agrees with the text up to a base that one comparison of
// packed words finds, and the row of the interval reached is the inverse SA of
// the position reached.  The helper's eight continuations of a change point
// whose interval is one row are comparisons too, and only three of them can
// match: the deletion, and insertion and mismatch of the one base the text has.
//
// Launches:
//   text_head_kernel    a thread per chain: start table, then rank steps until
//                       the interval is empty or has stayed one row for a step
//                       (its SA value, as an alignment, to `diag`), or is still
//                       several rows where the helper branches (up to 32: row queue)
//                       or after kHeadSteps steps (up to 4: row queue); else rest list
//   text_read_kernel    a thread per read: its one-row chains compared with the
//                       text, hits
//   text_wide_kernel    persistent warps: the wider chains until they are not (-> row
//                       queue), one rank step per lane and iteration; their change
//                       points that can have hits queued
//   text_branch_kernel  persistent warps: the queued change points' continuations,
//                       one rank step per lane and iteration; walks that narrow
//                       to one row -> walk queue
//   text_rows_kernel    a lane per row of the queued chains, all their change
//                       points from one comparison of each row's text
//   text_walk_kernel    a thread per queued walk
//   text_block_kernel   a thread per j = 1 / j = n-1 block
//
// Positions are counted in search order: symbol i of a chain is W[len-1-i]
// (backward) or W[i] (forward), complemented on the '-' strand, so both
// directions and strands run the same code; J of the helper is len - t
// (backward) or t - 1 (forward) for an interval of t matched symbols, and its
// order key's t field is len - t in both.
//
// Bound by random sectors, as rank walks are, but about 20 a read of 100 bp at 100
// Mbp against 180, and by the latency of some 8 dependent accesses a chain, whatever
// the read's length.  Search stage, rank walks (wave.cu) -> here:
//   2M x 100 bp, 100 Mbp                          3704 ->  700 us
//   4M x 36-250 bp, 100 Mbp                      12570 -> 1610 us
//   1000 x 50-300 bp, 100 Mbp                      510 ->   80 us
//   2M x 150 bp, 600 Mbp with 45 % repeats        9809 -> 2760 us
// Indexes without the arrays, and batches above kTextMaxReads (the queues'
// counters), take the warp-cooperative form.
#include <cuda_runtime.h>

#include <algorithm>

#include "batched.cuh"
#include "batched_dev.cuh"
#include "kernels.cuh"
#include "text_dev.cuh"

namespace hpgbwt {

namespace {

using namespace bdev;

constexpr int kHeadTpb = 256, kReadTpb = 256, kWalkTpb = 256, kWideTpb = 128, kRowsTpb = 128;
constexpr int kRowsWarps = kRowsTpb / 32;
// Rank steps of a head past its start table: nearly all chains are empty or one row
// by then (search stage at 4 / 5 / 6 / 8 steps, 2M x 100 bp, 100 Mbp: 899 / 884 / 891 /
// 901 us; the lanes of the others, some in most warps, would hold their warps longer).
constexpr int kHeadSteps = 6;
// Rows of a chain in the row queue at most.  Where the helper does not branch yet a wide
// chain steps on down to kRowsBefore (2M x 150 bp, 600 Mbp: 4660 us a call at 32, 4560 at
// 16, 4500 at 8, 4470 at 4, 4450 at 2): a step is two sectors for all its rows, a row in the
// queue two to three.  Within the branching window every step may queue a change point, and
// all 32 are taken.
constexpr uint32_t kRows = 32, kRowsBefore = 4;
// Claims of a warp of the wide and the branch kernel, at least about, where the queues are
// short (2M x 150 bp, 600 Mbp, a call: 3966 us at 1, 3938 at 4, 3888 at 16, 4585 at 64, where
// a claim fills half a warp).
constexpr uint32_t kClaims = 16;
// A chain's entry of `diag` that is no alignment: its first symbols (kHeadSteps past the
// table at most) do not occur, or it was left to the row queue or the rest list.
constexpr uint32_t kAbsent = 0xFFFFFFFFu, kMany = 0xFFFFFFFEu;
__device__ __forceinline__ bool is_diag(uint32_t x) { return x < kMany; }
constexpr unsigned kFull = 0xFFFFFFFFu;

// First t at which the helper branches: J <= n/2 backward, J >= n/2 - 1 forward (n = len - 1).
__device__ __forceinline__ int branch_from(int len, bool fwd) {
  const int half = (len - 1) / 2;
  return fwd ? half : len - half;
}

// What the head found of the strand's chain on the other index (an entry of `diag`),
// which reads the symbols from t on from their other end; kMany where they do not
// reach past its head.
__device__ __forceinline__ uint32_t other_chain(const DevIndex& X, const BatchedParams& p, uint32_t rs, uint32_t d,
                                                int len, int t) {
  if (len - t < (int)X.tmer_len + kHeadSteps || len < 2 * (int)X.tmer_len + 2) return kMany;
  return p.diag[(uint64_t)((d ^ 1u) * 2u + (rs & 1u)) * p.n_reads + (rs >> 1)];
}

// An entry of the block list (j = 1 / j = n-1).
__device__ __forceinline__ void push_block(const BatchedParams& p, uint32_t k, uint32_t l, uint32_t rs, int len,
                                           bool fwd) {
  const unsigned q = atomicAdd(p.block_n, 1u);
  const uint32_t jt = fwd ? (uint32_t)(len - 2) | (kBlkN << 16) : 1u | (kBlk1 << 16);
  if (q < p.block_cap) p.blocks[q] = SpillEntry{k, l, rs, jt};
  else atomicOr(p.status, kStatusSpillFull);
}

__device__ __forceinline__ uint32_t branch_meta(bool fwd, int len, int t, uint32_t kind, uint32_t base) {
  return pack_meta(fwd ? 1u : 0u, 1, kind, base, fwd ? t : len - t - 1);
}

// Entries of the row queue and the rest list: x = k, y = l, z = rs, w = symbols matched |
// forward << 16; of the walk queue: x = row, y = order key, z = rs, w the same.

// blockIdx.y 0, 1: the chains on the backward index ('+' backward, '-' forward),
// 2, 3: those on the forward index ('+' forward, '-' backward), so that the
// blocks in flight read one direction's table and blocks at a time.
template <bool CENSUS>
__global__ void __launch_bounds__(kHeadTpb, 7) text_head_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[2][kHeadTpb / 32], s_base[2];
  const uint32_t n_reads = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  if ((uint64_t)blockIdx.x * kHeadTpb >= n_reads) return;
  const uint32_t read = blockIdx.x * kHeadTpb + threadIdx.x;
  const uint32_t d = blockIdx.y >> 1, strand = blockIdx.y & 1u;
  const bool fwd = (d ^ strand) != 0;
  uint32_t dest = 0, sectors = 0;  // 1: row queue, 2: rest list
  uint32_t diag = kAbsent;
  uint4 e = make_uint4(0, 0, 0, 0);
  if (read < n_reads && p.ok[read]) {
    const uint64_t b0 = p.offs[read], b1 = p.offs[read + 1];
    if (b1 >= b0 + 3 && b1 - b0 <= 32767 && b1 <= p.packed_len) {
      const int len = (int)(b1 - b0);
      const OccBlock* occ = d ? X.dir[1].occ : X.dir[0].occ;
      const uint32_t dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
      uint64_t q = query32(X, p.packed, b0, len, fwd, strand, 0);
      uint32_t k = 0, l = X.top;
      int t = 0;
      // the first L steps from the full interval reach no branching position: one lookup
      const int L = (int)X.tmer_len;
      if (len >= 2 * L + 2) {
        const uint32_t r = __brev((uint32_t)q) >> (32 - 2 * L);
        const uint2 s = load_row_pair((d ? X.tmer[1] : X.tmer[0]) +
                                      (((r & 0x55555555u) << 1) | ((r >> 1) & 0x55555555u)));
        if (CENSUS) ++sectors;
        k = s.x;
        l = s.y;
        t = L;
        q >>= 2 * L;
      }
      const int ts = branch_from(len, fwd), stop = min(t + kHeadSteps, len - 1);
      bool one = false;
      while (k <= l) {
        if (t == stop) {
          one = k == l;
          dest = one ? 0 : (l - k < kRowsBefore ? 1 : 2);
          e = make_uint4(k, l, 0, (uint32_t)t);
          break;
        }
        const uint32_t pk = k, pl = l;
        if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
        rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
        if (t >= ts && l - k != pl - pk) {  // a change point: the interval before it
          one = pk == pl;
          dest = one ? 0 : (pl - pk < kRows ? 1 : 2);
          e = make_uint4(pk, pl, 0, (uint32_t)t);
          break;
        }
        ++t;
        q >>= 2;
        if (k == l && pk == pl) {  // one row that has matched on: not a chance match about to end
          one = true;
          e = make_uint4(k, l, 0, (uint32_t)t);
          break;
        }
      }
      if (one) {  // symbol i of the chain lies at T_d[diag - 1 - i]
        diag = load_row_word((d ? X.dir[1].sa : X.dir[0].sa) + e.x) + e.w;
        if (CENSUS) ++sectors;
      }
      if (dest) diag = kMany;
      e.z = (read << 1) | strand;
      e.w |= fwd ? 1u << 16 : 0u;
    }
  }
  if (read < n_reads) __stcs(p.diag + (uint64_t)blockIdx.y * p.n_reads + read, diag);
  // the block's entries appended with one atomic per queue
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!__syncthreads_or(dest)) {
    if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
    return;
  }
  const unsigned m1 = __ballot_sync(kFull, dest == 1), m2 = __ballot_sync(kFull, dest == 2);
  if (lane == 0) {
    s_cnt[0][warp] = (uint32_t)__popc(m1);
    s_cnt[1][warp] = (uint32_t)__popc(m2);
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t tot = 0;
    for (int w = 0; w < kHeadTpb / 32; ++w) {
      const uint32_t c = s_cnt[threadIdx.x][w];
      s_cnt[threadIdx.x][w] = tot;
      tot += c;
    }
    s_base[threadIdx.x] = tot ? atomicAdd(threadIdx.x ? p.rest_n : p.rows_n, tot) : 0u;
  }
  __syncthreads();
  // (either holds one entry per chain: no bound to check)
  if (dest == 1) p.rows[s_base[0] + s_cnt[0][warp] + (uint32_t)__popc(m1 & ((1u << lane) - 1u))] = e;
  else if (dest == 2) p.rest[s_base[1] + s_cnt[1][warp] + (uint32_t)__popc(m2 & ((1u << lane) - 1u))] = e;
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// The least i >= lo from which on symbols i .. len-1 of a chain agree with T(i + shift)
// beside them, T(i) = T_d[P - 1 - i]; len + shift <= P, and symbol lo inside the text.
__device__ __forceinline__ int agree_back(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len, bool fwd,
                                          uint32_t strand, uint32_t d, uint32_t P, int shift, int lo) {
  int hi = len;  // symbols hi .. len-1 agree
  while (hi > lo) {
    // symbols hi-32 .. hi-1 against T(hi-32+shift) .. T(hi-1+shift), the last symbol in the top bits
    uint64_t qw = fwd ? load32(packed, (int64_t)b0 + hi - 32) : load32(packed, (int64_t)b0 + len - hi);
    qw ^= comp_word(X, strand);
    uint64_t tw = d ? load32(X.text, (int64_t)X.top - P + hi - 32 + shift) : load32(X.text, (int64_t)P - hi - shift);
    if (!fwd) qw = rev32(qw);
    if (!d) tw = rev32(tw);
    const uint64_t x = qw ^ tw;
    const int same = x ? __clzll((long long)x) >> 1 : 32;
    hi -= same;
    if (same < 32) break;
  }
  return max(hi, lo);
}

// The first t in ts .. near a wide chain's change points can have hits from (near: none
// before it), where the strand's other chain has the one alignment `other`: the symbols
// after a failing one at te < near lie there or nowhere (text_branch_kernel).  So they agree
// from te + 1 on, and the ones before te agree one place nearer (deletion), there
// (mismatch, te then the last symbol that disagrees) or one place farther (insertion).
__device__ __forceinline__ int hits_from(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len, bool fwd,
                                         uint32_t strand, uint32_t d, uint32_t other, int ts, int near) {
  const int64_t P64 = (int64_t)X.top + len - other;
  if (P64 < len || P64 > (int64_t)X.top + 1) return near;
  const uint32_t P = (uint32_t)P64;
  const int m = agree_back(X, packed, b0, len, fwd, strand, d, P, 0, ts), te = max(ts, m - 1);
  if (te >= near) return near;
  if (agree(X, packed, b0, len, fwd, strand, d, 0, P - 1, te) == te) return te;
  if (m > ts && P <= X.top && agree(X, packed, b0, len, fwd, strand, d, 0, P, te) == te) return te;
  if (P < X.top && agree(X, packed, b0, len, fwd, strand, d, 0, P + 1, te) == te) return te;
  return near;
}

// The hits of a change point whose interval is one row: with the chain's symbol i
// beside T(i) = T_d[P - 1 - i], symbol te the first that disagrees.  Bit 0 the deletion
// (symbol i + 1 beside T(i) from te on), 1 the insertion and 2 the mismatch of the
// text's symbol `base` (as a query base): symbol i beside T(i + 1) from te on, beside T(i)
// after te.  One pass over the words for all three, 31 places a round.
__device__ __forceinline__ uint32_t one_row_branches(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len,
                                                     bool fwd, uint32_t strand, uint32_t d, int te, uint32_t P,
                                                     uint32_t& base) {
  // the text has to hold len - 1, len + 1 and len symbols
  uint32_t mask = (P + 1u >= (uint32_t)len ? 1u : 0u) | (P >= (uint32_t)len + 1u ? 2u : 0u) |
                  (P >= (uint32_t)len ? 4u : 0u);
  for (int m = te; mask && m < len; m += 31) {
    const uint64_t q = query32(X, packed, b0, len, fwd, strand, m), w = text32(X, d, P, m);
    if (m == te) base = ((uint32_t)w & 3u) ^ (strand ? X.comp_xor : 0u);
    const int left = len - 1 - m;  // places of the deletion and the mismatch; the insertion has one more
    const uint64_t some = (1ull << (2 * min(left, 31))) - 1ull, more = (1ull << (2 * min(left + 1, 31))) - 1ull;
    if (((q >> 2) ^ w) & some) mask &= ~1u;
    if ((q ^ (w >> 2)) & more) mask &= ~2u;
    if (((q ^ w) >> 2) & some) mask &= ~4u;
  }
  return mask;
}

// Sum over the block of v before this thread, plus *ctr advanced by the block's total.
template <int TPB>
__device__ __forceinline__ uint32_t block_slots(uint32_t v, unsigned int* ctr, uint32_t* s_cnt, uint32_t* s_base) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(kFull, incl, o);
    if (lane >= (uint32_t)o) incl += x;
  }
  if (lane == 31) s_cnt[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int w = 0; w < TPB / 32; ++w) {
      const uint32_t c = s_cnt[w];
      s_cnt[w] = tot;
      tot += c;
    }
    *s_base = tot ? atomicAdd(ctr, tot) : 0u;
  }
  __syncthreads();
  return *s_base + s_cnt[warp] + incl - v;
}

// The one-row chains of a read, a strand at a time.  With R the read ('+') or
// its reverse complement ('-'), the strand's chain on the forward index reads R
// from its left end and the one on the backward index from its right end; where
// both lie on the same alignment (all but the reads with an indel) one pass over
// the text serves both.  Up to seven hits a strand: the exact one, three a chain.
__global__ void __launch_bounds__(kReadTpb) text_read_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[kReadTpb / 32], s_base;
  const uint32_t n_reads = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  if ((uint64_t)blockIdx.x * kReadTpb >= n_reads) return;
  const uint32_t read = blockIdx.x * kReadTpb + threadIdx.x;
  uint32_t dg[4] = {kAbsent, kAbsent, kAbsent, kAbsent};  // '+' right, '-' right, '+' left, '-' left
  uint64_t b0 = 0;
  int len = 0;
  if (read < n_reads) {
#pragma unroll
    for (int c = 0; c < 4; ++c) dg[c] = __ldcs(p.diag + (uint64_t)c * p.n_reads + read);
    b0 = p.offs[read];
    len = (int)(p.offs[read + 1] - b0);
  }
  const uint32_t n = X.top;
  uint32_t turns = (is_diag(dg[0]) || is_diag(dg[2]) ? 1u : 0u) | (is_diag(dg[1]) || is_diag(dg[3]) ? 2u : 0u);
  while (__syncthreads_or((int)turns)) {
    // bits 0: exact; 1..3: deletion, insertion, mismatch of the right chain's change point; 4..6: the left chain's
    uint32_t mask = 0, base_r = 0, base_l = 0, strand = 0, right = 0, left = 0;
    int te_r = 0, te_l = 0;
    if (turns) {
      strand = (turns & 1u) ? 0u : 1u;
      turns &= turns - 1;
      right = strand ? dg[1] : dg[0];
      left = strand ? dg[3] : dg[2];
      const uint64_t cw = comp_word(X, strand);
      auto R32 = [&](int j) -> uint64_t {  // symbols j .. j+31 of R
        const uint64_t x = load32(p.packed, (int64_t)b0 + (strand ? len - 32 - j : j));
        const uint64_t r = rev32(x) ^ cw;
        return strand ? r : x;
      };
      // the alignment: R[j] at text[a + j]
      const bool has_r = is_diag(right), has_l = is_diag(left);
      const int64_t a_r = (int64_t)right - len, a_l = (int64_t)n - left;
      const bool same = has_r && has_l && a_r == a_l;
      te_r = te_l = len;
      {  // one pass for the left chain (or the right one alone): its first and last disagreement
        const int64_t a = has_l ? a_l : a_r;
        const int lo = a < 0 ? (int)-a : 0, hi = (int)min((int64_t)len, (int64_t)n - a);  // inside the text
        int first = -1, last = -1;
        for (int j = 0; j < len; j += 32) {
          uint64_t x = 0;
          if (j + 32 > lo && j < hi) x = load32(X.text, a + j) ^ R32(j);
          if (j < lo) x |= lo - j >= 32 ? ~0ull : (1ull << (2 * (lo - j))) - 1ull;
          if (j + 32 > hi) x = (j >= hi ? 0ull : x & ((1ull << (2 * (hi - j))) - 1ull)) |
                               (j >= hi ? ~0ull : ~0ull << (2 * (hi - j)));
          if (j + 32 > len) x &= (1ull << (2 * (len - j))) - 1ull;
          if (x) {
            if (first < 0) first = j + ((__ffsll((long long)x) - 1) >> 1);
            last = j + ((63 - __clzll((long long)x)) >> 1);
          }
        }
        if (has_l && first >= 0) te_l = first;
        if ((same || !has_l) && last >= 0) te_r = len - 1 - last;
      }
      if (has_r && has_l && !same) {  // another alignment: the right chain from its end, down to the text's start
        const int lo = a_r < 0 ? (int)-a_r : 0;
        int top = len;  // R[top .. len-1] matches
        for (; top > lo; top -= 32) {
          const uint64_t x = load32(X.text, a_r + top - 32) ^ R32(top - 32);
          if (x) {
            top -= __clzll((long long)x) >> 1;
            break;
          }
        }
        if (top > lo) te_r = len - top;
        else if (lo > 0) te_r = len - lo;
      }
      // the chain on the right is the backward one of '+', the forward one of '-'
      if (is_diag(strand ? left : right) && (strand ? te_l : te_r) == len) mask = 1;
#pragma unroll
      for (int side = 0; side < 2; ++side) {  // 0: right (backward index), 1: left (forward index)
        const uint32_t dgs = side ? left : right;
        const int te = side ? te_l : te_r;
        const bool fwd = (side != 0) == (strand == 0);
        if (!is_diag(dgs) || te >= len || te < branch_from(len, fwd)) continue;
        const uint32_t Q = dgs - (uint32_t)te;
        if (te == len - 1) {
          const uint32_t r = load_row_word((side ? X.dir[1].isa : X.dir[0].isa) + Q);
          push_block(p, r, r, (read << 1) | strand, len, fwd);
        } else {
          uint32_t base = 0;
          const uint32_t m = one_row_branches(X, p.packed, b0, len, fwd, strand, (uint32_t)side, te, dgs, base);
          if (side) {
            mask |= m << 4;
            base_l = base;
          } else {
            mask |= m << 1;
            base_r = base;
          }
        }
      }
    }
    uint32_t slot = block_slots<kReadTpb>((uint32_t)__popc(mask), p.res_total, s_cnt, &s_base);
    while (mask) {
      const int h = __ffs(mask) - 1;
      mask &= mask - 1;
      uint32_t key, meta, at;
      uint32_t side;
      if (h == 0) {  // the backward chain's
        side = strand;
        at = (side ? left : right) - (uint32_t)len;
        key = order_key(0, 0, 0);
        meta = pack_meta(0, 0, 0, 0, 0);
      } else {
        side = h >= 4 ? 1u : 0u;
        const int te = side ? te_l : te_r, item = (h - 1) % 3;
        const uint32_t b = side ? base_l : base_r;
        const bool fwd = (side != 0) == (strand == 0);
        // symbols taken from the text: one fewer for the deletion, one more for the insertion
        at = (side ? left : right) - (uint32_t)(len + (item == 0 ? -1 : (item == 1 ? 1 : 0)));
        key = order_key(fwd ? 4u : 2u, (uint32_t)(len - te), item == 0 ? 0u : (item == 1 ? 1 + 2 * b : 2 + 2 * b));
        meta = branch_meta(fwd, len, te, item == 0 ? 1u : (item == 1 ? 3u : 2u), item == 0 ? 0xFFu : b);
      }
      const uint32_t row = load_row_word((side ? X.dir[1].isa : X.dir[0].isa) + at);
      write_hit(p, slot++, (read << 1) | strand, key, row, row, meta, at + 1);
    }
    // (the loop's barrier is passed before s_cnt and s_base are rewritten)
  }
}

// A lane per row of the queued chains.  Row r of a chain, matched for t symbols,
// lies on an alignment: symbol i at T_r(i) = T_d[P - 1 - i], P = SA[r] + t.  With
//   te_r  the first symbol that disagrees,
//   D_r   the least i from which on symbol i+1 agrees with T_r(i)   (deletion),
//   I_r   the least i from which on symbol i agrees with T_r(i+1)   (insertion),
//   M_r   the least i from which on symbol i agrees with T_r(i)     (mismatch),
// all by comparing words, the chain's interval at t is the rows with te_r >= t;
// it changes at each te_r, and the helper's continuations at such a te keep the
// rows of that interval with D_r <= te; with I_r <= te and T_r(te) = b; with
// te_r = te, M_r <= te + 1 and T_r(te) = b.  Extending rows by the same symbols
// keeps their order, so the first and the last row kept give the hit's interval.
struct RowsShared {
  uint4 item[32];
  uint32_t n, next;
};

__global__ void __launch_bounds__(kRowsTpb) text_rows_kernel(DevIndex X, BatchedParams p) {
  __shared__ RowsShared rsh[kRowsWarps];
  __shared__ uint32_t c_res[kRowsTpb];
  const int tid = threadIdx.x;
  const uint32_t lane = tid & 31;
  RowsShared& ws = rsh[tid >> 5];
  const uint32_t n_items = *(volatile unsigned int*)p.rows_n;
  // sixteen chains a claim (most have two to five rows), fewer when every warp then still has some
  const uint32_t batch = min(max(n_items / (gridDim.x * kRowsWarps), 1u), 16u);
  c_res[tid] = 0;
  if (lane == 0) ws.n = ws.next = 0;
  __syncwarp();
  bool exhausted = false;
  for (;;) {
    if (ws.next == ws.n) {  // claim the next chains
      if (exhausted) break;
      uint32_t c0 = 0;
      if (lane == 0) c0 = atomicAdd(p.rows_head, batch);
      c0 = __shfl_sync(kFull, c0, 0);
      if (c0 + batch >= n_items) exhausted = true;
      const uint32_t got = c0 < n_items ? min(batch, n_items - c0) : 0u;
      if (lane < got) ws.item[lane] = p.rows[c0 + lane];
      __syncwarp();
      if (lane == 0) {
        ws.n = got;
        ws.next = 0;
      }
      __syncwarp();
      if (!got) break;
    }
    // as many of the held chains as 32 lanes hold rows of
    const uint32_t first = ws.next, held = ws.n - first;
    uint32_t rows = 0;
    if (lane < held) rows = min(ws.item[first + lane].y - ws.item[first + lane].x + 1u, kRows);
    uint32_t incl = rows;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    const unsigned fit = __ballot_sync(kFull, lane < held && incl <= 32);
    const uint32_t take = (uint32_t)__popc(fit);  // (sizes are positive: the fitting ones are the first ones)
    // this lane's chain and its lanes, start .. end-1
    const uint32_t total = __shfl_sync(kFull, incl, (int)take - 1);
    const uint32_t widest = __reduce_max_sync(kFull, lane < take ? rows : 0u);
    const unsigned starts = __reduce_or_sync(kFull, lane < take ? 1u << (incl - rows) : 0u), upto = (2u << lane) - 1u;
    const uint32_t mine = lane < total ? (uint32_t)__popc(starts & upto) - 1u : 0xFFFFFFFFu;
    const uint32_t start = lane < total ? 31u - (uint32_t)__clz(starts & upto) : lane, j = lane - start;
    const uint32_t end = lane < total ? ((starts & ~upto) ? (uint32_t)__ffs(starts & ~upto) - 1u : total) : lane + 1;
    const unsigned seg = lane < total ? (kFull >> (32u - end)) & (kFull << start) : 0u;
    uint32_t rs = 0, d = 0, P = 0, strand = 0;
    bool fwd = false;
    int len = 0, t0 = 0, ts = 0, te = -1, D = 0x7FFFFFFF, I = 0x7FFFFFFF, M = 0x7FFFFFFF;
    uint64_t b0 = 0;
    if (mine != 0xFFFFFFFFu) {
      const uint4 e = ws.item[first + mine];
      rs = e.z;
      strand = rs & 1u;
      fwd = (e.w >> 16) & 1u;
      d = (fwd ? 1u : 0u) ^ strand;
      t0 = (int)(e.w & 0xFFFFu);
      b0 = p.offs[rs >> 1];
      len = (int)(p.offs[(rs >> 1) + 1] - b0);
      ts = max(t0, branch_from(len, fwd));  // change points before it are not the helper's
      const uint32_t sa = __ldg((d ? X.dir[1].sa : X.dir[0].sa) + e.x + j);
      P = sa + (uint32_t)t0;
      te = t0 + agree(X, p.packed, b0, len, fwd, strand, d, t0, sa, (int)min((uint32_t)(len - t0), sa));
    }
    __syncwarp();
    if (lane == 0) ws.next = first + take;
    if (te >= ts) {  // of use to the helper: where the three shifted alignments begin to agree for good
      auto from_end = [&](int shift) -> int {
        const int64_t need = (int64_t)len + shift;  // text symbols the read takes
        if (need > (int64_t)P) return 0x7FFFFFFF;
        return agree_back(X, p.packed, b0, len, fwd, strand, d, P, shift, shift < 0 ? ts + 1 : ts);  // (the deletion's first symbol is te + 1)
      };
      D = from_end(-1) - 1;
      I = from_end(1);
      M = from_end(0);
    }
    // the row each alignment ends in, where it may be asked for
    const uint32_t* isa = d ? X.dir[1].isa : X.dir[0].isa;
    const int last = min(te, len - 2);  // the last change point whose interval holds this row
    uint32_t row_d = 0, row_i = 0, row_m = 0;
    // a change at the last symbol: the interval before it goes to the block list
    const unsigned ends = __ballot_sync(kFull, mine != 0xFFFFFFFFu && te == len - 1) & seg;
    const bool block = ends && te >= len - 1;
    if (te >= ts) {
      if (D <= last || block) row_d = load_row_word(isa + P - (uint32_t)(len - 1));
      if (I <= last) row_i = load_row_word(isa + P - (uint32_t)(len + 1));
      if (te == len || (te <= len - 2 && M <= te + 1)) row_m = load_row_word(isa + P - (uint32_t)len);
    }
    auto emit = [&](uint32_t key, uint32_t k, uint32_t l, uint32_t meta, uint32_t at) {  // at: this lane's SA value
      uint32_t r = c_res[tid];
      const unsigned slot = res_slot(p, r);
      c_res[tid] = r;
      write_hit(p, slot, rs, key, k, l, meta, k == l ? at + 1 : 0u);
    };
    const uint32_t at = P - (uint32_t)len;  // the whole read's and the mismatch's; the deletion ends one on, the insertion one before
    auto interval = [&](bool in, uint32_t row, bool& lead, uint32_t& k, uint32_t& l) {  // of the chain's lanes with `in`
      const unsigned m = __ballot_sync(kFull, in) & seg;
      lead = m && lane == (uint32_t)__ffs(m) - 1u;
      k = row;
      l = __shfl_sync(kFull, row, m ? 31 - __clz(m) : (int)lane);
    };
    bool lead;
    uint32_t k, l;
    // the whole read: the backward chain's exact hit
    interval(te == len, row_m, lead, k, l);
    if (lead && !fwd) emit(order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0), at);
    interval(block, row_d, lead, k, l);
    if (lead) push_block(p, k, l, rs, len, fwd);
    // the other change points, in order
    bool todo = te >= ts && te <= len - 2;
    while (__ballot_sync(kFull, todo)) {
      int cp = todo ? te : 0x7FFFFFFF;  // the least te left among the chain's lanes
      for (uint32_t o = 1; o < widest; o <<= 1) {
        const int v = __shfl_down_sync(kFull, cp, o);
        if (lane + o < end) cp = min(cp, v);
      }
      cp = __shfl_sync(kFull, cp, (int)start);
      const bool live = cp != 0x7FFFFFFF;
      const bool in = live && te >= cp;
      uint32_t b = 0;  // the row's text symbol at cp, as a query base
      if (in && P > (uint32_t)cp) {
        const uint64_t tw = d ? load32(X.text, (int64_t)(X.top - P) + cp) : load32(X.text, (int64_t)P - 1 - cp);
        b = ((uint32_t)tw & 3u) ^ (strand ? X.comp_xor : 0u);
      }
      const uint32_t tf = (uint32_t)(len - cp);
      const uint32_t sec = fwd ? 4u : 2u;
      interval(in && D <= cp, row_d, lead, k, l);
      if (lead) emit(order_key(sec, tf, 0), k, l, branch_meta(fwd, len, cp, 1, 0xFFu), at + 1);
      const bool ins = in && I <= cp, mis = in && te == cp && M <= cp + 1;
      // insertions and mismatches of the bases that occur
      for (uint32_t some = __reduce_or_sync(kFull, (ins ? 1u << (2 * b) : 0u) | (mis ? 2u << (2 * b) : 0u)); some;
           some &= some - 1) {
        const uint32_t item = (uint32_t)__ffs(some) - 1u, v = item >> 1;
        const bool is_mis = item & 1u;
        interval((is_mis ? mis : ins) && b == v, is_mis ? row_m : row_i, lead, k, l);
        if (lead)
          emit(order_key(sec, tf, 1 + item), k, l, branch_meta(fwd, len, cp, is_mis ? 2 : 3, v), is_mis ? at : at - 1);
      }
      if (te == cp) todo = false;
    }
    __syncwarp();
  }
  res_leave(p, c_res[tid]);
}

// Marks a slot of the walk queue that holds no walk.
__device__ __forceinline__ void no_walk(const BatchedParams& p, uint32_t slot) { p.walk[slot].z = 0xFFFFFFFFu; }

// Persistent: the chains still more than kRows rows wide, a lane each, one rank
// step per iteration until they are not (-> row queue); the change points they
// pass inside the helper's window go to the spill queue.  A warp prepares 32
// chains at a time, every lane one (five or six dependent loads), and its lanes
// take them from shared memory as they run out; what they queue is gathered and written 32
// at a time.  A lane that fetched its own next chain, and an atomic per entry queued: 1189 us
// for the wide chains of 2M x 150 bp at 600 Mbp; so: 951, and 773 once an interval's two
// blocks were loaded together (rank_step).  Latency of the steps, some 130 at most in a row.
struct WideShared {
  uint4 chain[32];  // k, l, rs, t | len << 15 | forward << 31
  uint64_t q[32];
  int ts[32];
  uint4 rows[64];         // for the row queue
  SpillEntry change[64];  // for the spill queue
};

// Entries a warp takes from a queue at a time: 32, fewer where that would leave warps without.
__device__ __forceinline__ uint32_t per_claim(uint32_t n, uint32_t warps) {
  return min(max(n / (kClaims * warps), 1u), 32u);
}

template <bool CENSUS>
__global__ void __launch_bounds__(kWideTpb) text_wide_kernel(DevIndex X, BatchedParams p) {
  __shared__ WideShared wsh[kWideTpb / 32];
  __shared__ uint32_t c_res[kWideTpb];
  const int tid = threadIdx.x;
  const uint32_t lane = tid & 31;
  WideShared& ws = wsh[tid >> 5];
  const uint32_t n_src = *(volatile unsigned int*)p.rest_n;
  const uint32_t batch = per_claim(n_src, gridDim.x * (kWideTpb / 32));
  c_res[tid] = 0;
  bool active = false, exhausted = false;
  uint32_t ready = 0;  // chains prepared and not taken
  uint32_t n_rows = 0, n_change = 0;  // entries held for the queues
  uint32_t k = 0, l = 0, rs = 0;
  int t = 0, len = 0, ts = 0;
  bool fwd = false;
  uint64_t q = 0;  // the next symbols
  int ql = 0;      // how many q holds
  const OccBlock* occ = nullptr;
  uint32_t dollar = 0, sectors = 0;
  const uint32_t bi = p.batch_idle < 1 ? 1u : p.batch_idle;
  auto flush_rows = [&](uint32_t from, uint32_t n) {
    __syncwarp();
    uint32_t c0 = 0;
    if (lane == 0) c0 = atomicAdd(p.rows_n, n);
    c0 = __shfl_sync(kFull, c0, 0);
    if (lane < n) p.rows[c0 + lane] = ws.rows[from + lane];  // (one entry per chain: no bound to check)
    __syncwarp();
  };
  auto flush_change = [&](uint32_t from, uint32_t n) {
    __syncwarp();
    uint32_t c0 = 0;
    if (lane == 0) c0 = atomicAdd(p.spill_tail, n);
    c0 = __shfl_sync(kFull, c0, 0);
    if (lane < n) {
      if (c0 + lane < p.spill_cap) p.spill[c0 + lane] = ws.change[from + lane];
      else atomicOr(p.status, kStatusSpillFull);
    }
    __syncwarp();
  };
  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !active);  // every lane, every iteration
    if (!ready && !exhausted && (uint32_t)__popc(idle) >= bi) {
      uint32_t c0 = 0;
      if (lane == 0) c0 = atomicAdd(p.rest_head, batch);
      c0 = __shfl_sync(kFull, c0, 0);
      if (c0 + batch >= n_src) exhausted = true;
      ready = c0 < n_src ? min(batch, n_src - c0) : 0u;
      if (lane < ready) {
        const uint4 e = p.rest[c0 + lane];
        const uint64_t b0 = p.offs[e.z >> 1];
        const int c_len = (int)(p.offs[(e.z >> 1) + 1] - b0), c_t = (int)(e.w & 0xFFFFu);
        const bool c_fwd = (e.w >> 16) & 1u;
        const uint32_t strand = e.z & 1u, d = (c_fwd ? 1u : 0u) ^ strand;
        int c_ts = branch_from(c_len, c_fwd);
        // change points without hits are not queued: their remaining symbols hold a head that
        // does not occur, or that occurs once and not where the read's two parts would meet
        const uint32_t other = other_chain(X, p, e.z, d, c_len, c_ts + 1);
        if (other != kMany) {
          const int near = c_len - (int)X.tmer_len - kHeadSteps;
          c_ts = other == kAbsent ? near : hits_from(X, p.packed, b0, c_len, c_fwd, strand, d, other, c_ts, near);
        }
        ws.chain[lane] = make_uint4(e.x, e.y, e.z, (uint32_t)c_t | (uint32_t)c_len << 15 | (c_fwd ? 1u << 31 : 0u));
        ws.q[lane] = query32(X, p.packed, b0, c_len, c_fwd, strand, c_t);
        ws.ts[lane] = c_ts;
      }
      __syncwarp();
    }
    if (ready) {
      const uint32_t rank = (uint32_t)__popc(idle & ((1u << lane) - 1u));
      if (!active && rank < ready) {
        const uint32_t i = ready - 1 - rank;
        const uint4 e = ws.chain[i];
        k = e.x;
        l = e.y;
        rs = e.z;
        t = (int)(e.w & 0x7FFFu);
        len = (int)((e.w >> 15) & 0x7FFFu);
        fwd = e.w >> 31;
        q = ws.q[i];
        ts = ws.ts[i];
        const uint32_t d = (fwd ? 1u : 0u) ^ (rs & 1u);
        occ = d ? X.dir[1].occ : X.dir[0].occ;
        dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
        ql = 32;
        active = true;
      }
      ready -= min(ready, (uint32_t)__popc(idle));
      __syncwarp();
    } else if (exhausted && idle == kFull) {
      break;
    }
    bool row = false, change = false;
    const uint32_t pk = k, pl = l;
    const int pt = t;
    if (active) {
      if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
      rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
      if (t >= ts && l - k != pl - pk) {  // a change point
        change = t != len - 1;
        if (!change) push_block(p, pk, pl, rs, len, fwd);
      }
      active = k <= l && t + 1 < len;
      if (active) {
        ++t;
        q >>= 2;
        row = l - k < (t < ts ? kRowsBefore : kRows);  // few enough rows for a lane each
        active = !row;
        if (--ql == 0) {  // 32 symbols on
          q = query32(X, p.packed, p.offs[rs >> 1], len, fwd, rs & 1u, t);
          ql = 32;
        }
      } else if (k <= l && !fwd) {  // the whole read: the exact hit
        uint32_t r = c_res[tid];
        const unsigned slot = res_slot(p, r);
        c_res[tid] = r;
        write_hit(p, slot, rs, order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0));
      }
    }
    // entries for the two queues are written 32 at a time
    const unsigned mr = __ballot_sync(kFull, row), mc = __ballot_sync(kFull, change);
    const unsigned below = (1u << lane) - 1u;
    if (row) ws.rows[n_rows + __popc(mr & below)] = make_uint4(k, l, rs, (uint32_t)t | (fwd ? 1u << 16 : 0u));
    if (change) ws.change[n_change + __popc(mc & below)] = SpillEntry{pk, pl, rs, (uint32_t)pt | (fwd ? 1u << 16 : 0u)};
    n_rows += (uint32_t)__popc(mr);
    n_change += (uint32_t)__popc(mc);
    if (n_rows >= 32) {
      n_rows -= 32;
      flush_rows(n_rows, 32);
    }
    if (n_change >= 32) {
      n_change -= 32;
      flush_change(n_change, 32);
    }
  }
  if (n_rows) flush_rows(0, n_rows);
  if (n_change) flush_change(0, n_change);
  res_leave(p, c_res[tid]);  // slots of this lane's last chunk that were reserved but not used
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// The interval's steps with all four symbols (physical codes), from its one or two blocks.
__device__ __forceinline__ void rank_step4(const DevIndex& X, const OccBlock* occ, uint32_t dollar, uint32_t k,
                                           uint32_t l, uint32_t (&nk)[4], uint32_t (&nl)[4]) {
  const uint32_t q0 = k >> 6, q1 = l >> 6;
  uint32_t cnt[4], cnt1[4];
  uint4 bits, bits1;
  load_block_pair(occ, q0, q1, X.load_mode, cnt, bits, cnt1, bits1);
  const bool two = q1 != q0;
  const uint64_t mk = row_mask(k & 63), ml = row_mask((l & 63) + 1);
#pragma unroll
  for (uint32_t b = 0; b < 4; ++b) {
    const uint64_t m0 = match_mask(bits, b), m1 = two ? match_mask(bits1, b) : m0;
    nk[b] = X.C[b] + 1u + cnt[b] + (uint32_t)__popcll(m0 & mk);
    nl[b] = X.C[b] + (two ? cnt1[b] : cnt[b]) + (uint32_t)__popcll(m1 & ml);
  }
  // the '$' row is stored as code 0 in its block
  if (k > dollar && q0 == (dollar >> 6)) nk[0] -= 1;
  if (l >= dollar && q1 == (dollar >> 6)) nl[0] -= 1;
}

// Persistent: the spilled change points, 32 a warp at a time.  The eight continuations of
// one begin with one step from the same interval (the deletion with the symbol after the
// failing one, the insertions and mismatches with b), so one or two blocks give all their
// first intervals; those that are not empty wait in the lane that holds the change point
// until a lane of the warp is free to run one, a rank step per iteration, without touching
// memory between them.  (One lane for all of a change point's: 1246 us on 2M x 150 bp, 600
// Mbp; the few long ones held their warps.  So: 884, 780 with an interval's two blocks
// loaded together.)  What has narrowed to one row and matched on goes to the walk queue.
//
// Most wide change points lie in tandem runs whose read goes on into sequence that
// occurs once, or with an error in its head nowhere: there the strand's other chain
// decides them without a rank step (about 100 sectors a change point otherwise, its
// intervals being thousands of rows wide), here or, for a chain's leading ones, before
// they are queued (hits_from).
template <bool CENSUS>
__global__ void __launch_bounds__(kWideTpb, 7) text_branch_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t c_res[kWideTpb], c_walk[kWideTpb], s_k[4][kWideTpb], s_l[4][kWideTpb];
  __shared__ uint8_t s_from[kWideTpb];
  const int tid = threadIdx.x;
  const uint32_t lane = tid & 31;
  const uint32_t n_src = min(*(volatile unsigned int*)p.spill_tail, p.spill_cap);
  const uint32_t batch = per_claim(n_src, gridDim.x * (kWideTpb / 32));
  c_res[tid] = c_walk[tid] = 0;
  bool exhausted = false, walk_full = false, stepping = false;
  // the change point this lane holds for the warp
  uint32_t todo = 0;  // continuations left: bit 0 deletion, 1 + b insertion, 5 + b mismatch
  uint32_t h_rs = 0, h_at = 0;  // h_at: te | len << 15 | forward << 31
  uint64_t h_q = 0;   // symbols from te on
  // the continuation it runs
  uint32_t k = 0, l = 0, rs = 0, key = 0;
  int t = 0, te = 0, len = 0;
  bool fwd = false;
  uint64_t q = 0;  // the next symbols
  int ql = 0;
  const OccBlock* occ = nullptr;
  uint32_t dollar = 0, sectors = 0;
  const uint32_t bi = p.batch_idle < 1 ? 1u : p.batch_idle;
  auto hit = [&]() {
    const uint32_t s = key & 0xFFu;
    uint32_t r = c_res[tid];
    const unsigned slot = res_slot(p, r);
    c_res[tid] = r;
    write_hit(p, slot, rs, key, k, l,
              branch_meta(fwd, len, te, s == 0 ? 1u : ((s & 1u) ? 3u : 2u), s == 0 ? 0xFFu : (s - 1) >> 1));
  };
  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !stepping);  // every lane, every iteration
    unsigned give = idle ? __ballot_sync(kFull, todo != 0) : 0u;
    if (!give && !exhausted && (uint32_t)__popc(idle) >= bi) {  // the next change points
      uint32_t c0 = 0;
      if (lane == 0) c0 = atomicAdd(p.spill_head, batch);
      c0 = __shfl_sync(kFull, c0, 0);
      if (c0 + batch >= n_src) exhausted = true;
      if (lane < batch && c0 + lane < n_src) {
        const SpillEntry e = p.spill[c0 + lane];
        const uint32_t rs = e.rs;
        const int te = (int)(e.jtype & 0xFFFFu);
        const bool fwd = (e.jtype >> 16) & 1u;
        const uint64_t b0 = p.offs[rs >> 1];
        const int len = (int)(p.offs[(rs >> 1) + 1] - b0);
        const uint32_t strand = rs & 1u, d = (fwd ? 1u : 0u) ^ strand;
        const uint64_t q0 = query32(X, p.packed, b0, len, fwd, strand, te);
        // The symbols after the failing one, read from the other end, begin the strand's
        // other chain.  Where they reach past its head, its one row is the only place a
        // continuation can match, and there is none if the head found it absent.
        const uint32_t other = other_chain(X, p, rs, d, len, te + 1);
        if (other == kMany) {
          h_rs = rs;
          h_at = (uint32_t)te | (uint32_t)len << 15 | (fwd ? 1u << 31 : 0u);
          h_q = q0;
          uint32_t nk[4], nl[4];
          rank_step4(X, d ? X.dir[1].occ : X.dir[0].occ, d ? X.dir[1].dollar : X.dir[0].dollar, e.k, e.l, nk, nl);
          if (CENSUS) sectors += (e.k >> 6) == (e.l >> 6) ? 1u : 2u;
          const uint32_t w = (uint32_t)q0 & 3u, w1 = (uint32_t)(q0 >> 2) & 3u;
#pragma unroll
          for (uint32_t b = 0; b < 4; ++b) {
            s_k[b][tid] = nk[b];
            s_l[b][tid] = nl[b];
            if (nk[b] <= nl[b]) todo |= (b == w1 ? 1u : 0u) | 2u << b | (b != w ? 32u << b : 0u);
          }
        } else if (other != kAbsent) {
          // symbol i at T_d[P - 1 - i] for the symbols after the failing one; the ones
          // before it one place nearer (deletion), there (mismatch) or one farther (insertion)
          const int r = len - te - 1;
          const int64_t P64 = (int64_t)X.top + len - other;
          if (P64 >= len && P64 <= (int64_t)X.top + 1) {
            const uint32_t P = (uint32_t)P64;
            if (agree(X, p.packed, b0, len, fwd, strand, d, te + 1, P - (uint32_t)te - 1, r) == r) {
              const uint32_t row = load_row_word((d ? X.dir[1].isa : X.dir[0].isa) + (P - (uint32_t)len));
              const uint32_t cx = strand ? X.comp_xor : 0u, sec = fwd ? 4u : 2u, tf = (uint32_t)(len - te);
              auto text_at = [&](uint32_t at) -> uint32_t {  // T_d[at]
                return (uint32_t)load32(X.text, d ? (int64_t)X.top - 1 - at : (int64_t)at) & 3u;
              };
              auto found = [&](uint32_t slot_key, uint32_t kind, uint32_t base) {
                uint32_t c = c_res[tid];
                const unsigned slot = res_slot(p, c);
                c_res[tid] = c;
                write_hit(p, slot, rs, order_key(sec, tf, slot_key), row, row, branch_meta(fwd, len, te, kind, base),
                          P - (uint32_t)len + 1);
              };
              if (agree(X, p.packed, b0, len, fwd, strand, d, 0, P - 1, te) == te) found(0, 1, 0xFFu);
              if (P <= X.top) {
                const uint32_t here = text_at(P - 1 - (uint32_t)te);  // beside the failing symbol
                const uint32_t w = (uint32_t)q0 & 3u;
                if (here == w && P < X.top && agree(X, p.packed, b0, len, fwd, strand, d, 0, P + 1, te) == te) {
                  const uint32_t b = text_at(P - (uint32_t)te) ^ cx;
                  found(1 + 2 * b, 3, b);
                }
                if (here != w && agree(X, p.packed, b0, len, fwd, strand, d, 0, P, te) == te)
                  found(2 + 2 * (here ^ cx), 2, here ^ cx);
              }
            }
          }
        }
      }
      __syncwarp();
      give = __ballot_sync(kFull, todo != 0);
    }
    if (give) {  // the i-th idle lane takes a continuation of the i-th lane that holds some
      const unsigned below = (1u << lane) - 1u;
      const uint32_t n = (uint32_t)min(__popc(idle), __popc(give));
      const uint32_t nth = (uint32_t)__popc(give & below);
      const bool giver = ((give >> lane) & 1u) && nth < n;
      const bool taker = !stepping && (uint32_t)__popc(idle & below) < n;
      if (giver) s_from[(tid & ~31) + nth] = (uint8_t)lane;
      __syncwarp();
      const int src = taker ? s_from[(tid & ~31) + __popc(idle & below)] : (int)lane;
      const uint32_t item = (uint32_t)__shfl_sync(kFull, __ffs(todo) - 1, src);
      const uint32_t g_rs = __shfl_sync(kFull, h_rs, src), g_at = __shfl_sync(kFull, h_at, src);
      const uint64_t q0 = __shfl_sync(kFull, h_q, src);
      if (giver) todo &= todo - 1;
      if (taker) {
        rs = g_rs;
        te = (int)(g_at & 0x7FFFu);
        len = (int)((g_at >> 15) & 0x7FFFu);
        fwd = g_at >> 31;
        // the symbol stepped with, as a physical code; the next symbol; the order key's slot
        const uint32_t b = item == 0 ? (uint32_t)(q0 >> 2) & 3u : (item - 1) & 3u;
        const int skip = item == 0 ? 2 : (item <= 4 ? 0 : 1);
        const uint32_t qb = b ^ ((rs & 1u) ? X.comp_xor : 0u);
        key = order_key(fwd ? 4u : 2u, (uint32_t)(len - te), item == 0 ? 0u : (item <= 4 ? 1 + 2 * qb : 2 + 2 * qb));
        k = s_k[b][(tid & ~31) + src];
        l = s_l[b][(tid & ~31) + src];
        t = te + skip;
        q = q0 >> (2 * skip);
        ql = 32 - skip;
        const uint32_t d = (fwd ? 1u : 0u) ^ (rs & 1u);
        occ = d ? X.dir[1].occ : X.dir[0].occ;
        dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
        if (t == len) hit();  // the deletion of the last symbol but one
        else stepping = true;
      }
      __syncwarp();
    } else if (exhausted && idle == kFull) {
      break;
    }
    if (!stepping) continue;
    const bool was_one = k == l;
    if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
    rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
    if (k > l) {
      stepping = false;
      continue;
    }
    if (++t == len) {  // matched to the read end
      hit();
      stepping = false;
      continue;
    }
    q >>= 2;
    if (was_one && !walk_full) {  // one row that has matched on: the text tells the rest
      uint32_t cs = c_walk[tid];
      const unsigned slot = chunk_slot(
          p.walk_cap, cs, [&](unsigned n) { return claim(p.walk_n, n); }, [&](uint32_t i) { no_walk(p, i); });
      c_walk[tid] = cs;
      if (slot < p.walk_cap) {
        p.walk[slot] = make_uint4(k, key, rs, (uint32_t)t | (fwd ? 1u << 16 : 0u));
        stepping = false;
        continue;
      }
      walk_full = true;  // this lane's walks go on by rank steps
    }
    if (--ql == 0) {  // 32 symbols on
      q = query32(X, p.packed, p.offs[rs >> 1], len, fwd, rs & 1u, t);
      ql = 32;
    }
  }
  {  // slots of this lane's last chunks that were reserved but not used
    res_leave(p, c_res[tid]);
    chunk_leave(p.walk_cap, c_walk[tid], [&](uint32_t i) { no_walk(p, i); });
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// A thread per queued branch walk that has narrowed to one row.
template <bool CENSUS>
__global__ void __launch_bounds__(kWalkTpb) text_walk_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[kWalkTpb / 32], s_base;
  const uint32_t n = min(*(volatile unsigned int*)p.walk_n, p.walk_cap);
  uint32_t sectors = 0;
  for (uint32_t i0 = blockIdx.x * kWalkTpb; i0 < n; i0 += gridDim.x * kWalkTpb) {
    const uint32_t i = i0 + threadIdx.x;
    bool hit = false;
    uint32_t row = 0, meta = 0, at = 0;
    uint4 e = make_uint4(0, 0, 0xFFFFFFFFu, 0);
    if (i < n) e = __ldcs(p.walk + i);
    if (e.z != 0xFFFFFFFFu) {  // (no_walk)
      const uint32_t strand = e.z & 1u;
      const bool fwd = (e.w >> 16) & 1u;
      const uint32_t d = (fwd ? 1u : 0u) ^ strand;
      const uint32_t P = load_row_word((d ? X.dir[1].sa : X.dir[0].sa) + e.x);
      const uint64_t b0 = p.offs[e.z >> 1];
      const int len = (int)(p.offs[(e.z >> 1) + 1] - b0);
      const int t = (int)(e.w & 0xFFFFu), left = len - t;
      if (CENSUS) sectors += 2;
      if (P >= (uint32_t)left && agree(X, p.packed, b0, len, fwd, strand, d, t, P, left) == left) {
        const uint32_t s = e.y & 0xFFu;
        hit = true;
        at = P - (uint32_t)left;
        row = load_row_word((d ? X.dir[1].isa : X.dir[0].isa) + at);
        meta = branch_meta(fwd, len, len - (int)((e.y >> 8) & 0xFFFFu), s == 0 ? 1u : ((s & 1u) ? 3u : 2u),
                           s == 0 ? 0xFFu : (s - 1) >> 1);
        if (CENSUS) ++sectors;
      }
    }
    const uint32_t slot = block_slots<kWalkTpb>(hit ? 1u : 0u, p.res_total, s_cnt, &s_base);
    if (hit) write_hit(p, slot, e.z, e.y, row, row, meta, at + 1);
    __syncthreads();  // s_cnt and s_base are rewritten next round
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// A thread per block entry (k, l at the last symbol but one of the chain, as the
// fused kernel's drain maps them): the deletion is the interval itself; per base b
// the step with b gives the mismatch, and a further step with the read's end base
// the insertion.  In the j = 1 block an insertion is reported with base INSERTION
// and position b, and b stays the position of the block's later mismatches
// (search.c:1556).
template <bool CENSUS>
__global__ void __launch_bounds__(kWalkTpb) text_block_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[kWalkTpb / 32], s_base;
  const uint32_t n = min(*(volatile unsigned int*)p.block_n, p.block_cap);
  uint32_t sectors = 0;
  for (uint32_t i0 = blockIdx.x * kWalkTpb; i0 < n; i0 += gridDim.x * kWalkTpb) {
    const uint32_t i = i0 + threadIdx.x;
    SpillEntry e{1, 0, 0, 0};
    uint32_t nk[4], nl[4], ik[4], il[4], mask = 0;  // bit 0 deletion, 1 + b mismatch, 5 + b insertion
    bool last = false;
    int end = 0;
    if (i < n) {
      e = p.blocks[i];
      last = ((e.jtype >> 16) & 3u) == kBlkN;
      const uint32_t strand = e.rs & 1u, d = (last ? 1u : 0u) ^ strand;
      const OccBlock* occ = d ? X.dir[1].occ : X.dir[0].occ;
      const uint32_t dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
      const uint64_t b0 = p.offs[e.rs >> 1];
      end = (int)(p.offs[(e.rs >> 1) + 1] - b0) - 1;
      const uint32_t w = (uint32_t)load32(p.packed, (int64_t)b0 + (last ? end : 0)) & 3u;
      const uint32_t cx = strand ? X.comp_xor : 0u;
      uint32_t pk[4], pl[4];  // by physical symbol
      rank_step4(X, occ, dollar, e.k, e.l, pk, pl);
      if (CENSUS) sectors += (e.k >> 6) == (e.l >> 6) ? 1u : 2u;
      mask = 1;
#pragma unroll
      for (uint32_t b = 0; b < 4; ++b) {
        nk[b] = sel4(pk, b ^ cx);
        nl[b] = sel4(pl, b ^ cx);
        ik[b] = nk[b];
        il[b] = nl[b];
        if (nk[b] > nl[b]) continue;
        if (b != w) mask |= 2u << b;
        if (CENSUS) sectors += (ik[b] >> 6) == (il[b] >> 6) ? 1u : 2u;
        rank_step(X, occ, dollar, w ^ cx, ik[b], il[b]);
        if (ik[b] <= il[b]) mask |= 32u << b;
      }
    }
    uint32_t slot = block_slots<kWalkTpb>((uint32_t)__popc(mask), p.res_total, s_cnt, &s_base);
    const uint32_t sec = last ? 3u : 1u;
    if (mask & 1u)
      write_hit(p, slot++, e.rs, order_key(sec, 0, 0), e.k, e.l, pack_meta(last ? 1 : 0, 1, 1, 0xFF, last ? end : 0));
    uint32_t bpos = 0;  // the base of the block's last insertion so far
#pragma unroll
    for (uint32_t b = 0; b < 4; ++b) {
      if (mask & (2u << b))
        write_hit(p, slot++, e.rs, order_key(sec, 0, 1 + 2 * b), nk[b], nl[b],
                  pack_meta(last ? 1 : 0, 1, 2, b, last ? end : (int)bpos));
      if (mask & (32u << b)) {
        write_hit(p, slot++, e.rs, order_key(sec, 0, 2 + 2 * b), ik[b], il[b],
                  last ? pack_meta(1, 1, 3, b, end) : pack_meta(0, 1, 3, 3, (int)b));
        bpos = b;
      }
    }
    __syncthreads();  // s_cnt and s_base are rewritten next round
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// Exact search of both strands (BWExactSearchBackward over backward, '-': over
// forward_rev; search.h:9-65) with the text: a thread per (read, strand), its start table
// entry, rank steps until the interval is empty or has stayed one row for a step, then one
// comparison with the text.  (200k x 100 bp, 4 Mbp: 163 us with rank steps to the end.)
template <bool CENSUS>
__global__ void __launch_bounds__(kHeadTpb) text_exact_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[kHeadTpb / 32], s_base;
  const uint32_t n_reads = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  if ((uint64_t)blockIdx.x * kHeadTpb >= n_reads) return;
  const uint32_t read = blockIdx.x * kHeadTpb + threadIdx.x, strand = blockIdx.y, d = strand;
  uint32_t k = 1, l = 0, sectors = 0, sa1 = 0;
  if (read < n_reads && p.ok[read]) {
    const uint64_t b0 = p.offs[read], b1 = p.offs[read + 1];
    if (b1 >= b0 + 3 && b1 - b0 <= 32767 && b1 <= p.packed_len) {
      const int len = (int)(b1 - b0);
      const OccBlock* occ = d ? X.dir[1].occ : X.dir[0].occ;
      const uint32_t dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
      uint64_t q = query32(X, p.packed, b0, len, false, strand, 0);
      int t = 0;
      k = 0;
      l = X.top;
      const int L = (int)X.tmer_len;
      if (len >= L) {
        const uint32_t r = __brev((uint32_t)q) >> (32 - 2 * L);
        const uint2 s = load_row_pair((d ? X.tmer[1] : X.tmer[0]) + (((r & 0x55555555u) << 1) | ((r >> 1) & 0x55555555u)));
        if (CENSUS) ++sectors;
        k = s.x;
        l = s.y;
        t = L;
        q >>= 2 * L;
      }
      while (k <= l && t < len) {
        const uint32_t pk = k, pl = l;
        if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
        rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
        ++t;
        if ((t & 31) == 0) q = query32(X, p.packed, b0, len, false, strand, t);
        else q >>= 2;
        if (k == l && pk == pl && t < len) {
          const uint32_t P = load_row_word((d ? X.dir[1].sa : X.dir[0].sa) + k);
          const int left = len - t;
          if (CENSUS) sectors += 2;
          if (P >= (uint32_t)left && agree(X, p.packed, b0, len, false, strand, d, t, P, left) == left) {
            k = l = load_row_word((d ? X.dir[1].isa : X.dir[0].isa) + P - (uint32_t)left);
            sa1 = P - (uint32_t)left + 1;
            if (CENSUS) ++sectors;
          } else {
            k = 1;
            l = 0;
          }
          break;
        }
      }
    }
  }
  const bool hit = k <= l;
  const uint32_t slot = block_slots<kHeadTpb>(hit ? 1u : 0u, p.res_total, s_cnt, &s_base);
  if (hit) write_hit(p, slot, (read << 1) | strand, order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0), sa1);
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

template <bool CENSUS>
void launch_text_stage(const DevIndex& X, const BatchedParams& p, int num_sms, cudaStream_t s) {
  const uint32_t cap = p.n_reads;
  if (!cap) return;
  count_launches(7);
  text_head_kernel<CENSUS><<<dim3((cap + kHeadTpb - 1) / kHeadTpb, 4), kHeadTpb, 0, s>>>(X, p);
  text_read_kernel<<<(cap + kReadTpb - 1) / kReadTpb, kReadTpb, 0, s>>>(X, p);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, text_wide_kernel<CENSUS>, kWideTpb, 0);
  text_wide_kernel<CENSUS><<<(unsigned)(num_sms * std::max(per_sm, 1)), kWideTpb, 0, s>>>(X, p);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, text_branch_kernel<CENSUS>, kWideTpb, 0);
  text_branch_kernel<CENSUS><<<(unsigned)(num_sms * std::max(per_sm, 1)), kWideTpb, 0, s>>>(X, p);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, text_rows_kernel, kRowsTpb, 0);
  text_rows_kernel<<<(unsigned)(num_sms * std::max(per_sm, 1)), kRowsTpb, 0, s>>>(X, p);
  text_walk_kernel<CENSUS><<<(unsigned)std::min<uint64_t>((4ull * cap + kWalkTpb - 1) / kWalkTpb, 8ull * num_sms),
                             kWalkTpb, 0, s>>>(X, p);
  text_block_kernel<CENSUS><<<(unsigned)num_sms, kWalkTpb, 0, s>>>(X, p);
}

}  // namespace

// Entries of the walk queue: four a read and the chunk tails of the branch kernel's lanes; walks
// that find it full go on by rank steps.
static size_t text_walk_cap(size_t n_reads, int num_sms) {
  return std::min<size_t>(4 * n_reads + (size_t)num_sms * 2048 * kResChunk, (1u << 28) - 1);
}

size_t text_queue_bytes(size_t n_reads, int num_sms) {
  return (8 * n_reads + text_walk_cap(n_reads, num_sms)) * sizeof(uint4) + 4 * n_reads * sizeof(uint32_t);
}

void text_queues(BatchedParams& p, void* buffer, size_t n_reads, int num_sms) {
  p.rows = static_cast<uint4*>(buffer);
  p.rest = p.rows + 4 * n_reads;
  p.walk = p.rest + 4 * n_reads;
  p.walk_cap = (uint32_t)text_walk_cap(n_reads, num_sms);
  p.diag = reinterpret_cast<uint32_t*>(p.walk + p.walk_cap);
}

void launch_text_exact(const DevIndex& X, const BatchedParams& p, cudaStream_t s) {
  if (!p.n_reads) return;
  count_launches(1);
  const dim3 grid((p.n_reads + kHeadTpb - 1) / kHeadTpb, 2);
  if (p.census) text_exact_kernel<true><<<grid, kHeadTpb, 0, s>>>(X, p);
  else text_exact_kernel<false><<<grid, kHeadTpb, 0, s>>>(X, p);
}

void launch_text_search(const DevIndex& X, const BatchedParams& p, int num_sms, cudaStream_t s) {
  if (p.census) launch_text_stage<true>(X, p, num_sms, s);
  else launch_text_stage<false>(X, p, num_sms, s);
}

}  // namespace hpgbwt
