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
// Three launches:
//   text_head_kernel    a thread per chain: start table, then rank steps until
//                       the interval is empty, has stayed one row for a step
//                       (-> finish queue), or is still several rows where the
//                       helper branches or after kHeadSymbols (-> rest list)
//   text_rest_kernel    persistent warps: the chains still several rows wide and
//                       their change points, one rank step per lane and
//                       iteration; what narrows to one row -> finish queue
//   text_finish_kernel  a thread per queued one-row search: SA, comparison,
//                       inverse SA, hits
//
// Positions are counted in search order: symbol i of a chain is W[len-1-i]
// (backward) or W[i] (forward), complemented on the '-' strand, so both
// directions and strands run the same code; J of the helper is len - t
// (backward) or t - 1 (forward) for an interval of t matched symbols, and its
// order key's t field is len - t in both.
//
// Bound by random 32-byte sectors, as rank walks are, but about 26 a read of
// 100 bp at 100 Mbp against 180.  Search stage there on 2M reads 3704 -> 1165 us;
// 4M reads of 36-250 bp 12570 -> 2333 us; 1000 reads of 50-300 bp 510 -> 98 us (a
// chain is some 8 dependent accesses, whatever its length); 2M x 150 bp on a
// 600 Mbp genome with 45 % repeats 9809 -> 8390 us, most of it the rest kernel's
// change points.  Indexes without the arrays, and batches above kTextMaxReads
// (the queues' counters), take the warp-cooperative form (wave.cu).
#include <cuda_runtime.h>

#include <algorithm>

#include "batched.cuh"
#include "batched_dev.cuh"
#include "kernels.cuh"

namespace hpgbwt {

namespace {

using namespace bdev;

constexpr int kHeadTpb = 256, kFinishTpb = 256, kRestTpb = 128;
constexpr int kRestWarps = kRestTpb / 32;
constexpr uint32_t kRestStack = 64;   // change points per warp
constexpr uint32_t kHeadSymbols = 28; // symbols a head matches at most (it holds 32)
constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t kNoKey = 0xFFFFFFFFu;  // of a queue entry: a chain, not a branch walk

// 32 symbols of a 2-bit stream from symbol i on (i may be -31 or reach past the
// end by as much: the streams are padded), symbol i in the low bits.
__device__ __forceinline__ uint64_t load32(const uint64_t* s, int64_t i) {
  const int64_t w = i >> 5;
  const uint32_t sh = ((uint32_t)i & 31u) << 1;
  const uint64_t a = __ldg(s + w);
  return sh ? (a >> sh) | (__ldg(s + w + 1) << (64 - sh)) : a;
}

// The 32 symbols in reverse order.
__device__ __forceinline__ uint64_t rev32(uint64_t x) {
  const uint64_t r = __brevll(x);
  return ((r & 0x5555555555555555ull) << 1) | ((r >> 1) & 0x5555555555555555ull);
}

__device__ __forceinline__ uint64_t comp_word(const DevIndex& X, uint32_t strand) {
  return strand ? 0x5555555555555555ull * X.comp_xor : 0ull;
}

// Symbols i .. i+31 of a chain (past the read's end: whatever the stream holds), symbol i in the low bits.
__device__ __forceinline__ uint64_t query32(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len,
                                            bool fwd, uint32_t strand, int i) {
  const uint64_t x = fwd ? load32(packed, (int64_t)b0 + i) : rev32(load32(packed, (int64_t)b0 + len - 32 - i));
  return x ^ comp_word(X, strand);
}

// How many of the symbols i .. i+want-1 of a chain agree with the text read
// leftwards from position P of physical direction d (whose next symbol is
// T_d[P-1]); want <= P.  Text words and query words are taken in the query's
// order in the stream, so that at most the text word is reversed.
__device__ __forceinline__ int agree(const DevIndex& X, const uint64_t* packed, uint64_t b0, int len, bool fwd,
                                     uint32_t strand, uint32_t d, int i, uint32_t P, int want) {
  const uint64_t cw = comp_word(X, strand);
  for (int m = 0; m < want; m += 32) {
    // the text's next 32 symbols: text[P-1], text[P-2], ... (d = 0) or text[n-P], text[n-P+1], ... (d = 1)
    uint64_t tw = d ? load32(X.text, (int64_t)(X.top - P) + m) : load32(X.text, (int64_t)P - 32 - m);
    const uint64_t qw =
        (fwd ? load32(packed, (int64_t)b0 + i + m) : load32(packed, (int64_t)b0 + len - 32 - i - m)) ^ cw;
    if (fwd != (d != 0)) tw = rev32(tw);
    const uint64_t x = tw ^ qw;
    const int same = x == 0 ? 32 : (fwd ? __ffsll((long long)x) - 1 : __clzll((long long)x)) >> 1;
    if (same < 32) return min(want, m + same);
  }
  return want;
}

// One rank step on a physical symbol.
__device__ __forceinline__ void rank_step(const DevIndex& X, const OccBlock* occ, uint32_t dollar, uint32_t ph,
                                          uint32_t& k, uint32_t& l) {
  const uint32_t q0 = k >> 6, q1 = l >> 6;
  uint32_t cnt[4];
  uint4 bits;
  load_block_m(occ + q0, X.load_mode, cnt, bits);
  uint64_t mm = match_mask(bits, ph);
  const uint32_t c0 = sel4(cnt, ph);
  uint32_t rk = c0 + (uint32_t)__popcll(mm & row_mask(k & 63));
  uint32_t rl;
  if (q1 == q0) {
    rl = c0 + (uint32_t)__popcll(mm & row_mask((l & 63) + 1));
  } else {
    load_block_m(occ + q1, X.load_mode, cnt, bits);
    mm = match_mask(bits, ph);
    rl = sel4(cnt, ph) + (uint32_t)__popcll(mm & row_mask((l & 63) + 1));
  }
  if (ph == 0) {  // the '$' row is stored as code 0 in its block
    if (k > dollar && q0 == (dollar >> 6)) rk -= 1;
    if (l >= dollar && q1 == (dollar >> 6)) rl -= 1;
  }
  const uint32_t cc = sel4(X.C, ph);  // C1 = C + 1 (checked when the index is loaded)
  k = cc + 1u + rk;
  l = cc + rl;
}

// First t at which the helper branches: J <= n/2 backward, J >= n/2 - 1 forward (n = len - 1).
__device__ __forceinline__ int branch_from(int len, bool fwd) {
  const int half = (len - 1) / 2;
  return fwd ? half : len - half;
}

// The block entry (j = 1 / j = n-1) for the fused drain.
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

// Queue entries: x = row (finish) or k (rest), y = l (rest) or order key (finish),
// z = rs, w = symbols matched | forward << 16.

// blockIdx.y 0, 1: the chains on the backward index ('+' backward, '-' forward),
// 2, 3: those on the forward index ('+' forward, '-' backward), so that the
// blocks in flight read one direction's table and blocks at a time.
template <bool CENSUS>
__global__ void __launch_bounds__(kHeadTpb) text_head_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[2][kHeadTpb / 32], s_base[2];
  const uint32_t n_reads = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  if ((uint64_t)blockIdx.x * kHeadTpb >= n_reads) return;
  const uint32_t read = blockIdx.x * kHeadTpb + threadIdx.x;
  const uint32_t d = blockIdx.y >> 1, strand = blockIdx.y & 1u;
  const bool fwd = (d ^ strand) != 0;
  uint32_t dest = 0, sectors = 0;  // 1: finish queue, 2: rest list
  uint4 e = make_uint4(0, 0, 0, 0);
  if (read < n_reads && p.ok[read]) {
    const uint64_t b0 = p.offs[read], b1 = p.offs[read + 1];
    if (b1 >= b0 + 3 && b1 - b0 <= 32767 && b1 <= p.packed_len) {
      const int len = (int)(b1 - b0);
      const OccBlock* occ = d ? X.dir[1].occ : X.dir[0].occ;
      const uint32_t dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
      uint64_t q = query32(X, p.packed, b0, len, fwd, strand, 0);
      const int L = (int)X.kmer_len;
      uint32_t k = 0, l = X.top;
      int t = 0;
      if (L && len >= 2 * L + 2) {
        // the first L steps from the full interval reach no branching position: one lookup
        const uint32_t r = __brev((uint32_t)q) >> (32 - 2 * L);
        const uint2 s = __ldg((d ? X.kmer[1] : X.kmer[0]) +
                              (((r & 0x55555555u) << 1) | ((r >> 1) & 0x55555555u)));
        if (CENSUS) ++sectors;
        k = s.x;
        l = s.y;
        t = L;
        q >>= 2 * L;
      }
      const int ts = branch_from(len, fwd);
      while (k <= l) {
        if (t == len - 1 || t >= (int)kHeadSymbols) {  // the last symbol, or still several rows
          dest = 2;
          e = make_uint4(k, l, 0, (uint32_t)t);
          break;
        }
        const uint32_t pk = k, pl = l;
        if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
        rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
        if (t >= ts && l - k != pl - pk) {  // a change point
          dest = pk == pl ? 1 : 2;
          e = make_uint4(pk, pk == pl ? kNoKey : pl, 0, (uint32_t)t);
          break;
        }
        ++t;
        q >>= 2;
        if (k == l && pk == pl) {  // one row that has matched on: not a chance match about to end
          dest = 1;
          e = make_uint4(k, kNoKey, 0, (uint32_t)t);
          break;
        }
      }
      e.z = (read << 1) | strand;
      e.w |= fwd ? 1u << 16 : 0u;
    }
  }
  // the block's entries appended with one atomic per queue
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
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
    s_base[threadIdx.x] = tot ? atomicAdd(threadIdx.x ? p.rest_n : p.fin_n, tot) : 0u;
  }
  __syncthreads();
  if (dest == 1) {  // (the queue holds one entry per chain and more: no bound to check)
    p.fin[s_base[0] + s_cnt[0][warp] + (uint32_t)__popc(m1 & ((1u << lane) - 1u))] = e;
  } else if (dest == 2) {
    p.rest[s_base[1] + s_cnt[1][warp] + (uint32_t)__popc(m2 & ((1u << lane) - 1u))] = e;
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

struct RestShared {
  uint4 stk[kRestStack];  // change points: k, l, rs, t | forward << 16
  unsigned top;
};

// Persistent: a lane runs one chain or one branch walk, a rank step per
// iteration.  Idle lanes wait, masked, until `batch_idle` of the warp are idle
// and are handed work together: eight lanes per stacked change point (its eight
// continuations share the interval's one or two blocks, so their first step is
// one or two sectors for all), then chains of the rest list; with `spilled` set
// the change points of the spill queue instead of chains.
template <bool CENSUS>
__global__ void __launch_bounds__(kRestTpb, 8) text_rest_kernel(DevIndex X, BatchedParams p, int spilled) {
  __shared__ RestShared rsh[kRestWarps];
  __shared__ uint32_t c_res[kRestTpb], c_spl[kRestTpb], c_fin[kRestTpb];
  const int tid = threadIdx.x;
  const uint32_t lane = tid & 31;
  RestShared& ws = rsh[tid >> 5];
  const uint32_t n_src = spilled ? min(*(volatile unsigned int*)p.spill_tail, p.spill_cap)
                                 : *(volatile unsigned int*)p.rest_n;
  unsigned int* src_ctr = spilled ? p.spill_head : p.rest_head;
  c_res[tid] = c_spl[tid] = c_fin[tid] = 0;
  if (lane == 0) ws.top = 0;
  __syncwarp();
  bool active = false, exhausted = false, fin_full = false;
  uint32_t k = 0, l = 0, rs = 0, key = kNoKey;
  int t = 0, len = 0;
  bool fwd = false;
  uint64_t q = 0;  // the next symbols
  int ql = 0;      // how many q holds
  const OccBlock* occ = nullptr;
  uint32_t dollar = 0, sectors = 0;

  // The item's read, direction and symbols from symbol t on.
  auto open_item = [&](uint32_t rs_, bool fwd_, int t_) {
    rs = rs_;
    fwd = fwd_;
    t = t_;
    const uint64_t b0 = p.offs[rs >> 1];
    len = (int)(p.offs[(rs >> 1) + 1] - b0);
    const uint32_t strand = rs & 1u, d = (fwd ? 1u : 0u) ^ strand;
    occ = d ? X.dir[1].occ : X.dir[0].occ;
    dollar = d ? X.dir[1].dollar : X.dir[0].dollar;
    q = query32(X, p.packed, b0, len, fwd, strand, t);
    ql = 32;
    active = true;
  };
  // Continuation `item` (0..7) of change point e, as listed at wave_branch_kernel.
  auto start_walk = [&](const uint4& e, uint32_t item) {
    const int te = (int)(e.w & 0xFFFFu);
    k = e.x;
    l = e.y;
    // deletion and mismatch go on after symbol te, the insertion with it
    const bool ins = item >= 1 && item <= 4;
    open_item(e.z, (e.w >> 16) & 1u, ins ? te : te + 1);
    uint32_t slot = 0;
    if (item) {
      uint32_t b;
      const uint32_t cx = (rs & 1u) ? X.comp_xor : 0u;
      if (ins) {
        b = item - 1;
        slot = 1 + 2 * b;
      } else {
        const uint64_t b0 = p.offs[rs >> 1];
        const uint32_t w = (uint32_t)load32(p.packed, fwd ? (int64_t)b0 + te : (int64_t)b0 + len - 1 - te) & 3u;
        b = (item - 5) + ((item - 5) >= w ? 1u : 0u);
        slot = 2 + 2 * b;
      }
      // b is stepped first, in the place of the symbol before t (the symbol that
      // falls out of q is fetched again when q runs out)
      q = (q << 2) | (b ^ cx);
      --t;
    }
    key = order_key(fwd ? 4u : 2u, (uint32_t)(len - te), slot);
  };
  auto refill = [&]() {
    for (;;) {
      __syncwarp();
      const unsigned nd = __ballot_sync(kFull, !active);
      if (!nd) return;
      const uint32_t rank = (uint32_t)__popc(nd & ((1u << lane) - 1u));
      const uint32_t n_nd = (uint32_t)__popc(nd);
      const unsigned top = min(ws.top, kRestStack);  // pushes past the end went to the spill queue
      if (top && n_nd >= 8) {
        const uint32_t take = min(n_nd >> 3, top);
        __syncwarp();
        if (!active && (rank >> 3) < take) start_walk(ws.stk[top - 1 - (rank >> 3)], rank & 7u);
        __syncwarp();
        if (lane == 0) ws.top = top - take;
        __syncwarp();
        continue;
      }
      if (exhausted || (spilled && n_nd < 8)) return;
      const uint32_t want = spilled ? n_nd >> 3 : n_nd;
      uint32_t c0 = 0;
      if (lane == 0) c0 = atomicAdd(src_ctr, want);
      c0 = __shfl_sync(kFull, c0, 0);
      if (c0 + want >= n_src) exhausted = true;
      if (spilled) {
        if (!active && (rank >> 3) < want && c0 + (rank >> 3) < n_src) {
          const SpillEntry s = p.spill[c0 + (rank >> 3)];
          if (s.rs != 0xFFFFFFFFu) start_walk(make_uint4(s.k, s.l, s.rs, s.jtype), rank & 7u);
        }
      } else if (!active && c0 + rank < n_src) {
        const uint4 e = p.rest[c0 + rank];
        k = e.x;
        l = e.y;
        key = kNoKey;
        open_item(e.z, (e.w >> 16) & 1u, (int)(e.w & 0xFFFFu));
      }
      __syncwarp();
      // (one claim a pass: lanes left idle by holes or by the list's end wait for the next)
      return;
    }
  };

  const uint32_t bi = p.batch_idle < 8 ? 8u : p.batch_idle;
  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !active);  // every lane, every iteration
    if (idle == kFull || (uint32_t)__popc(idle) >= bi) {
      refill();
      __syncwarp();
      if (__ballot_sync(kFull, !active) == kFull && exhausted && ws.top == 0) break;
    }
    if (!active) continue;
    const uint32_t pk = k, pl = l;
    if (CENSUS) sectors += (k >> 6) == (l >> 6) ? 1u : 2u;
    rank_step(X, occ, dollar, (uint32_t)q & 3u, k, l);
    const bool walk = key != kNoKey;
    if (!walk && l - k != pl - pk && t >= branch_from(len, fwd)) {  // a change point
      if (t == len - 1) {
        push_block(p, pk, pl, rs, len, fwd);
      } else {
        const uint32_t w = (uint32_t)t | (fwd ? 1u << 16 : 0u);
        const unsigned at = atomicAdd(&ws.top, 1u);
        if (at < kRestStack) {
          ws.stk[at] = make_uint4(pk, pl, rs, w);
        } else {  // in chunks of slots
          uint32_t cs = c_spl[tid];
          unsigned slot;
          if ((cs >> 28) == 0) {
            cs = claim(p.spill_tail, kResChunk);
            if (cs >= (1u << 28) - kResChunk) {  // beyond what the packed form holds
              slot = cs;
              cs = 0;
              for (unsigned i = 1; i < kResChunk; ++i)
                if (slot + i < p.spill_cap) p.spill[slot + i].rs = 0xFFFFFFFFu;
            } else {
              slot = cs;
              cs = (cs + 1) | ((kResChunk - 1) << 28);
            }
          } else {
            slot = cs & 0x0FFFFFFFu;
            cs = (slot + 1) | (((cs >> 28) - 1) << 28);
          }
          c_spl[tid] = cs;
          if (slot < p.spill_cap) p.spill[slot] = SpillEntry{pk, pl, rs, w};
          else atomicOr(p.status, kStatusSpillFull);
        }
      }
    }
    if (k <= l && t + 1 < len) {
      ++t;
      q >>= 2;
      if (k == l && pk == pl && !fin_full) {  // one row that has matched on: the text tells the rest
        uint32_t cs = c_fin[tid];
        if ((cs >> 28) == 0) {
          cs = claim(p.fin_n, kResChunk);
          if (cs >= (1u << 28) - kResChunk || cs + kResChunk > p.fin_cap) {
            for (unsigned i = 0; i < kResChunk; ++i)
              if (cs + i < p.fin_cap) p.fin[cs + i].z = 0xFFFFFFFFu;
            fin_full = true;  // this lane's searches go on by rank steps
            cs = 0;
          } else {
            cs |= kResChunk << 28;
          }
        }
        if (!fin_full) {
          const unsigned slot = cs & 0x0FFFFFFFu;
          p.fin[slot] = make_uint4(k, key, rs, (uint32_t)t | (fwd ? 1u << 16 : 0u));
          cs = (slot + 1) | (((cs >> 28) - 1) << 28);
          active = false;
        }
        c_fin[tid] = cs;
        if (!active) continue;
      }
      if (--ql == 0) {  // 32 symbols on
        const uint64_t b0 = p.offs[rs >> 1];
        q = query32(X, p.packed, b0, len, fwd, rs & 1u, t);
        ql = 32;
      }
      continue;
    }
    if (k <= l && (walk || !fwd)) {  // matched to the read end: a branch's hit, or the exact hit
      uint32_t r = c_res[tid];
      const unsigned slot = res_slot(p, r);
      c_res[tid] = r;
      if (walk) {
        const uint32_t s = key & 0xFFu;
        const int te = len - (int)((key >> 8) & 0xFFFFu);
        const uint32_t kind = s == 0 ? 1u : ((s & 1u) ? 3u : 2u);
        write_hit(p, slot, rs, key, k, l, branch_meta(fwd, len, te, kind, s == 0 ? 0xFFu : (s - 1) >> 1));
      } else {
        write_hit(p, slot, rs, order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0));
      }
    }
    active = false;
  }
  {  // slots of this lane's last chunks that were reserved but not used
    const uint32_t r = c_res[tid];
    for (unsigned i = 0, left = r >> 28, slot = r & 0x0FFFFFFFu; i < left; ++i)
      if (slot + i < p.res_cap) p.res[slot + i].rs = 0xFFFFFFFFu;
    const uint32_t cs = c_spl[tid];
    for (unsigned i = 0, left = cs >> 28, s = cs & 0x0FFFFFFFu; i < left; ++i)
      if (s + i < p.spill_cap) p.spill[s + i].rs = 0xFFFFFFFFu;
    const uint32_t cf = c_fin[tid];
    for (unsigned i = 0, left = cf >> 28, s = cf & 0x0FFFFFFFu; i < left; ++i)
      if (s + i < p.fin_cap) p.fin[s + i].z = 0xFFFFFFFFu;
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// A thread per queued one-row search; up to three hits each, appended with one
// atomic per block and round.
template <bool CENSUS>
__global__ void __launch_bounds__(kFinishTpb) text_finish_kernel(DevIndex X, BatchedParams p) {
  __shared__ uint32_t s_cnt[kFinishTpb / 32], s_base;
  const uint32_t n = min(*(volatile unsigned int*)p.fin_n, p.fin_cap);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t sectors = 0;
  for (uint32_t i0 = blockIdx.x * kFinishTpb; i0 < n; i0 += gridDim.x * kFinishTpb) {
    const uint32_t i = i0 + threadIdx.x;
    uint32_t rs = 0, key = 0, meta = 0;
    uint32_t at[3] = {0, 0, 0};  // SA^-1 index of: the exact hit, the walk's hit or the deletion; the insertion; the mismatch
    uint32_t mask = 0;           // which of them match
    uint32_t d = 0, ins_key = 0, ins_meta = 0, mis_meta = 0;
    uint4 e = make_uint4(0, 0, 0xFFFFFFFFu, 0);
    if (i < n) e = __ldcs(p.fin + i);
    if (e.z != 0xFFFFFFFFu) {  // (a reserved slot nothing was written to)
      rs = e.z;
      const uint32_t strand = rs & 1u;
      const bool fwd = (e.w >> 16) & 1u;
      d = (fwd ? 1u : 0u) ^ strand;
      const uint32_t P = load_row_word((d ? X.dir[1].sa : X.dir[0].sa) + e.x);
      const uint64_t b0 = p.offs[rs >> 1];
      const int len = (int)(p.offs[(rs >> 1) + 1] - b0);
      const int t = (int)(e.w & 0xFFFFu), left = len - t;
      const int m = agree(X, p.packed, b0, len, fwd, strand, d, t, P, (int)min((uint32_t)left, P));
      const uint32_t Q = P - (uint32_t)m;
      if (CENSUS) sectors += 2u + (uint32_t)(m >> 7);
      if (e.y != kNoKey) {  // a branch walk
        if (m == left) {
          const uint32_t s = e.y & 0xFFu;
          mask = 1;
          at[0] = Q;
          key = e.y;
          meta = branch_meta(fwd, len, len - (int)((e.y >> 8) & 0xFFFFu), s == 0 ? 1u : ((s & 1u) ? 3u : 2u),
                             s == 0 ? 0xFFu : (s - 1) >> 1);
        }
      } else if (m == left) {  // the whole read: the exact hit, reported by the backward chain
        if (!fwd) {
          mask = 1;
          at[0] = Q;
          key = order_key(0, 0, 0);
          meta = pack_meta(0, 0, 0, 0, 0);
        }
      } else {
        const int te = t + m;  // the symbol that fails
        if (te == len - 1) {
          const uint32_t r = load_row_word((d ? X.dir[1].isa : X.dir[0].isa) + Q);
          push_block(p, r, r, rs, len, fwd);
        } else if (te >= branch_from(len, fwd)) {
          const int after = len - te - 1;  // symbols after the failing one
          key = order_key(fwd ? 4u : 2u, (uint32_t)(len - te), 0);
          if (Q >= (uint32_t)after && agree(X, p.packed, b0, len, fwd, strand, d, te + 1, Q, after) == after) {
            mask = 1;
            at[0] = Q - (uint32_t)after;
            meta = branch_meta(fwd, len, te, 1, 0xFFu);
          }
          if (Q >= 1) {
            // the text's next symbol, as a query base: the one insertion and the one mismatch that match it
            const uint64_t tw = d ? load32(X.text, (int64_t)(X.top - Q)) : load32(X.text, (int64_t)Q - 1);
            const uint32_t b = ((uint32_t)tw & 3u) ^ (strand ? X.comp_xor : 0u);
            const uint32_t R = Q - 1;
            ins_key = key + 1 + 2 * b;
            ins_meta = branch_meta(fwd, len, te, 3, b);
            mis_meta = branch_meta(fwd, len, te, 2, b);
            if (R >= (uint32_t)after + 1 &&
                agree(X, p.packed, b0, len, fwd, strand, d, te, R, after + 1) == after + 1) {
              mask |= 2;
              at[1] = R - (uint32_t)after - 1;
            }
            if (R >= (uint32_t)after && agree(X, p.packed, b0, len, fwd, strand, d, te + 1, R, after) == after) {
              mask |= 4;
              at[2] = R - (uint32_t)after;
            }
          }
        }
      }
    }
    uint32_t row[3];
    const uint32_t* isa = d ? X.dir[1].isa : X.dir[0].isa;
#pragma unroll
    for (int h = 0; h < 3; ++h) row[h] = (mask >> h) & 1u ? load_row_word(isa + at[h]) : 0u;
    const uint32_t n_hits = (uint32_t)__popc(mask);
    if (CENSUS) sectors += n_hits;
    // slots of the block's hits
    uint32_t incl = n_hits;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, incl, o);
      if (lane >= (uint32_t)o) incl += v;
    }
    if (lane == 31) s_cnt[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t tot = 0;
      for (int w = 0; w < kFinishTpb / 32; ++w) {
        const uint32_t c = s_cnt[w];
        s_cnt[w] = tot;
        tot += c;
      }
      s_base = tot ? atomicAdd(p.res_total, tot) : 0u;
    }
    __syncthreads();
    uint32_t slot = s_base + s_cnt[warp] + incl - n_hits;
    if (mask & 1u) write_hit(p, slot++, rs, key, row[0], row[0], meta);
    if (mask & 2u) write_hit(p, slot++, rs, ins_key, row[1], row[1], ins_meta);
    if (mask & 4u) write_hit(p, slot, rs, ins_key + 1, row[2], row[2], mis_meta);
    __syncthreads();  // s_cnt and s_base are rewritten next round
  }
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

template <bool CENSUS>
void launch_text_stage(const DevIndex& X, const BatchedParams& p, int num_sms, cudaStream_t s) {
  const uint32_t cap = p.n_reads;
  if (!cap) return;
  count_launches(4);
  text_head_kernel<CENSUS><<<dim3((cap + kHeadTpb - 1) / kHeadTpb, 4), kHeadTpb, 0, s>>>(X, p);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, text_rest_kernel<CENSUS>, kRestTpb, 0);
  const unsigned rest_grid = (unsigned)(num_sms * std::max(per_sm, 1));
  text_rest_kernel<CENSUS><<<rest_grid, kRestTpb, 0, s>>>(X, p, 0);
  text_rest_kernel<CENSUS><<<rest_grid, kRestTpb, 0, s>>>(X, p, 1);
  text_finish_kernel<CENSUS><<<(unsigned)std::min<uint64_t>((4ull * cap + kFinishTpb - 1) / kFinishTpb,
                                                            8ull * num_sms),
                               kFinishTpb, 0, s>>>(X, p);
}

}  // namespace

// Entries of the finish queue: one per chain, as many again for branch walks, and the chunk
// tails of the rest kernel's lanes.
size_t text_fin_cap(size_t n_reads, int num_sms) {
  return std::min<size_t>(8 * n_reads + (size_t)num_sms * 2048 * kResChunk, (1u << 28) - 1);
}

void launch_text_search(const DevIndex& X, const BatchedParams& p, int num_sms, cudaStream_t s) {
  if (p.census) launch_text_stage<true>(X, p, num_sms, s);
  else launch_text_stage<false>(X, p, num_sms, s);
}

}  // namespace hpgbwt
