// batched.cu -- persistent work-queue search, ordered finalize and persistent
// locate of the batched pipeline form.
#include <cooperative_groups.h>
#include <cooperative_groups/scan.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "batched.cuh"
#include "batched_dev.cuh"
#include "kernels.cuh"
#include "search_core.cuh"

namespace cg = cooperative_groups;

namespace hpgbwt {

namespace {

constexpr int kBlock = 128;

using namespace bdev;

// Next read of a chain set (part 0: the chains on the backward index, 1: those
// on the forward index, 2: all four), aggregated per warp and per set.
__device__ __forceinline__ unsigned claim_part(const BatchedParams& p, uint32_t part) {
  cg::coalesced_group g = cg::coalesced_threads();
  cg::coalesced_group sub = cg::labeled_partition(g, part);
  unsigned base = 0;
  if (sub.thread_rank() == 0) base = atomicAdd(part == 1 ? p.chain_ctr2 : p.chain_ctr, (unsigned)sub.size());
  return sub.shfl(base, 0) + sub.thread_rank();
}

__device__ __forceinline__ uint32_t sm_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
  return r;
}

template <int D, int MINB, bool CENSUS>
__global__ void __launch_bounds__(kBlock, MINB) batched_search_kernel(DevIndex X, BatchedParams p, int drain,
                                                                      int chunk) {
  __shared__ uint32_t stk_k[D][kBlock], stk_l[D][kBlock], stk_j[D][kBlock];
  __shared__ uint32_t c_ek[kBlock], c_el[kBlock], c_meta[kBlock], c_misc[kBlock], c_res[kBlock], c_part[kBlock];
  __shared__ uint32_t c_read[kBlock];  // read whose chains this lane runs
  __shared__ uint32_t s_nreads, s_spill_end;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_nreads = p.read_list ? min(*p.read_list_n, p.long_cap) : (p.n_reads_dev ? *p.n_reads_dev : p.n_reads);
    s_spill_end = drain ? min(*(volatile unsigned int*)p.spill_tail, p.spill_cap) : 0u;
  }
  c_meta[tid] = 0;
  c_misc[tid] = 4u << 4;  // no chain of a read left
  c_res[tid] = 0;
  __syncthreads();

  // hot state
  uint32_t rs = 0;                  // 2 * read + strand
  const uint8_t* W = nullptr;
  int len = 0;
  uint32_t k = 0, l = 0;            // interval of the pending / last step
  uint32_t pk = 0, pl = 0;          // chain: previous interval; entry: aux interval
  int pos = 0, dir = 0;             // read position of the pending step; -1 backward, +1 forward
  uint32_t nb = 0;                  // base of the pending step
  uint32_t mode = kNone;
  uint32_t win = 0;                 // chain: first J where the helper branches | how many J (<< 16)
  uint32_t sectors = 0;
  // read-level work: the current read's next chain, and the next read claimed
  // and its offsets fetched ahead of time (their loads complete while the
  // current read is searched)
  // With the direction split, SMs of the first half take the two chains of a
  // read that run on the backward index ('+' backward, '-' forward) and the
  // others the two on the forward index ('+' forward, '-' backward): every
  // chain and its branches stay on one index direction, so each half's L2
  // holds one direction's blocks.  A half that runs out takes the other's reads.
  // (claim state in shared memory, touched once per read: bits 0-1 the chain
  // set being claimed, bit 2 set once it moved to the other half's reads,
  // bits 3-4 the set of the current read, bits 5-6 that of the prefetched one)
  {
    const uint32_t part0 = p.dir_split == 1 ? (sm_id() >= p.num_sms / 2 ? 1u : 0u)
                                             : (p.dir_split == 2 ? 0u : (p.dir_split == 3 ? 1u : 2u));
    c_part[tid] = part0 | (part0 << 3) | (part0 << 5);
  }
  // The claim state (read, chain of the read, chain set) lives in shared
  // memory: a lane touches it once per chain, and the registers it frees let
  // more blocks stay resident.  A read's offsets are loaded when it is claimed.
  auto next_claim = [&]() -> uint32_t {
    uint32_t st = c_part[tid];
    for (;;) {
      const uint32_t part = st & 3u;
      const uint32_t r = claim_part(p, part);
      if (r < s_nreads || part == 2u || (st & 4u) || p.dir_split != 1) {
        c_part[tid] = (st & ~(3u << 3)) | (part << 3);
        return r;
      }
      st = (st & ~3u) | (part ^ 1u) | 4u;
    }
  };
  (void)chunk;

  auto push = [&](uint32_t a, uint32_t b, uint32_t jt) {
    const uint32_t misc = c_misc[tid];
    const uint32_t sp = misc & 15u;
    if (sp < (uint32_t)D) {
      stk_k[sp][tid] = a;
      stk_l[sp][tid] = b;
      stk_j[sp][tid] = jt;
      c_misc[tid] = misc + 1;
    } else {
      const unsigned s = claim(p.spill_tail, 1);
      if (s < p.spill_cap) p.spill[s] = SpillEntry{a, b, rs, jt};
      else atomicOr(p.status, kStatusSpillFull);
    }
  };
  // Result of a continuation search that matched to the read end.
  auto emit = [&](uint32_t key, uint32_t a, uint32_t b, uint32_t meta) {
    uint32_t r = c_res[tid];
    const unsigned slot = res_slot(p, r);
    c_res[tid] = r;
    write_hit(p, slot, rs, key, a, b, meta);
  };
  auto emit_cont = [&](uint32_t m) {
    const uint32_t ej = meta_j(m), sub = meta_sub(m);
    const bool bwd = meta_type(m) == kCpBwd;
    const uint32_t b = sub == 0 ? 0u : (sub - 1) / 3;
    const bool ins = sub != 0 && (sub - 1) % 3 == 1;
    const uint32_t kind = sub == 0 ? 1u : (ins ? 3u : 2u);
    const uint32_t slot = sub == 0 ? 0u : (ins ? 1u + 2 * b : 2u + 2 * b);
    const uint32_t basev = sub == 0 ? 0xFFu : b;
    if (bwd)
      emit(order_key(2, ej, slot), k, l, pack_meta(0, 1, kind, basev, (int32_t)ej - 1));
    else
      emit(order_key(4, (uint32_t)(len - 1 - (int)ej), slot), k, l,
               pack_meta(1, 1, kind, basev, (int32_t)ej + 1));
  };

  for (;;) {
    // ---- transitions: next sub-operation, next change point, next chain ----
    // A lane out of work waits (riding along masked) until p.batch_idle lanes
    // of its converged group are out of work too, or all of them are, so the
    // transition code runs for many lanes at once instead of one at a time.
    bool go = mode == kNone;
    if (p.batch_idle > 1) {
      const unsigned grp = __activemask();
      const unsigned idle = __ballot_sync(grp, mode == kNone);
      go = go && ((uint32_t)__popc(idle) >= p.batch_idle || idle == grp);
    }
    if (go) {
    while (mode == kNone) {
      uint32_t m = c_meta[tid];
      if (meta_in(m)) {
        const uint32_t sub = meta_sub(m), etype = meta_type(m), ej = meta_j(m);
        if (sub >= kSubEnd) {
          c_meta[tid] = 0;
          continue;
        }
        const bool bwd = (etype == kCpBwd || etype == kBlk1);
        const bool blk = etype >= kBlk1;
        const int end = len - 1;
        dir = bwd ? -1 : 1;
        if (sub == 0) {
          if (blk) {  // the block's direct deletion result
            if (etype == kBlk1)
              emit(order_key(1, 0, 0), c_ek[tid], c_el[tid], pack_meta(0, 1, 1, 0xFF, 0));
            else
              emit(order_key(3, 0, 0), c_ek[tid], c_el[tid], pack_meta(1, 1, 1, 0xFF, end));
            c_meta[tid] = m + (1u << 18);
            continue;
          }
          k = c_ek[tid];
          l = c_el[tid];
          pos = bwd ? (int)ej - 2 : (int)ej + 2;
        } else {
          const uint32_t b = (sub - 1) / 3, r = (sub - 1) % 3;
          if (r == 0) {  // aux step with base b
            k = c_ek[tid];
            l = c_el[tid];
            nb = b;
            mode = kSingle;
            break;
          }
          if (blk) {
            if (r == 1) {  // block insertion: one step with the read's end base
              k = pk;
              l = pl;
              nb = etype == kBlk1 ? W[0] : W[end];
              mode = kSingle;
              break;
            }
            c_meta[tid] = m + (1u << 18);  // blocks emit their mismatch right after the aux step
            continue;
          }
          if (r == 2 && b == W[bwd ? ej - 1 : ej + 1]) {  // no mismatch with the read's own base
            c_meta[tid] = m + (1u << 18);
            continue;
          }
          k = pk;
          l = pl;
          pos = bwd ? (int)ej - (int)r : (int)ej + (int)r;
        }
        if (bwd ? pos < 0 : pos > end) {  // nothing left to match: the interval is the hit
          if (k <= l) emit_cont(m);
          c_meta[tid] = m + (1u << 18);
          continue;
        }
        nb = W[pos];
        mode = kCont;
        break;
      }
      const uint32_t misc = c_misc[tid];
      if (misc & 15u) {  // next change point of this lane's read
        const uint32_t sp = (misc & 15u) - 1;
        c_misc[tid] = misc - 1;
        c_ek[tid] = stk_k[sp][tid];
        c_el[tid] = stk_l[sp][tid];
        const uint32_t jt = stk_j[sp][tid];
        c_meta[tid] = make_meta(jt & 0xFFFFu, jt >> 16, 0, 0, true);
        continue;
      }
      if (drain) {
        const unsigned s = claim(p.spill_head, 1);
        if (s >= s_spill_end) break;
        const SpillEntry e = p.spill[s];
        if (e.rs == 0xFFFFFFFFu) continue;  // reserved but unused slot
        rs = e.rs;
        const uint32_t read = rs >> 1;
        const uint64_t b0 = p.offs[read];
        W = p.codes + b0;
        len = (int)(p.offs[read + 1] - b0);
        c_ek[tid] = e.k;
        c_el[tid] = e.l;
        c_meta[tid] = make_meta(e.jtype & 0xFFFFu, e.jtype >> 16, 0, 0, true);
        continue;
      }
      uint32_t chain = (misc >> 4) & 7u;
      if (chain >= ((((c_part[tid] >> 3) & 3u) == 2u) ? 4u : 2u)) {  // next read
        const uint32_t rc = next_claim();
        if (rc >= s_nreads) break;
        const uint32_t r = p.read_list ? p.read_list[rc] : rc;
        c_read[tid] = r;
        const uint64_t b0 = p.offs[r];
        const int L = (int)(p.offs[r + 1] - b0);
        if (!p.ok[r] || L < 3 || L > 32767) continue;  // no chains for this read (chain stays at its end)
        W = p.codes + b0;
        len = L;
        chain = 0;
      }
      c_misc[tid] = (misc & 15u) | ((chain + 1) << 4);
      const uint32_t ci = chain;
      const uint32_t cur_read = c_read[tid];
      const uint32_t cur_part = (c_part[tid] >> 3) & 3u;
      // 0: '+' backward, 1: '+' forward, 2: '-' backward, 3: '-' forward
      const uint32_t c = cur_part == 2u ? ci : (cur_part == 0u ? (ci ? 3u : 0u) : (ci ? 2u : 1u));
      rs = (cur_read << 1) | (c >> 1);
      k = 0;
      l = X.top;
      pk = 0;
      pl = X.top;
      dir = (c & 1u) ? 1 : -1;
      pos = (c & 1u) ? 0 : len - 1;
      {  // branching positions of this vector search: J in [2, n/2] backward, [n/2 - 1, n - 1] forward
        const int n = len - 1;
        const int lo = dir > 0 ? n / 2 - 1 : 2, hi = dir > 0 ? n - 1 : n / 2;
        win = (uint32_t)lo | ((uint32_t)(hi >= lo ? hi - lo + 1 : 0) << 16);
      }
      const uint32_t L = X.kmer_len;
      if (L && len >= 2 * (int)L + 2) {
        // The first L steps of a chain from the full interval never reach a
        // branching position (J stays above n/2 backward, below n/2 - 1
        // forward): one table lookup stands for them.
        const uint32_t strand = rs & 1u;
        uint32_t code = 0;
        for (uint32_t i = 0; i < L; ++i) {
          const uint32_t b = W[dir > 0 ? (int)i : len - 1 - (int)i];
          code = (code << 2) | (strand ? sel4(X.comp, b) : b);
        }
        nb = code;
        mode = kKmer;
      } else {
        nb = W[pos];
        mode = kChain;
      }
    }
    if (mode == kNone) break;  // no work left for this lane
    }
    if (mode == kNone) continue;  // waiting for more lanes to move on with

    // ---- the one gather of this iteration --------------------------------
    {
      const uint32_t strand = rs & 1u;
      const uint32_t vsel = dir > 0 ? 1u : 0u;  // forward searches use the strand's forward view
      if (mode == kKmer) {
        if (CENSUS) sectors += 1u;
        const uint2 t = __ldg(((vsel ^ strand) ? X.kmer[1] : X.kmer[0]) + nb);
        k = t.x;
        l = t.y;
      } else {
        if (CENSUS) sectors += ((k >> 6) == (l >> 6)) ? 1u : 2u;
        bw_step(X, View{vsel ^ strand, strand}, nb, k, l);
      }
    }
    if (mode == kKmer) {
      if (k > l) {  // failed within the first L steps: no change point, no hit
        mode = kNone;
        continue;
      }
      pk = k;
      pl = l;
      pos = dir > 0 ? (int)X.kmer_len : len - 1 - (int)X.kmer_len;
      nb = W[pos];
      mode = kChain;
      continue;
    }
    if (mode == kChain) {
      // (k,l) = vector entry at pos, (pk,pl) = entry at J = pos - dir.  The helper
      // branches at J in [2, n/2] (backward, block at 1) and [n/2 - 1, n - 2]
      // (forward, block at n - 1).
      const int J = pos - dir;
      const bool differ = (l - k) != (pl - pk);  // sizes are >= -1 here, so 32-bit differences suffice
      if (differ && (uint32_t)(J - (int)(win & 0xFFFFu)) < (win >> 16))
        push(pk, pl, (uint32_t)J | ((dir > 0 ? (J == len - 2 ? kBlkN : kCpFwd) : kCpBwd) << 16));
      if (k <= l && (uint32_t)(pos + dir) < (uint32_t)len) {  // a next base to match
        pk = k;
        pl = l;
        pos += dir;
        nb = W[pos];
        continue;
      }
      if (dir < 0 && pos == 0) {  // backward vector complete: exact hit, then the j = 1 block on vec[1]
        if (k <= l) emit(order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0));
        if (differ) push(pk, pl, 1u | (kBlk1 << 16));
      }
      mode = kNone;
    } else if (mode == kCont) {
      if (k <= l && (uint32_t)(pos + dir) < (uint32_t)len) {
        pos += dir;
        nb = W[pos];
        continue;
      }
      const uint32_t m = c_meta[tid];
      if (k <= l) emit_cont(m);
      c_meta[tid] = m + (1u << 18);
      mode = kNone;
    } else {  // kSingle: an aux step or a block insertion step
      const uint32_t m = c_meta[tid];
      const uint32_t sub = meta_sub(m), etype = meta_type(m);
      const uint32_t b = (sub - 1) / 3;
      if ((sub - 1) % 3 == 0) {
        if (k > l) {
          c_meta[tid] = m + (3u << 18);
        } else {
          pk = k;
          pl = l;
          if (etype >= kBlk1) {
            const int end = len - 1;
            const uint32_t w = etype == kBlk1 ? W[0] : W[end];
            if (b != w) {
              if (etype == kBlk1)
                emit(order_key(1, 0, 1 + 2 * b), k, l, pack_meta(0, 1, 2, b, (int32_t)meta_bpos(m)));
              else
                emit(order_key(3, 0, 1 + 2 * b), k, l, pack_meta(1, 1, 2, b, end));
            }
          }
          c_meta[tid] = m + (1u << 18);
        }
      } else {
        uint32_t nm = m + (2u << 18);
        if (k <= l) {
          if (etype == kBlk1) {
            emit(order_key(1, 0, 2 + 2 * b), k, l, pack_meta(0, 1, 3, 3, (int32_t)b));
            nm = (nm & ~(3u << 22)) | (b << 22);
          } else {
            emit(order_key(3, 0, 2 + 2 * b), k, l, pack_meta(1, 1, 3, b, len - 1));
          }
        }
        c_meta[tid] = nm;
      }
      mode = kNone;
    }
  }
  res_leave(p, c_res[tid]);  // slots of this lane's last chunk that were reserved but not used
  if (CENSUS && p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// Chain-only variant (the "split" form): lanes run only the vector searches,
// with the smallest possible loop, and append every change point to the
// device queue; a drain launch of batched_search_kernel then expands them.
// `phase` 0 runs only the chains on the backward index ('+' backward and '-'
// forward), 1 only those on the forward index ('+' forward, '-' backward), so
// each launch keeps one direction's occurrence blocks hot in L2; 2 runs all.
template <int MINB>
__global__ void __launch_bounds__(kBlock, MINB) chain_kernel(DevIndex X, BatchedParams p, int chunk, int phase) {
  const uint32_t n_reads_ = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  const uint32_t n_chains = (phase == 2 ? 4u : 2u) * n_reads_;
  uint32_t rs = 0;
  const uint8_t* W = nullptr;
  int len = 0;
  uint32_t k = 0, l = 0, pk = 0, pl = 0;
  int pos = 0, dir = 0;
  uint32_t nb = 0;
  bool active = false;
  uint32_t next = 0, left = 0, sectors = 0;
  for (;;) {
    // lanes out of chains wait (masked) until p.batch_idle lanes of the
    // converged group are, or all of them are, and claim the next ones together
    bool go = !active;
    if (p.batch_idle > 1) {
      const unsigned grp = __activemask();
      const unsigned idle = __ballot_sync(grp, !active);
      go = go && ((uint32_t)__popc(idle) >= p.batch_idle || idle == grp);
    }
    if (!go && !active) continue;
    while (!active) {
      if (left == 0) {
        next = claim(p.chain_ctr, (unsigned)chunk);
        left = (unsigned)chunk;
      }
      if (next >= n_chains) break;
      const uint32_t c = next++;
      --left;
      const uint32_t read = phase == 2 ? c >> 2 : c >> 1;
      const uint64_t b0 = p.offs[read];
      const int L = (int)(p.offs[read + 1] - b0);
      if (!p.ok[read] || L < 3 || L > 32767) continue;
      const uint32_t strand = phase == 2 ? (c >> 1) & 1u : c & 1u;
      const bool fwd = phase == 2 ? (c & 1u) != 0 : ((strand ^ (uint32_t)phase) != 0);
      rs = (read << 1) | strand;
      W = p.codes + b0;
      len = L;
      k = 0;
      l = X.top;
      pk = 0;
      pl = X.top;
      dir = fwd ? 1 : -1;
      pos = fwd ? 0 : L - 1;
      const uint32_t KL = X.kmer_len;
      if (KL && L >= 2 * (int)KL + 2) {
        // start table: one lookup for the first KL steps, which reach no
        // branching position (as in the fused kernel)
        uint32_t code = 0;
        for (uint32_t i = 0; i < KL; ++i) {
          const uint32_t b = W[fwd ? (int)i : L - 1 - (int)i];
          code = (code << 2) | (strand ? sel4(X.comp, b) : b);
        }
        const uint2 t = __ldg(((((uint32_t)fwd) ^ strand) ? X.kmer[1] : X.kmer[0]) + code);
        if (p.census) sectors += 1u;
        if (t.x > t.y) continue;  // failed within the first KL steps: no change point, no hit
        k = pk = t.x;
        l = pl = t.y;
        pos = fwd ? (int)KL : L - 1 - (int)KL;
      }
      nb = W[pos];
      active = true;
    }
    if (!active) break;
    const int stop = dir > 0 ? len - 1 : 0;
    // next base, fetched alongside the gather instead of after it
    const uint32_t nb_next = pos != stop ? W[pos + dir] : 0u;
    {
      const uint32_t strand = rs & 1u;
      if (p.census) sectors += ((k >> 6) == (l >> 6)) ? 1u : 2u;
      bw_step(X, View{(dir > 0 ? 1u : 0u) ^ strand, strand}, nb, k, l);
    }
    const int J = pos - dir, n = len - 1;
    const int jlo = dir > 0 ? n / 2 - 1 : 2, jhi = dir > 0 ? n - 1 : n / 2;
    const bool differ = (l - k) != (pl - pk);
    if (differ && J >= jlo && J <= jhi) {
      const uint32_t jt = (uint32_t)J | ((dir > 0 ? (J == n - 1 ? kBlkN : kCpFwd) : kCpBwd) << 16);
      const unsigned s = claim(p.spill_tail, 1);
      if (s < p.spill_cap) p.spill[s] = SpillEntry{pk, pl, rs, jt};
      else atomicOr(p.status, kStatusSpillFull);
    }
    if (k <= l && pos != stop) {
      pk = k;
      pl = l;
      pos += dir;
      nb = nb_next;
      continue;
    }
    if (dir < 0 && pos == 0) {
      if (k <= l) emit_hit(p, rs, order_key(0, 0, 0), k, l, pack_meta(0, 0, 0, 0, 0));
      if (differ) {
        const unsigned s = claim(p.spill_tail, 1);
        if (s < p.spill_cap) p.spill[s] = SpillEntry{pk, pl, rs, 1u | (kBlk1 << 16)};
        else atomicOr(p.status, kStatusSpillFull);
      }
    }
    active = false;
  }
  if (p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// Lockstep variant: one lane per read runs the read's four vector searches
// together -- '+' backward over the backward index, '-' backward over the
// forward index with complemented bases, both moving down the read, and the
// two forward searches moving up -- so every lane spends about one read length
// per read whatever the strand, and up to four independent gathers are in
// flight per lane.  Change points go to the device queue for the drain launch.
__device__ __forceinline__ void spill_push(const BatchedParams& p, uint32_t& chunk_state, uint32_t a, uint32_t b,
                                           uint32_t rs, uint32_t jt) {
  const unsigned slot = spill_slot(p, chunk_state);
  if (slot < p.spill_cap) p.spill[slot] = SpillEntry{a, b, rs, jt};
  else atomicOr(p.status, kStatusSpillFull);
}

template <int MINB>
__global__ void __launch_bounds__(kBlock, MINB) chain4_kernel(DevIndex X, BatchedParams p) {
  const uint32_t n_reads_ = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  __shared__ uint32_t c_res[kBlock], c_spill[kBlock];
  const int tid = threadIdx.x;
  c_res[tid] = 0;
  c_spill[tid] = 0;
  uint32_t read = claim(p.chain_ctr, 1);
  uint32_t nxt = read < n_reads_ ? claim(p.chain_ctr, 1) : 0xFFFFFFFFu;
  uint64_t nb0 = 0, nb1 = 0;
  uint32_t nok = 0;
  if (nxt < n_reads_) {
    nb0 = p.offs[nxt];
    nb1 = p.offs[nxt + 1];
    nok = p.ok[nxt];
  }
  uint64_t b0 = 0, b1 = 0;
  uint32_t okr = 0;
  if (read < n_reads_) {
    b0 = p.offs[read];
    b1 = p.offs[read + 1];
    okr = p.ok[read];
  }
  while (read < n_reads_) {
    const int len = (int)(b1 - b0);
    if (okr && len >= 3 && len <= 32767) {
      const uint8_t* W = p.codes + b0;
      const int n = len - 1;
      // chains: 0 '+' bwd, 1 '+' fwd, 2 '-' bwd, 3 '-' fwd
      uint32_t k0 = 0, l0 = X.top, k1 = 0, l1 = X.top, k2 = 0, l2 = X.top, k3 = 0, l3 = X.top;
      uint32_t pk0 = 0, pl0 = X.top, pk1 = 0, pl1 = X.top, pk2 = 0, pl2 = X.top, pk3 = 0, pl3 = X.top;
      uint32_t alive = 0xFu;
      for (int t = 0; t <= n; ++t) {
        const int jb = n - t, jf = t;
        const uint32_t bb = W[jb], bf = W[jf];
        if (alive & 1u) bw_step(X, View{0, 0}, bb, k0, l0);
        if (alive & 2u) bw_step(X, View{1, 0}, bf, k1, l1);
        if (alive & 4u) bw_step(X, View{1, 1}, bb, k2, l2);
        if (alive & 8u) bw_step(X, View{0, 1}, bf, k3, l3);
        // backward chains: entry at jb vs entry at J = jb + 1; window [2, n/2], block at J = 1
        // forward chains:  entry at jf vs entry at J = jf - 1; window [n/2 - 1, n - 2], block at n - 1
        const int Jb = jb + 1, Jf = jf - 1;
        const bool wb = Jb >= 2 && Jb <= n / 2;
        const bool wf = Jf >= n / 2 - 1 && Jf <= n - 1 && jf >= 1;
        const uint32_t tf = (uint32_t)Jf | ((Jf == n - 1 ? kBlkN : kCpFwd) << 16);
        const uint32_t tb = (uint32_t)Jb | (kCpBwd << 16);
#define HPG_CHAIN_TAIL(I, K, L, PK, PL, WIN, JT, STRAND, BWD)                                      \
  if (alive & (1u << I)) {                                                                         \
    const bool differ = (L - K) != (PL - PK);                                                      \
    if (differ && WIN) {                                                                           \
      uint32_t cs = c_spill[tid];                                                                  \
      spill_push(p, cs, PK, PL, (read << 1) | STRAND, JT);                                         \
      c_spill[tid] = cs;                                                                           \
    }                                                                                              \
    if (K > L || (BWD ? jb == 0 : jf == n)) {                                                      \
      if (BWD && jb == 0) {                                                                        \
        const uint32_t rs_ = (read << 1) | STRAND;                                                 \
        if (K <= L) {                                                                              \
          uint32_t r = c_res[tid];                                                                 \
          const unsigned slot = res_slot(p, r);                                                    \
          c_res[tid] = r;                                                                          \
          write_hit(p, slot, rs_, order_key(0, 0, 0), K, L, pack_meta(0, 0, 0, 0, 0));             \
        }                                                                                          \
        if (differ) {                                                                              \
          uint32_t cs = c_spill[tid];                                                              \
          spill_push(p, cs, PK, PL, rs_, 1u | (kBlk1 << 16));                                      \
          c_spill[tid] = cs;                                                                       \
        }                                                                                          \
      }                                                                                            \
      alive &= ~(1u << I);                                                                         \
    } else {                                                                                       \
      PK = K;                                                                                      \
      PL = L;                                                                                      \
    }                                                                                              \
  }
        HPG_CHAIN_TAIL(0, k0, l0, pk0, pl0, wb, tb, 0u, true)
        HPG_CHAIN_TAIL(1, k1, l1, pk1, pl1, wf, tf, 0u, false)
        HPG_CHAIN_TAIL(2, k2, l2, pk2, pl2, wb, tb, 1u, true)
        HPG_CHAIN_TAIL(3, k3, l3, pk3, pl3, wf, tf, 1u, false)
#undef HPG_CHAIN_TAIL
        if (!alive) break;
      }
    }
    // next read: the prefetched one; prefetch the one after
    read = nxt;
    b0 = nb0;
    b1 = nb1;
    okr = nok;
    if (read < n_reads_) {
      nxt = claim(p.chain_ctr, 1);
      if (nxt < n_reads_) {
        nb0 = p.offs[nxt];
        nb1 = p.offs[nxt + 1];
        nok = p.ok[nxt];
      }
    }
  }
  {  // reserved but unused slots of the last chunks
    res_leave(p, c_res[tid]);
    spill_leave(p, c_spill[tid]);
  }
}

// Phased lockstep variant: one lane per read runs the two vector searches of
// a phase together -- phase 0: '+' backward and '-' forward (both on the
// backward index), phase 1: '-' backward and '+' forward (forward index).
// Lanes then spend about one read length per read whatever the strand, the
// next read is claimed and fetched ahead, and only one direction's blocks
// are live in L2.  Change points go to the device queue for the drain launch.
template <int MINB>
__global__ void __launch_bounds__(kBlock, MINB) chain2_kernel(DevIndex X, BatchedParams p, int phase) {
  const uint32_t n_reads_ = p.n_reads_dev ? *p.n_reads_dev : p.n_reads;
  __shared__ uint32_t c_res[kBlock], c_spill[kBlock];
  const int tid = threadIdx.x;
  c_res[tid] = 0;
  c_spill[tid] = 0;
  const uint32_t sA = (uint32_t)phase, sB = 1u - (uint32_t)phase;  // strands of the backward / forward chain
  const View vA{(uint32_t)phase, sA}, vB{(uint32_t)phase, sB};
  uint32_t read = claim(p.chain_ctr, 1);
  uint32_t nxt = read < n_reads_ ? claim(p.chain_ctr, 1) : 0xFFFFFFFFu;
  uint64_t b0 = 0, b1 = 0, nb0 = 0, nb1 = 0;
  uint32_t okr = 0, nok = 0;
  if (read < n_reads_) {
    b0 = p.offs[read];
    b1 = p.offs[read + 1];
    okr = p.ok[read];
  }
  if (nxt < n_reads_) {
    nb0 = p.offs[nxt];
    nb1 = p.offs[nxt + 1];
    nok = p.ok[nxt];
  }
  uint32_t sectors = 0;
  while (read < n_reads_) {
    const int len = (int)(b1 - b0);
    if (okr && len >= 3 && len <= 32767) {
      const uint8_t* W = p.codes + b0;
      const int n = len - 1, half = n / 2;
      uint32_t kA = 0, lA = X.top, pkA = 0, plA = X.top, kB = 0, lB = X.top, pkB = 0, plB = X.top;
      bool aA = true, aB = true;
      uint32_t bA = W[n], bB = W[0];
      for (int t = 0; t <= n; ++t) {
        const int jb = n - t, jf = t;
        const uint32_t nbA = (aA && jb > 0) ? W[jb - 1] : 0u;  // next bases, fetched with this step's gathers
        const uint32_t nbB = (aB && jf < n) ? W[jf + 1] : 0u;
        if (p.census) sectors += (aA ? (((kA >> 6) == (lA >> 6)) ? 1u : 2u) : 0u) +
                                 (aB ? (((kB >> 6) == (lB >> 6)) ? 1u : 2u) : 0u);
        if (aA) bw_step(X, vA, bA, kA, lA);
        if (aB) bw_step(X, vB, bB, kB, lB);
        if (aA) {  // backward: entry at jb vs J = jb + 1; window [2, n/2], block at J = 1
          const int J = jb + 1;
          const bool differ = (lA - kA) != (plA - pkA);
          if (differ && J >= 2 && J <= half) {
            uint32_t cs = c_spill[tid];
            spill_push(p, cs, pkA, plA, (read << 1) | sA, (uint32_t)J | (kCpBwd << 16));
            c_spill[tid] = cs;
          }
          if (kA > lA || jb == 0) {
            if (jb == 0) {
              const uint32_t rs = (read << 1) | sA;
              if (kA <= lA) {
                uint32_t r = c_res[tid];
                const unsigned slot = res_slot(p, r);
                c_res[tid] = r;
                write_hit(p, slot, rs, order_key(0, 0, 0), kA, lA, pack_meta(0, 0, 0, 0, 0));
              }
              if (differ) {
                uint32_t cs = c_spill[tid];
                spill_push(p, cs, pkA, plA, rs, 1u | (kBlk1 << 16));
                c_spill[tid] = cs;
              }
            }
            aA = false;
          } else {
            pkA = kA;
            plA = lA;
            bA = nbA;
          }
        }
        if (aB) {  // forward: entry at jf vs J = jf - 1; window [n/2 - 1, n - 2], block at n - 1
          const int J = jf - 1;
          const bool differ = (lB - kB) != (plB - pkB);
          if (differ && jf >= 1 && J >= half - 1 && J <= n - 1) {
            uint32_t cs = c_spill[tid];
            spill_push(p, cs, pkB, plB, (read << 1) | sB, (uint32_t)J | ((J == n - 1 ? kBlkN : kCpFwd) << 16));
            c_spill[tid] = cs;
          }
          if (kB > lB || jf == n) {
            aB = false;
          } else {
            pkB = kB;
            plB = lB;
            bB = nbB;
          }
        }
        if (!aA && !aB) break;
      }
    }
    read = nxt;
    b0 = nb0;
    b1 = nb1;
    okr = nok;
    if (read < n_reads_) {
      nxt = claim(p.chain_ctr, 1);
      if (nxt < n_reads_) {
        nb0 = p.offs[nxt];
        nb1 = p.offs[nxt + 1];
        nok = p.ok[nxt];
      }
    }
  }
  {  // reserved but unused slots of the last chunks
    res_leave(p, c_res[tid]);
    spill_leave(p, c_spill[tid]);
  }
  if (p.census) atomicAdd(p.census, (unsigned long long)sectors);
}

// ------------------------------------------------------------- finalize --

__global__ void scatter_hits_kernel(const PendingHit* __restrict__ res, const unsigned int* res_total,
                                    const uint64_t* __restrict__ seg_off, PendingHit* __restrict__ sorted,
                                    uint32_t res_cap, uint32_t* __restrict__ cursor, const unsigned* gate) {
  if (gate && *gate) return;  // a pool overflowed: the graph's host reruns the batch
  const uint32_t n = min(*res_total, res_cap);
  const uint32_t stride = gridDim.x * blockDim.x;
  // four entries a thread and round, each stage's loads and atomics issued together
  for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
    PendingHit h[4];
    uint64_t at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * stride;
      if (i < n) h[u] = res[i];
      else h[u].rs = 0xFFFFFFFFu;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)  // 0xFFFFFFFF: past the pool, or reserved but never written (chunk tail)
      if (h[u].rs != 0xFFFFFFFFu) at[u] = seg_off[h[u].rs];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (h[u].rs != 0xFFFFFFFFu) at[u] += atomicAdd(&cursor[h[u].rs], 1u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (h[u].rs != 0xFFFFFFFFu) sorted[at[u]] = h[u];
  }
}

constexpr uint32_t kLongList = 32;  // longer lists are sorted by a whole block (sort_long_lists_kernel)
constexpr int kRankTpb = 512, kRankTile = 2048;

// Lists are taken a tile at a time: `tile` of them (a multiple of 256) per block of the
// order and emit kernels, whose per-tile sums of kept hits and rows give every list's
// place in the outputs without a pass over per-list offsets.
__host__ __device__ constexpr uint32_t finalize_tile(uint32_t n_rs) { return n_rs <= (1u << 20) ? 256u : 1024u; }

// Lists of more hits or rows than these are emitted by a block each (emit_big_kernel).
constexpr uint32_t kBigHits = 32, kBigRows = 256;

__device__ __forceinline__ uint32_t rows_of(const PendingHit& x) { return x.k <= x.l ? x.l - x.k + 1 : 0u; }

// The list's rows to locate: none when they pass the limit (0: no limit), which sets bit 1 of its flag.
__device__ __forceinline__ uint32_t limited(uint64_t rows, uint64_t limit, uint8_t& flag) {
  if (limit && rows > limit) {
    flag |= 2;
    return 0;
  }
  return rows > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)rows;  // beyond kMaxLocateRows either way
}

__device__ __forceinline__ uint64_t warp_sum64(uint64_t v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

// Sorts every (read, strand) list of up to kLongList entries by emission key, in
// place, and decides its kept count, flag and rows.  A lane per list; a list of more
// than one entry is sorted by the whole warp, a lane per entry: the entry's place is
// the number of smaller keys.  (One lane inserting entry by entry held its warp for
// the longest list, every move a round trip to memory: 209 us on 2M x 150 bp, 600
// Mbp, of which 2 % of the lists are longer than one.)  Longer lists go to `longs`.
__global__ void __launch_bounds__(256)
    order_lists_kernel(PendingHit* __restrict__ sorted, const uint64_t* __restrict__ seg_off, FinalizeLists f,
                       const unsigned* gate) {
  __shared__ uint64_t s_rows[8];
  __shared__ uint32_t s_kept[8];
  if (gate && *gate) return;
  const uint32_t max_results = f.max_dev ? *f.max_dev : f.max_results;
  const uint64_t limit = f.limit_dev ? *f.limit_dev : f.limit;
  const uint32_t n_rs = f.n_reads_dev ? min(f.n_rs, 2u * *f.n_reads_dev) : f.n_rs;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t sum_rows = 0;
  uint32_t sum_kept = 0;
  for (uint32_t r0 = 0; r0 < f.tile; r0 += 256) {
    const uint64_t rs64 = (uint64_t)blockIdx.x * f.tile + r0 + threadIdx.x;
    if ((uint64_t)blockIdx.x * f.tile + r0 >= n_rs) break;  // uniform over the block
    const uint32_t rs = (uint32_t)rs64;
    const bool live = rs64 < n_rs;
    uint64_t b = 0;
    uint32_t cnt = 0;
    if (live) {
      b = seg_off[rs];
      cnt = (uint32_t)(seg_off[rs + 1] - b);
    }
    const uint32_t keep = min(cnt, max_results);
    uint64_t rows = 0;
    if (cnt == 1 && keep) {
      const uint2 kl = *reinterpret_cast<const uint2*>(&sorted[b].k);
      rows = kl.x <= kl.y ? (uint64_t)(kl.y - kl.x) + 1 : 0;
    }
    if (cnt > kLongList && keep) {  // the long sort's work (the list holds enough room for every such list)
      const unsigned q = atomicAdd(f.n_longs, 1u);
      if (q < f.longs_cap) f.longs[q] = rs;
    }
    unsigned some = __ballot_sync(0xFFFFFFFFu, cnt > 1 && cnt <= kLongList && keep);
    while (some) {
      const int j = __ffs(some) - 1;
      some &= some - 1;
      const uint64_t bj = __shfl_sync(0xFFFFFFFFu, b, j);
      const uint32_t cj = __shfl_sync(0xFFFFFFFFu, cnt, j), kj = __shfl_sync(0xFFFFFFFFu, keep, j);
      PendingHit x;
      x.key = 0xFFFFFFFFu;
      if (lane < cj) x = sorted[bj + lane];
      uint32_t rank = 0;
      for (uint32_t i = 0; i < cj; ++i) rank += __shfl_sync(0xFFFFFFFFu, x.key, i) < x.key ? 1u : 0u;
      __syncwarp();
      const bool kept = lane < cj && rank < kj;
      if (kept) sorted[bj + rank] = x;
      const uint64_t sum = warp_sum64(kept ? rows_of(x) : 0u);
      if ((int)lane == j) rows = sum;
    }
    if (live) {
      uint8_t flag = cnt > max_results ? 1 : 0;
      const uint32_t lim = limited(rows, limit, flag);
      f.kept[rs] = keep;
      f.trunc[rs] = flag;
      f.list_rows[rs] = lim;
      sum_kept += keep;
      sum_rows += lim ? rows : 0;
    }
  }
  sum_rows = warp_sum64(sum_rows);
  sum_kept = __reduce_add_sync(0xFFFFFFFFu, sum_kept);
  if (lane == 0) {
    s_rows[warp] = sum_rows;
    s_kept[warp] = sum_kept;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t k = 0, r = 0;
    for (int w = 0; w < 8; ++w) {
      k += s_kept[w];
      r += s_rows[w];
    }
    f.part[blockIdx.x] = make_ulonglong2(k, r);
  }
}

// Lists longer than kLongList (low-complexity reads emit thousands of pending
// hits), one list at a time per block.  Up to kRankTile entries: a bitonic
// sort of the (key, position) pairs in shared memory, O(m log^2 m / 512).
// Longer: the rank of an entry is the number of entries of its list with a
// smaller pair, counted against tiles of the list's keys in shared memory,
// O(m^2 / 512).
// Entries placed below the kept count are written to `scratch` (the unsorted pending
// array, dead after the scatter) and copied back; then the list's rows, as above.
__global__ void __launch_bounds__(kRankTpb)
    sort_long_lists_kernel(PendingHit* __restrict__ sorted, PendingHit* __restrict__ scratch,
                           const uint64_t* __restrict__ seg_off, FinalizeLists f, const unsigned* gate) {
  if (gate && *gate) return;
  __shared__ uint64_t tile[kRankTile];
  __shared__ uint64_t s_rows[kRankTpb / 32];
  const uint64_t limit = f.limit_dev ? *f.limit_dev : f.limit;
  const uint32_t n_items = min(*f.n_longs, f.longs_cap);
  for (uint32_t item = blockIdx.x; item < n_items; item += gridDim.x) {
    const uint32_t r = f.longs[item];
    const uint64_t b = seg_off[r];
    const uint32_t m = (uint32_t)(seg_off[r + 1] - b), keep = f.kept[r];
    if (m <= kRankTile) {
      // bitonic sort of (key, position) pairs in shared memory, padded to a power of two
      uint32_t P = 64;
      while (P < m) P <<= 1;
      for (uint32_t t = threadIdx.x; t < P; t += kRankTpb)
        tile[t] = t < m ? ((uint64_t)sorted[b + t].key << 32 | t) : ~0ull;
      __syncthreads();
      for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
          for (uint32_t t = threadIdx.x; t < P / 2; t += kRankTpb) {
            const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1)), q2 = i + j;
            const uint64_t x = tile[i], y = tile[q2];
            if ((x > y) == ((i & k) == 0)) {
              tile[i] = y;
              tile[q2] = x;
            }
          }
          __syncthreads();
        }
      }
      for (uint32_t t = threadIdx.x; t < keep; t += kRankTpb) scratch[b + t] = sorted[b + (uint32_t)tile[t]];
    } else {
      for (uint32_t i0 = 0; i0 < m; i0 += kRankTpb) {
        const uint32_t i = i0 + threadIdx.x;
        const uint64_t mine = i < m ? ((uint64_t)sorted[b + i].key << 32 | i) : ~0ull;
        uint32_t rank = 0;
        for (uint32_t t0 = 0; t0 < m; t0 += kRankTile) {
          const uint32_t tn = min((uint32_t)kRankTile, m - t0);
          __syncthreads();  // the previous tile is no longer read
          for (uint32_t t = threadIdx.x; t < tn; t += kRankTpb)
            tile[t] = (uint64_t)sorted[b + t0 + t].key << 32 | (t0 + t);
          __syncthreads();
          for (uint32_t t = 0; t < tn; ++t) rank += tile[t] < mine ? 1u : 0u;
        }
        if (i < m && rank < keep) scratch[b + rank] = sorted[b + i];
      }
    }
    __syncthreads();  // every entry written before the copy back
    uint64_t rows = 0;
    for (uint32_t i = threadIdx.x; i < keep; i += kRankTpb) {
      const PendingHit x = scratch[b + i];
      sorted[b + i] = x;
      rows += rows_of(x);
    }
    rows = warp_sum64(rows);
    if ((threadIdx.x & 31) == 0) s_rows[threadIdx.x >> 5] = rows;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t sum = 0;
      for (int w = 0; w < kRankTpb / 32; ++w) sum += s_rows[w];
      uint8_t flag = f.trunc[r];
      const uint32_t lim = limited(sum, limit, flag);
      f.list_rows[r] = lim;
      f.trunc[r] = flag;
      if (lim) atomicAdd(reinterpret_cast<unsigned long long*>(&f.part[r / f.tile].y), (unsigned long long)sum);
    }
    __syncthreads();  // s_rows and the tile are rewritten for the next list
  }
}

__device__ __forceinline__ hpg_hit_t hit_record(const PendingHit& x, uint32_t rs) {
  hpg_hit_t h;
  h.read = rs >> 1;
  h.strand = (uint8_t)(rs & 1u);
  h.dir = (uint8_t)(x.meta & 1u);
  h.nm = (uint8_t)((x.meta >> 1) & 1u);
  h.err_kind = (uint8_t)((x.meta >> 2) & 3u);
  h.err_base = (uint8_t)((x.meta >> 4) & 0xFFu);
  h.pad0 = 0;
  h.err_pos = (int16_t)(uint16_t)(x.meta >> 16);
  h.pad1 = 0;
  h.k = (int64_t)x.k;
  h.l = (int64_t)x.l;
  return h;
}

// Sums of all tiles (block 0), and of the tiles before each tile in place of the tiles'
// sums when `excl`: for tile counts that the emit kernel's blocks should not each add up.
__global__ void __launch_bounds__(1024) tile_sums_kernel(ulonglong2* __restrict__ part, uint32_t n_tiles,
                                                         uint64_t* __restrict__ totals, int excl) {
  __shared__ uint64_t s_k[32], s_r[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t ck = 0, cr = 0;
  for (uint32_t t0 = 0; t0 < n_tiles; t0 += 1024) {
    const uint32_t t = t0 + threadIdx.x;
    const ulonglong2 v = t < n_tiles ? part[t] : make_ulonglong2(0, 0);
    uint64_t k = v.x, r = v.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t a = __shfl_up_sync(0xFFFFFFFFu, k, o), b = __shfl_up_sync(0xFFFFFFFFu, r, o);
      if (lane >= (uint32_t)o) {
        k += a;
        r += b;
      }
    }
    if (lane == 31) {
      s_k[warp] = k;
      s_r[warp] = r;
    }
    __syncthreads();
    uint64_t bk = ck, br = cr;
    for (uint32_t w = 0; w < 32; ++w) {
      if (w < warp) {
        bk += s_k[w];
        br += s_r[w];
      }
      ck += s_k[w];
      cr += s_r[w];
    }
    if (excl && t < n_tiles) part[t] = make_ulonglong2(bk + k - v.x, br + r - v.y);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    totals[0] = ck;
    totals[1] = cr;
  }
}

// --------------------------------------------------------------- locate --

// Rows on the backward index fill the item array from the front, rows on the
// forward index from the back, so walks claimed in order touch one direction
// at a time.  A block takes 256 consecutive hits a round: one scan of the
// (backward, forward) row counts over the block, one atomic per direction.
constexpr int kExpandTpb = 256;

__global__ void __launch_bounds__(kExpandTpb)
    expand_rows_kernel(const hpg_hit_t* __restrict__ hits, const uint64_t* __restrict__ loc_off, uint32_t n_hits,
                       uint64_t n_locs, const uint64_t* __restrict__ read_offs, RowItem* __restrict__ items,
                       unsigned int* __restrict__ side, LocateSizes z) {
  if (z.status) {  // graph form: sizes from device memory, rows checked against the item capacity
    if (*z.status) return;
    n_hits = (uint32_t)*z.n_hits;
    n_locs = *z.n_locs;
    if (n_locs > z.locs_cap) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(z.status, kStatusLocFull);
      return;
    }
  }
  __shared__ uint64_t s_warp[kExpandTpb / 32];
  __shared__ uint64_t s_base;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t h0 = (uint64_t)blockIdx.x * kExpandTpb; h0 < n_hits; h0 += (uint64_t)gridDim.x * kExpandTpb) {
    const uint64_t h = h0 + threadIdx.x;
    RowItem it{0, 0, 0, 0};
    uint32_t cnt = 0, phys = 0, k = 0;
    uint64_t b = 0;
    if (h < n_hits) {
      const hpg_hit_t x = hits[h];
      b = loc_off[h];
      cnt = (uint32_t)(loc_off[h + 1] - b);
      if (cnt) {
        const uint64_t len = read_offs[x.read + 1] - read_offs[x.read];
        const uint32_t err = x.nm ? x.err_kind : 0u;
        phys = (uint32_t)x.dir ^ (uint32_t)x.strand;  // direction = type ? dir : !dir, type = !strand
        it.hit = (uint32_t)h;
        it.phys_len = (phys << 31) | (uint32_t)(len - (err == 1 ? 1 : 0) + (err == 3 ? 1 : 0));
        k = (uint32_t)x.k;
      }
    }
    // (forward << 32 | backward) row counts, scanned over the block
    const uint64_t v = phys ? (uint64_t)cnt << 32 : (uint64_t)cnt;
    uint64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t tot = 0;
      for (int w = 0; w < kExpandTpb / 32; ++w) {
        const uint64_t t = s_warp[w];
        s_warp[w] = tot;
        tot += t;
      }
      const uint32_t b0 = (uint32_t)tot ? atomicAdd(&side[0], (uint32_t)tot) : 0u;
      const uint32_t b1 = (uint32_t)(tot >> 32) ? atomicAdd(&side[1], (uint32_t)(tot >> 32)) : 0u;
      s_base = (uint64_t)b1 << 32 | b0;
    }
    __syncthreads();
    const uint64_t excl = s_base + s_warp[warp] + incl - v;
    const uint32_t at = phys ? (uint32_t)(excl >> 32) : (uint32_t)excl;
    // a hit's rows: up to 4 by its own thread; more (repeats, up to the locate
    // limit) by the whole warp, 32 rows a round, so one long hit does not hold
    // the block for thousands of serial stores
    if (cnt <= 4) {
      for (uint32_t i = 0; i < cnt; ++i) {
        it.row = k + i;
        it.out = (uint32_t)(b + i);
        items[phys ? n_locs - 1 - (at + i) : at + i] = it;
      }
    }
    unsigned big = __ballot_sync(0xFFFFFFFFu, cnt > 4);
    while (big) {
      const int j = __ffs(big) - 1;
      big &= big - 1;
      const uint32_t cj = __shfl_sync(0xFFFFFFFFu, cnt, j), aj = __shfl_sync(0xFFFFFFFFu, at, j);
      const uint32_t kj = __shfl_sync(0xFFFFFFFFu, k, j), pj = __shfl_sync(0xFFFFFFFFu, phys, j);
      const uint32_t bj = (uint32_t)__shfl_sync(0xFFFFFFFFu, b, j);
      RowItem w;
      w.hit = __shfl_sync(0xFFFFFFFFu, it.hit, j);
      w.phys_len = __shfl_sync(0xFFFFFFFFu, it.phys_len, j);
      for (uint32_t i = lane; i < cj; i += 32) {
        w.row = kj + i;
        w.out = bj + i;
        items[pj ? n_locs - 1 - (aj + i) : aj + i] = w;
      }
    }
    __syncthreads();  // s_warp and s_base are rewritten next round
  }
}

// Key, chromosome and position of one located row (bwt.c:2025-2036,2158-2166).
__device__ __forceinline__ hpg_loc_t located(const DevIndex& X, uint32_t sa, uint32_t phys_len, uint32_t hit) {
  const uint32_t phys = phys_len >> 31;
  const uint64_t len_calc = phys_len & kRowLenMask;
  uint64_t key = sa;
  if (phys && (phys_len & kRowKey32))  // an int length: the SA_TYPE (32-bit) difference wraps
    key = (uint32_t)((X.top + 1u) - sa - (uint32_t)len_calc - 1u);
  else if (phys)
    key = (uint64_t)((X.top + 1u) - sa) - len_calc - 1u;
  const uint32_t id = kar_search(X, key);
  hpg_loc_t o;
  o.key = key;
  o.hit = hit;
  o.pad = 0;
  if (key + len_calc <= X.kar_offset[id]) {
    o.valid = 1;
    o.chrom = id - 1;
    o.position = X.kar_start[id - 1] + (key - X.kar_offset[id - 1]);
  } else {
    o.valid = 0;
    o.chrom = 0;
    o.position = 0;
  }
  return o;
}

// Row item of a hit: direction = type ? dir : !dir, type = !strand; the length by its edit.
__device__ __forceinline__ uint32_t item_phys_len(uint32_t meta, uint32_t rs, uint32_t len) {
  const uint32_t err = (meta >> 1) & 1u ? (meta >> 2) & 3u : 0u;
  return (((meta ^ rs) & 1u) << 31) | (len - (err == 1 ? 1u : 0u) + (err == 3 ? 1u : 0u));
}

// Hit records and located rows of every list, at the places the tiles' sums and a scan
// over the tile give.  A lane per list; lists of several hits, and hits of more than 4
// rows (repeats, up to the locate limit), are shared by the warp.  With the whole
// suffix array a row costs one gather, so nothing is staged between the lists and the
// records: one pass over the ordered hits (C2: one hit and one row a read, 64 bytes of
// records) bound by HBM and one random sector a row.  Without it the hits' row offsets
// go to loc_off for the LF walks.
template <bool DIRECT, bool CENSUS>
__global__ void __launch_bounds__(256)
    emit_lists_kernel(DevIndex X, const PendingHit* __restrict__ sorted, const uint64_t* __restrict__ seg_off,
                      FinalizeLists f, const uint64_t* __restrict__ read_offs, hpg_hit_t* __restrict__ hits,
                      hpg_loc_t* __restrict__ locs, uint64_t* __restrict__ loc_off, uint64_t* __restrict__ totals,
                      uint2* __restrict__ read_off, int part_is_prefix, int no_locs, unsigned long long* census,
                      LocateSizes z) {
  extern __shared__ uint32_t s_off[];  // the tile's first hit and first row per list
  __shared__ uint64_t s_red[2][8];
  __shared__ uint32_t s_warp[2][8];
  if (z.status && *z.status & ~kStatusLocFull) return;
  const uint32_t tile = f.tile, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_rs = f.n_reads_dev ? min(f.n_rs, 2u * *f.n_reads_dev) : f.n_rs;
  const uint32_t base = blockIdx.x * tile;
  if (base >= n_rs && base) return;
  const bool last_tile = n_rs - base <= tile;  // (of an empty batch: the first)
  // hits and rows before the tile
  uint64_t h0 = 0, r0 = 0;
  if (part_is_prefix) {
    h0 = f.part[blockIdx.x].x;
    r0 = f.part[blockIdx.x].y;
  } else {
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += 256) {
      const ulonglong2 v = f.part[t];
      h0 += v.x;
      r0 += v.y;
    }
    h0 = warp_sum64(h0);
    r0 = warp_sum64(r0);
    if (lane == 0) {
      s_red[0][warp] = h0;
      s_red[1][warp] = r0;
    }
    __syncthreads();
    h0 = r0 = 0;
    for (int w = 0; w < 8; ++w) {
      h0 += s_red[0][w];
      r0 += s_red[1][w];
    }
  }
  // exclusive scan over the tile's lists (rows saturate per list only past every capacity)
  uint64_t ch = 0, cr = 0;  // of the rounds before
  for (uint32_t i0 = 0; i0 < tile; i0 += 256) {
    const uint32_t i = i0 + threadIdx.x;
    const bool in = base + i < n_rs;
    const uint32_t kh = in ? f.kept[base + i] : 0u, kr = in && !no_locs ? f.list_rows[base + i] : 0u;
    uint32_t a = kh, b = kr;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, a, o), y = __shfl_up_sync(0xFFFFFFFFu, b, o);
      if (lane >= (uint32_t)o) {
        a += x;
        b += y;
      }
    }
    if (lane == 31) {
      s_warp[0][warp] = a;
      s_warp[1][warp] = b;
    }
    __syncthreads();
    uint32_t pa = 0, pb = 0, ta = 0, tb = 0;
    for (uint32_t w = 0; w < 8; ++w) {
      if (w < warp) {
        pa += s_warp[0][w];
        pb += s_warp[1][w];
      }
      ta += s_warp[0][w];
      tb += s_warp[1][w];
    }
    s_off[i] = (uint32_t)ch + pa + a - kh;
    s_off[tile + i] = (uint32_t)cr + pb + b - kr;
    ch += ta;
    cr += tb;
    __syncthreads();
    if (base + i0 + 256 >= n_rs) break;
  }
  // (a tile whose rows pass 32 bits lies past locs_cap: found here from the exact sums)
  bool full = false;
  if (!no_locs && z.status) {
    const uint64_t end = !part_is_prefix ? r0 + f.part[blockIdx.x].y
                                         : (blockIdx.x + 1 < gridDim.x ? f.part[blockIdx.x + 1].y : totals[1]);
    full = end > z.locs_cap;
    if (full && threadIdx.x == 0) atomicOr(z.status, kStatusLocFull);
  }
  if (last_tile && threadIdx.x == 0) {
    if (!part_is_prefix) {
      totals[0] = h0 + f.part[blockIdx.x].x;
      totals[1] = no_locs ? 0 : r0 + f.part[blockIdx.x].y;
      if (n_rs == 0) totals[0] = totals[1] = 0;
    }
    if (read_off) read_off[n_rs >> 1] = make_uint2((uint32_t)(h0 + ch), (uint32_t)(r0 + cr));
    if (!DIRECT) loc_off[h0 + ch] = r0 + cr;
  }
  unsigned long long sectors = 0;
  for (uint32_t i0 = 0; i0 < tile && base + i0 < n_rs; i0 += 256) {
    const uint32_t i = i0 + threadIdx.x, rs = base + i;
    const bool in = rs < n_rs;
    uint32_t m = in ? f.kept[rs] : 0u;
    const uint32_t rows = in && !no_locs && !full ? f.list_rows[rs] : 0u;
    const uint64_t oh = h0 + s_off[i], orow = r0 + s_off[tile + i];
    if (m > kBigHits || rows > kBigRows) {  // (the list has room for every such list)
      const unsigned q = atomicAdd(f.n_bigs, 1u);
      if (q < f.bigs_cap) f.bigs[q] = make_uint4(rs, (uint32_t)oh, (uint32_t)orow, rows);
      m = 0;
    }
    if (read_off && in && !(rs & 1u)) read_off[rs >> 1] = make_uint2((uint32_t)oh, (uint32_t)orow);
    uint64_t b = 0;
    uint32_t len = 0;
    if (m) {
      b = seg_off[rs];
      len = (uint32_t)(read_offs[(rs >> 1) + 1] - read_offs[rs >> 1]);
    }
    auto locate = [&](uint64_t at, uint32_t row, uint32_t pl, uint32_t h, uint32_t sa1 = 0) {
      const uint32_t* sa = (pl >> 31) ? X.dir[1].sa : X.dir[0].sa;
      locs[at] = located(X, sa1 ? sa1 - 1 : load_row_word(sa + row), pl, h);
      if (CENSUS) sectors += sa1 ? 0 : 1;
    };
    // the rows of 32 hits, one a lane (r rows each from `at` on): up to 4 by the lane, more by the warp
    auto write_rows = [&](uint64_t at, uint32_t k, uint32_t r, uint32_t pl, uint32_t h, uint32_t sa1) {
      if (r == 1) locate(at, k, pl, h, sa1);
      else if (r <= 4)
        for (uint32_t q = 0; q < r; ++q) locate(at + q, k + q, pl, h);
      unsigned many = __ballot_sync(0xFFFFFFFFu, r > 4);
      while (many) {
        const int j = __ffs(many) - 1;
        many &= many - 1;
        const uint32_t rj = __shfl_sync(0xFFFFFFFFu, r, j), kj = __shfl_sync(0xFFFFFFFFu, k, j);
        const uint32_t pj = __shfl_sync(0xFFFFFFFFu, pl, j), hj = __shfl_sync(0xFFFFFFFFu, h, j);
        const uint64_t aj = __shfl_sync(0xFFFFFFFFu, at, j);
        for (uint32_t q = lane; q < rj; q += 32) locate(aj + q, kj + q, pj, hj);
      }
    };
    {  // lists of one hit
      PendingHit x;
      x.k = x.l = x.meta = x.sa1 = 0;
      if (m == 1) {
        x = sorted[b];
        hits[oh] = hit_record(x, rs);
        if (!DIRECT) loc_off[oh] = orow;
      }
      if (DIRECT) write_rows(orow, x.k, m == 1 ? rows : 0u, item_phys_len(x.meta, rs, len), (uint32_t)oh, x.sa1);
    }
    unsigned some = __ballot_sync(0xFFFFFFFFu, m > 1);
    while (some) {
      const int j = __ffs(some) - 1;
      some &= some - 1;
      const uint64_t bj = __shfl_sync(0xFFFFFFFFu, b, j), hj = __shfl_sync(0xFFFFFFFFu, oh, j);
      const uint64_t rj = __shfl_sync(0xFFFFFFFFu, orow, j);
      const uint32_t mj = __shfl_sync(0xFFFFFFFFu, m, j), lj = __shfl_sync(0xFFFFFFFFu, len, j);
      const uint32_t sj = __shfl_sync(0xFFFFFFFFu, rs, j);
      const bool any = __shfl_sync(0xFFFFFFFFu, rows, j) != 0;
      PendingHit x;
      x.k = 1;
      x.l = 0;
      x.meta = x.sa1 = 0;
      const bool has = lane < mj;
      if (has) {
        x = sorted[bj + lane];
        hits[hj + lane] = hit_record(x, sj);
      }
      const uint32_t r = any && has ? rows_of(x) : 0u;
      uint32_t incl = r;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (!DIRECT && has) loc_off[hj + lane] = rj + incl - r;
      if (DIRECT) write_rows(rj + incl - r, x.k, r, item_phys_len(x.meta, sj, lj), (uint32_t)(hj + lane), x.sa1);
    }
  }
  if (CENSUS && census && sectors) atomicAdd(census, sectors);
}

// The lists the emit kernel left, a block each: 256 hits a round, their rows scanned over
// the block and shared out evenly, a row a thread, so that neither a list of a thousand
// hits nor a hit of ten thousand rows holds a warp.
template <bool DIRECT, bool CENSUS>
__global__ void __launch_bounds__(256)
    emit_big_kernel(DevIndex X, const PendingHit* __restrict__ sorted, const uint64_t* __restrict__ seg_off,
                    FinalizeLists f, const uint64_t* __restrict__ read_offs, hpg_hit_t* __restrict__ hits,
                    hpg_loc_t* __restrict__ locs, uint64_t* __restrict__ loc_off, unsigned long long* census,
                    const unsigned* gate) {
  __shared__ uint32_t s_off[257], s_k[256], s_pl[256], s_warp[8];
  if (gate && *gate & ~kStatusLocFull) return;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = min(*f.n_bigs, f.bigs_cap);
  unsigned long long sectors = 0;
  for (uint32_t item = blockIdx.x; item < n; item += gridDim.x) {
    const uint4 e = f.bigs[item];
    const uint32_t rs = e.x, m = f.kept[rs];
    const uint64_t b = seg_off[rs], oh = e.y;
    uint64_t orow = e.z;
    const uint32_t len = (uint32_t)(read_offs[(rs >> 1) + 1] - read_offs[rs >> 1]);
    for (uint32_t q0 = 0; q0 < m; q0 += 256) {
      const uint32_t q = q0 + threadIdx.x;
      PendingHit x;
      x.k = 1;
      x.l = 0;
      x.meta = 0;
      if (q < m) {
        x = sorted[b + q];
        hits[oh + q] = hit_record(x, rs);
      }
      const uint32_t r = e.w && q < m ? rows_of(x) : 0u;
      uint32_t incl = r;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      uint32_t before = 0, total = 0;
      for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) before += s_warp[w];
        total += s_warp[w];
      }
      const uint32_t first = before + incl - r;
      if (!DIRECT && q < m) loc_off[oh + q] = orow + first;
      if (DIRECT) {
        s_off[threadIdx.x] = first;
        s_k[threadIdx.x] = x.k;
        s_pl[threadIdx.x] = item_phys_len(x.meta, rs, len);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < total; i += 256) {
          uint32_t lo = 0, hi = min(256u, m - q0);  // last hit of the round with s_off <= i
          while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s_off[mid] <= i) lo = mid;
            else hi = mid;
          }
          const uint32_t pl = s_pl[lo];
          const uint32_t* sa = (pl >> 31) ? X.dir[1].sa : X.dir[0].sa;
          locs[orow + i] = located(X, load_row_word(sa + s_k[lo] + (i - s_off[lo])), pl, (uint32_t)(oh + q0 + lo));
          if (CENSUS) ++sectors;
        }
      }
      orow += total;
      __syncthreads();  // s_warp and the round's hits are rewritten
    }
  }
  if (CENSUS && census && sectors) atomicAdd(census, sectors);
}

// The same for caller-built rows: a thread per item.
__global__ void __launch_bounds__(kExpandTpb)
    locate_items_kernel(DevIndex X, const RowItem* __restrict__ items, uint64_t n_items, hpg_loc_t* __restrict__ out) {
  for (uint64_t i = (uint64_t)blockIdx.x * kExpandTpb + threadIdx.x; i < n_items;
       i += (uint64_t)gridDim.x * kExpandTpb) {
    const RowItem it = items[i];
    const uint32_t* sa = (it.phys_len >> 31) ? X.dir[1].sa : X.dir[0].sa;
    out[it.out] = located(X, load_row_word(sa + it.row), it.phys_len, it.hit);
  }
}

constexpr unsigned kRowsPerClaim = 4;
// Lanes whose walk reached a sampled row (or that hold no row) wait, masked,
// until this many lanes of their converged group have (or all have), and then
// finish their rows and start the next ones together: a finish makes dependent
// loads (the SA sample, the karyotype, the next row item), and a warp that
// waited for one or two finishing lanes almost every step ran at a quarter of
// the gather rate.
constexpr unsigned kLocateBatch = 8;

__global__ void __launch_bounds__(kBlock)
    locate_persistent_kernel(DevIndex X, const RowItem* __restrict__ items, uint64_t n_locs,
                             hpg_loc_t* __restrict__ out, unsigned int* row_ctr, unsigned long long* census,
                             LocateSizes z) {
  if (z.status) {
    if (*z.status) return;  // includes an item capacity overflow found by expand_rows_kernel
    n_locs = *z.n_locs;
  }
  uint32_t r = 0, left = 0;
  uint32_t i = 0, j = 0, slot = 0;
  RowItem it{0, 0, 0, 0};
  // Software pipeline: the next row item of the lane's claim is loaded while the
  // current walk runs, and a finished walk's sample is loaded then written out at
  // the lane's next refill, so a refill waits on no load.
  RowItem nx{0, 0, 0, 0};
  RowItem pit{0, 0, 0, 0};  // the finished walk whose output is pending
  uint32_t ps = 0, pj = 0;  // its sample and steps
  bool pending = false;
  bool active = false, reached = false;
  uint32_t sectors = 0;
  auto finish = [&]() {  // the pending walk's key and chromosome
    out[pit.out] = located(X, (ps + pj) % X.walk_mod, pit.phys_len, pit.hit);
    pending = false;
  };
  for (;;) {
    // one step of the walk: the row's mark entry and block are fetched together;
    // a text-sampled row ends it (at most ratio - 1 LF steps), else LF moves on
    if (active && !reached) {
      const DevDir D = dir_of(X, it.phys_len >> 31);
      uint32_t cnt[4];
      uint4 bits;
      const uint4 mk = load_mark(D, i, X.load_mode);
      load_block_m(D.occ + (i >> 6), X.load_mode, cnt, bits);
      sectors += 2;
      if (text_sampled(mk, i, slot)) {
        reached = true;
      } else {
        i = lf_from(X, D, i, cnt, bits);
        if (++j >= X.ratio) {  // only a corrupt index gets here
          atomicOr(X.err, kErrWalk);
          slot = 0;
          reached = true;
        }
      }
    }
    const bool done = !active || reached;
    const unsigned grp = __activemask();
    const unsigned ready = __ballot_sync(grp, done);
    if (!done) continue;
    if ((uint32_t)__popc(ready) < kLocateBatch && ready != grp) continue;  // wait for more lanes
    if (pending) finish();  // the previous walk of this lane: its sample has arrived by now
    if (active) {  // the walk reached a text-sampled row: load the sample, write the row next time
      ps = dir_of(X, it.phys_len >> 31).T[slot];
      ++sectors;
      pj = j;
      pit = it;
      pending = true;
      active = false;
      reached = false;
    }
    if (left == 0) {
      r = claim(row_ctr, kRowsPerClaim);
      left = kRowsPerClaim;
      if (r < n_locs) nx = items[r];
    } else {
      ++r;
    }
    --left;
    if (r >= n_locs) break;
    it = nx;
    if (left > 0 && r + 1 < n_locs) nx = items[r + 1];  // the next row, loaded during this walk
    i = it.row;
    j = 0;
    active = true;
  }
  if (pending) finish();
  if (census) atomicAdd(census, (unsigned long long)sectors);
}

template <int MINB>
void launch_chain_m(const DevIndex& X, const BatchedParams& p, const BatchedTuning& t, int num_sms, int phase,
                    cudaStream_t s) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain_kernel<MINB>, kBlock, 0);
  if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
  if (per_sm < 1) per_sm = 1;
  count_launches(1);
  chain_kernel<MINB><<<num_sms * per_sm, kBlock, 0, s>>>(X, p, t.chunk < 1 ? 1 : t.chunk, phase);
}

template <int D, int MINB>
void launch_search_dm(const DevIndex& X, const BatchedParams& p, const BatchedTuning& t, int num_sms, bool drain,
                      cudaStream_t s) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_search_kernel<D, MINB, false>, kBlock, 0);
  if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
  if (per_sm < 1) per_sm = 1;
  count_launches(1);
  const int ch = t.chunk < 1 ? 1 : t.chunk;
  if (p.census)
    batched_search_kernel<D, MINB, true><<<num_sms * per_sm, kBlock, 0, s>>>(X, p, drain ? 1 : 0, ch);
  else
    batched_search_kernel<D, MINB, false><<<num_sms * per_sm, kBlock, 0, s>>>(X, p, drain ? 1 : 0, ch);
}

template <int D>
void launch_search_d(const DevIndex& X, const BatchedParams& p, const BatchedTuning& t, int num_sms, bool drain,
                     cudaStream_t s) {
  if (t.min_blocks >= 16)
    launch_search_dm<D, 16>(X, p, t, num_sms, drain, s);
  else if (t.min_blocks >= 12)
    launch_search_dm<D, 12>(X, p, t, num_sms, drain, s);
  else if (t.min_blocks >= 10)
    launch_search_dm<D, 10>(X, p, t, num_sms, drain, s);
  else
    launch_search_dm<D, 1>(X, p, t, num_sms, drain, s);
}

template <int D>
int occupancy_d(const BatchedTuning& t) {
  int per_sm = 0;
  if (t.min_blocks >= 16)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_search_kernel<D, 16, false>, kBlock, 0);
  else if (t.min_blocks >= 12)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_search_kernel<D, 12, false>, kBlock, 0);
  else if (t.min_blocks >= 10)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_search_kernel<D, 10, false>, kBlock, 0);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_search_kernel<D, 1, false>, kBlock, 0);
  if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
  return per_sm;
}

}  // namespace

int batched_max_blocks_per_sm(const BatchedTuning& t) {
  if (t.split == 3) return wave_max_blocks_per_sm(t);
  if (t.split == 2) {
    int per_sm = 0;
    if (t.min_blocks >= 16)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<16>, kBlock, 0);
    else if (t.min_blocks >= 12)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<12>, kBlock, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<1>, kBlock, 0);
    if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
    return per_sm;
  }
  if (t.split) {
    int per_sm = 0;
    if (t.split == 1) {
      if (t.min_blocks >= 16)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<16>, kBlock, 0);
      else if (t.min_blocks >= 12)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<12>, kBlock, 0);
      else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<1>, kBlock, 0);
      if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
      return per_sm;
    }
    if (t.min_blocks >= 16)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain_kernel<16>, kBlock, 0);
    else if (t.min_blocks >= 12)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain_kernel<12>, kBlock, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain_kernel<1>, kBlock, 0);
    if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
    return per_sm;
  }
  if (t.stack <= 2) return occupancy_d<2>(t);
  if (t.stack <= 4) return occupancy_d<4>(t);
  return occupancy_d<8>(t);
}

void launch_batched_search(const DevIndex& X, const BatchedParams& p, const BatchedTuning& t, int num_sms, bool drain,
                           cudaStream_t s) {
  if (t.split == 3 && !drain) {  // warp-cooperative chains and branches
    launch_wave_search(X, p, t, num_sms, s);
    return;
  }
  if (t.split == 2 && !drain) {  // lockstep chains, one lane per read
    int per_sm = 0;
    if (t.min_blocks >= 16) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<16>, kBlock, 0);
      count_launches(1);
      chain4_kernel<16><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p);
    } else if (t.min_blocks >= 12) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<12>, kBlock, 0);
      count_launches(1);
      chain4_kernel<12><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p);
    } else {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain4_kernel<1>, kBlock, 0);
      if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
      count_launches(1);
      chain4_kernel<1><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p);
    }
    return;
  }
  if (t.split == 1 && !drain && t.phase < 2) {  // phased lockstep: the phase's two chains per read
    int per_sm = 0;
    if (t.min_blocks >= 16) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<16>, kBlock, 0);
      count_launches(1);
      chain2_kernel<16><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p, t.phase);
    } else if (t.min_blocks >= 12) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<12>, kBlock, 0);
      count_launches(1);
      chain2_kernel<12><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p, t.phase);
    } else {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, chain2_kernel<1>, kBlock, 0);
      if (t.blocks_per_sm > 0 && t.blocks_per_sm < per_sm) per_sm = t.blocks_per_sm;
      count_launches(1);
      chain2_kernel<1><<<num_sms * (per_sm > 0 ? per_sm : 1), kBlock, 0, s>>>(X, p, t.phase);
    }
    return;
  }
  if (t.split && !drain) {  // chains only; every change point goes to the queue
    const int phase = t.phase;
    if (t.min_blocks >= 16)
      launch_chain_m<16>(X, p, t, num_sms, phase, s);
    else if (t.min_blocks >= 12)
      launch_chain_m<12>(X, p, t, num_sms, phase, s);
    else
      launch_chain_m<1>(X, p, t, num_sms, phase, s);
    return;
  }
  if (t.stack <= 2)
    launch_search_d<2>(X, p, t, num_sms, drain, s);
  else if (t.stack <= 4)
    launch_search_d<4>(X, p, t, num_sms, drain, s);
  else
    launch_search_d<8>(X, p, t, num_sms, drain, s);
}

void launch_scatter_hits(const PendingHit* res, const unsigned int* res_total, const uint64_t* seg_off,
                         PendingHit* sorted, uint32_t res_cap, uint32_t* cursor, cudaStream_t s, const unsigned* gate) {
  count_launches(1);
  scatter_hits_kernel<<<1024, 256, 0, s>>>(res, res_total, seg_off, sorted, res_cap, cursor, gate);
}

size_t long_lists_cap(size_t res_cap) { return res_cap / (kLongList + 1) + 2; }

size_t big_lists_cap(uint64_t hits, uint64_t rows) { return hits / (kBigHits + 1) + rows / (kBigRows + 1) + 2; }

size_t finalize_tiles(uint32_t n_rs) { return (n_rs + finalize_tile(n_rs) - 1) / finalize_tile(n_rs) + 1; }

void launch_order_lists(PendingHit* sorted, PendingHit* scratch, const uint64_t* seg_off, FinalizeLists& f,
                        int num_sms, cudaStream_t s, const unsigned* gate) {
  f.tile = finalize_tile(f.n_rs);
  if (!f.n_rs) return;
  count_launches(2);
  order_lists_kernel<<<(f.n_rs + f.tile - 1) / f.tile, 256, 0, s>>>(sorted, seg_off, f, gate);
  sort_long_lists_kernel<<<(unsigned)(2 * num_sms), kRankTpb, 0, s>>>(sorted, scratch, seg_off, f, gate);
}

void launch_tile_sums(const FinalizeLists& f, uint64_t* totals, cudaStream_t s) {
  count_launches(1);
  tile_sums_kernel<<<1, 1024, 0, s>>>(f.part, f.n_rs ? (f.n_rs + f.tile - 1) / f.tile : 0, totals, 0);
}

void launch_emit_lists(const DevIndex& X, const PendingHit* sorted, const uint64_t* seg_off, const FinalizeLists& f,
                       const uint64_t* read_offs, hpg_hit_t* hits, hpg_loc_t* locs, uint64_t* loc_off,
                       uint64_t* totals, uint2* read_off, bool no_locs, unsigned long long* census, int num_sms,
                       cudaStream_t s, const LocateSizes& z) {
  if (!f.n_rs) {
    cudaMemsetAsync(totals, 0, 16, s);
    return;
  }
  const uint32_t tiles = (f.n_rs + f.tile - 1) / f.tile;
  const int prefix = tiles > 4096;
  if (prefix) {  // (fewer: every block adds up the tiles before its own)
    count_launches(1);
    tile_sums_kernel<<<1, 1024, 0, s>>>(f.part, tiles, totals, 1);
  }
  const size_t smem = 2 * f.tile * sizeof(uint32_t);
  count_launches(1);
  count_launches(1);
  const unsigned big_grid = (unsigned)(4 * num_sms);
  auto launch = [&](auto lists, auto big) {
    lists<<<tiles, 256, smem, s>>>(X, sorted, seg_off, f, read_offs, hits, locs, loc_off, totals, read_off, prefix,
                                   no_locs, census, z);
    big<<<big_grid, 256, 0, s>>>(X, sorted, seg_off, f, read_offs, hits, locs, loc_off, census, z.status);
  };
  if (X.text && census) launch(emit_lists_kernel<true, true>, emit_big_kernel<true, true>);
  else if (X.text) launch(emit_lists_kernel<true, false>, emit_big_kernel<true, false>);
  else launch(emit_lists_kernel<false, false>, emit_big_kernel<false, false>);
}

void launch_locate_persistent(const DevIndex& X, const hpg_hit_t* hits, const uint64_t* loc_off, uint32_t n_hits,
                              uint64_t n_locs, const uint64_t* read_offs, hpg_loc_t* out, void* row_items,
                              unsigned int* row_ctr, unsigned long long* census, int num_sms, cudaStream_t s,
                              const LocateSizes& z) {
  if (!n_locs) return;
  RowItem* items = static_cast<RowItem*>(row_items);
  unsigned int* side = row_ctr + 1;  // two counters after the row claim counter
  cudaMemsetAsync(side, 0, 8, s);
  count_launches(1);
  // graph form: grid-stride over the hits, 8 blocks per SM
  const uint64_t hit_grid = z.status ? 8ull * num_sms : (n_hits + kExpandTpb - 1) / kExpandTpb;
  expand_rows_kernel<<<(unsigned)(hit_grid ? hit_grid : 1), kExpandTpb, 0, s>>>(hits, loc_off, n_hits, n_locs,
                                                                                read_offs, items, side, z);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, locate_persistent_kernel, kBlock, 0);
  if (per_sm < 1) per_sm = 1;
  uint64_t blocks = (uint64_t)num_sms * per_sm;
  const uint64_t need = (n_locs + kBlock * kRowsPerClaim - 1) / (kBlock * kRowsPerClaim);
  if (need < blocks) blocks = need;
  count_launches(1);
  locate_persistent_kernel<<<(unsigned)blocks, kBlock, 0, s>>>(X, items, n_locs, out, row_ctr, census, z);
}

void launch_locate_items(const DevIndex& X, const RowItem* items, uint64_t n_items, hpg_loc_t* out,
                         unsigned int* row_ctr, int num_sms, cudaStream_t s) {
  if (!n_items) return;
  if (X.text) {
    const uint64_t blocks = std::min<uint64_t>((n_items + kExpandTpb - 1) / kExpandTpb, 16ull * num_sms);
    count_launches(1);
    locate_items_kernel<<<(unsigned)blocks, kExpandTpb, 0, s>>>(X, items, n_items, out);
    return;
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, locate_persistent_kernel, kBlock, 0);
  if (per_sm < 1) per_sm = 1;
  uint64_t blocks = (uint64_t)num_sms * per_sm;
  const uint64_t need = (n_items + kBlock * kRowsPerClaim - 1) / (kBlock * kRowsPerClaim);
  if (need < blocks) blocks = need;
  cudaMemsetAsync(row_ctr, 0, 4, s);
  count_launches(1);
  locate_persistent_kernel<<<(unsigned)blocks, kBlock, 0, s>>>(X, items, n_items, out, row_ctr, nullptr,
                                                               LocateSizes());
}

size_t locate_row_item_bytes() { return sizeof(RowItem); }

namespace {

// One thread per string of L symbols: the search from the full interval over
// them on physical direction d, stopped where it fails.
__global__ void build_kmer_kernel(DevIndex X, uint32_t d, uint32_t L, uint2* __restrict__ out) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= (1u << (2 * L))) return;
  uint32_t k = 0, l = X.top;
  for (uint32_t i = 0; i < L; ++i) {
    bw_step(X, View{d, 0}, (c >> (2 * (L - 1 - i))) & 3u, k, l);
    if (k > l) break;
  }
  out[c] = make_uint2(k, l);
}

}  // namespace

void launch_build_kmer(const DevIndex& X, uint32_t d, uint32_t L, uint2* out, cudaStream_t s) {
  const uint32_t n = 1u << (2 * L);
  count_launches(1);
  build_kmer_kernel<<<(n + 255) / 256, 256, 0, s>>>(X, d, L, out);
}


void launch_search_stage(const DevIndex& X, const BatchedParams& p, const BatchedTuning& t, int num_sms,
                         unsigned int* ctr, uint32_t* long_list, uint32_t long_cap, SpillEntry* blocks,
                         uint32_t block_cap, cudaEvent_t mid, bool external, cudaStream_t s) {
  auto mark = [&]() {
    if (!mid) return;
    if (external)
      cudaEventRecordWithFlags(mid, s, cudaEventRecordExternal);
    else
      cudaEventRecord(mid, s);
  };
  if (t.split == 1) {
    // one index direction at a time: chains on the backward index and their
    // change points, then chains on the forward index and theirs
    BatchedTuning t0 = t;
    BatchedParams p1 = p;
    p1.chain_ctr = ctr + 8;
    t0.phase = 0;
    launch_batched_search(X, p, t0, num_sms, false, s);
    launch_batched_search(X, p, t0, num_sms, true, s);
    cudaMemcpyAsync(ctr + 1, ctr + 2, 4, cudaMemcpyDeviceToDevice, s);  // drain resumes at the queue tail
    mark();
    t0.phase = 1;
    launch_batched_search(X, p1, t0, num_sms, false, s);
    launch_batched_search(X, p1, t0, num_sms, true, s);
  } else if (t.split == 3) {
    // warp-cooperative launches (one per index direction, or one for both), the
    // fused kernel over the reads too long for a warp's group buffer, then the
    // change points that did not fit the warps' stacks, and the blocks
    BatchedParams pw = p;
    pw.wave_group = (uint32_t)(t.group < 1 ? 1 : (t.group > 32 ? 32 : t.group));
    pw.long_list = long_list;
    pw.long_n = ctr + 10;
    pw.long_cap = long_cap;
    pw.blocks = blocks;
    pw.block_n = ctr + 13;
    pw.block_cap = block_cap;
    BatchedTuning tl = t;
    tl.split = 0;
    tl.dir_split = 0;
    if (X.text && p.walk) {
      // the text on the device: one-row searches by comparison (the queue's
      // counters take the place of the warp form's)
      pw.rest_head = ctr + 0;
      pw.rows_head = ctr + 8;
      pw.walk_n = ctr + 9;
      pw.rest_n = ctr + 10;
      pw.rows_n = ctr + 11;
      launch_text_search(X, pw, num_sms, s);
      mark();
      return;
    }
    if (t.dir_split == 2) {
      pw.dir_split = 2;
      launch_wave_search(X, pw, t, num_sms, s);
      pw.dir_split = 3;
      launch_wave_search(X, pw, t, num_sms, s);
    } else {
      pw.dir_split = 0;
      launch_wave_search(X, pw, t, num_sms, s);
    }
    BatchedParams pl = p;
    // reads above kWaveLongMin bases are at most 1/4000 of the bases: two
    // blocks per SM serve them, and an empty list costs a short launch
    tl.blocks_per_sm = 2;
    pl.dir_split = 0;
    pl.chain_ctr = ctr + 11;
    pl.read_list = long_list;
    pl.read_list_n = ctr + 10;
    pl.long_cap = long_cap;
    launch_batched_search(X, pl, tl, num_sms, false, s);
    mark();
    // queued change points' branches, eight per change point; the blocks among
    // them join the block list, which the fused kernel's drain then empties
    launch_wave_branches(X, p, blocks, ctr + 13, block_cap, num_sms, s);
    BatchedParams pb = p;
    pb.spill = blocks;
    pb.spill_head = ctr + 12;
    pb.spill_tail = ctr + 13;
    pb.spill_cap = block_cap;
    tl.blocks_per_sm = t.blocks_per_sm;
    launch_batched_search(X, pb, tl, num_sms, true, s);
  } else if (p.dir_split == 2) {  // one index direction after the other, then the queued change points
    launch_batched_search(X, p, t, num_sms, false, s);
    BatchedParams p1 = p;
    p1.dir_split = 3;
    launch_batched_search(X, p1, t, num_sms, false, s);
    mark();
    launch_batched_search(X, p, t, num_sms, true, s);
  } else {
    launch_batched_search(X, p, t, num_sms, false, s);
    mark();
    launch_batched_search(X, p, t, num_sms, true, s);
  }
}

}  // namespace hpgbwt
