// full_rows.cu -- the whole suffix array, its inverse and the packed text on
// the device, derived when an index is opened.
//
// The index files sample the suffix array (S.vec, one value per `ratio` rows)
// and hold no inverse and no text, so a row is located by walking LF and a
// match is extended base by base, each step one dependent random 32-byte
// sector.  With SA[row], SA^-1[position] and the text itself in HBM a row is
// located by one gather, and once a search's interval is a single row the rest
// of the match is a comparison of the read with the text: SA of the row, the
// text (25 bytes per 100 bases), SA^-1 of the position reached.  16.25 bytes
// per base for both directions, and a start table of log4(n) symbols, 14 at
// most, per direction (8 bytes an entry): 2.7 GB at 100 Mbp, 54 GB at 3.1 Gbp of
// the device's 284 GB.  Measured on 2M x 100 bp reads, 100 Mbp: the locate stage
// takes 406 us per 2M rows with LF walks (16 sectors a row), 80 us with the gather;
// the search 3704 us with rank steps only, 700 us with the text.
//
// Table length (search stage there / on 2M x 150 bp, 600 Mbp, each before the kernels that
// took it to 700 / 2760): 11 symbols 903 /
// 7783 us, 12: 903 / 7570, 13: 891 / 7550, 14: 864 / 7392; a table longer than
// log4(n) is mostly empty intervals and four times the memory.
//
// They are kept when they take at most a quarter of the device's free memory
// (several indexes and batch workspaces share the rest) and the derivation
// proves them consistent with the index; otherwise, and once a caller has
// dropped them, every path uses the sampled arrays and LF, with the same results.
//
// Derivation: as text_samples.cu, one LF walk from every sampled row to the
// next, which visits every row once with its SA value v known: SA[row] = v,
// SA^-1[v] = row, and the row's BWT symbol is the text's symbol v - 1 of that
// direction.  Checked on the way: each walk ends on a sampled row holding the
// value it arrived with, the '$' row and only it holds 0, the walks visit n + 1
// rows, and the forward index's symbols are the text's.  Then SA, SA^-1 and the
// text are exactly the index's own.
#include <cuda_runtime.h>

#include <string>

#include "engine_internal.hpp"
#include "fm_device.cuh"
#include "kernels.cuh"

namespace hpgbwt {

namespace {

// d = 0 writes the text, d = 1 compares with it.  bad[0] counts
// inconsistencies, bad[1] the rows visited.
__global__ void full_rows_kernel(DevIndex X, uint32_t d, uint32_t n_samples, uint32_t* __restrict__ sa,
                                 uint32_t* __restrict__ isa, uint64_t* __restrict__ text,
                                 unsigned long long* __restrict__ bad) {
  const DevDir D = dir_of(X, d);
  const uint32_t n_rows = X.walk_mod, n = n_rows - 1u;
  const uint32_t stride = gridDim.x * blockDim.x;
  unsigned long long visited = 0, wrong = 0;
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n_samples; s += stride) {
    const uint64_t r0 = (uint64_t)s * X.ratio;
    if (r0 >= n_rows) break;  // s only grows in this loop
    uint32_t i = (uint32_t)r0, v = D.S[s];
    if (v >= n_rows) {
      ++wrong;
      continue;
    }
    uint32_t at = 0xFFFFFFFFu;  // word of the text being gathered
    uint64_t acc = 0;
    for (uint32_t steps = 0; steps < n_rows; ++steps) {
      uint32_t cnt[4];
      uint4 bits;
      load_block_m(D.occ + (i >> 6), X.load_mode, cnt, bits);
      sa[i] = v;
      isa[v] = i;
      ++visited;
      if ((i == D.dollar) != (v == 0)) {
        ++wrong;
        break;
      }
      if (v) {
        const uint32_t r = i & 63;
        const uint32_t lo = r < 32 ? bits.x : bits.y, hi = r < 32 ? bits.z : bits.w;
        const uint64_t b = ((lo >> (r & 31)) & 1u) | (((hi >> (r & 31)) & 1u) << 1);
        const uint32_t p = d ? n - v : v - 1u;  // the forward index is that of the reversed text
        if (d == 0) {
          if ((p >> 5) != at) {
            if (acc) atomicOr(reinterpret_cast<unsigned long long*>(text + at), (unsigned long long)acc);
            acc = 0;
            at = p >> 5;
          }
          acc |= b << (2u * (p & 31u));
        } else if (((text[p >> 5] >> (2u * (p & 31u))) & 3u) != b) {
          ++wrong;
        }
      }
      i = lf_from(X, D, i, cnt, bits);
      v = v ? v - 1u : n;
      if (sampled_row(X, i)) {
        const uint32_t t = X.ratio_shift != 0xFFFFFFFFu ? i >> X.ratio_shift : i / X.ratio;
        if (D.S[t] != v) ++wrong;
        break;
      }
    }
    if (acc) atomicOr(reinterpret_cast<unsigned long long*>(text + at), (unsigned long long)acc);
  }
  if (wrong) atomicAdd(&bad[0], wrong);
  if (visited) atomicAdd(&bad[1], visited);
}

}  // namespace

// Symbols of the start table of the search with the text.
uint32_t tmer_symbols(const Engine* en) {
  uint32_t L = 1;
  while (L < 14 && (1ull << (2 * (L + 1))) <= en->X.walk_mod) ++L;
  return L;
}

constexpr size_t kTextPad = 2;  // words of padding on either side of the text

void free_full_rows(Engine* en) {
  for (int d = 0; d < 2; ++d) {
    cudaFree(en->d_sa[d]);
    cudaFree(en->d_isa[d]);
    en->d_sa[d] = en->d_isa[d] = nullptr;
  }
  for (uint2*& m : en->d_tmer) {
    cudaFree(m);
    m = nullptr;
  }
  cudaFree(en->d_text);
  en->d_text = nullptr;
  engine_set_full_rows(en, 0);
}

// Points the index at the arrays, or away from them.
int engine_set_full_rows(Engine* en, int on) {
  const bool use = on && en->d_text;
  for (int d = 0; d < 2; ++d) {
    en->X.dir[d].sa = use ? en->d_sa[d] : nullptr;
    en->X.dir[d].isa = use ? en->d_isa[d] : nullptr;
    en->X.tmer[d] = use ? en->d_tmer[d] : nullptr;
  }
  en->X.tmer_len = use ? tmer_symbols(en) : 0;
  en->X.text = use ? en->d_text + kTextPad : nullptr;
  return use ? 1 : 0;
}

int engine_full_rows(Engine* en) { return en->X.text ? 1 : 0; }

int engine_drop_full_rows(Engine* en, std::string* err) {
  HPG_CUDA(cudaSetDevice(en->device), "cudaSetDevice");
  HPG_CUDA(cudaStreamSynchronize(en->stream), "drop full suffix arrays");
  graph_plans_drop_text(en);
  for (DevBuf* b : {&en->b_packed, &en->b_text, &en->b_one}) {
    cudaFree(b->p);
    *b = DevBuf();
  }
  free_full_rows(en);
  en->last = DeviceResult();  // may have been in one of the plans
  return 0;
}

int build_full_rows(Engine* en, const uint32_t n_samples[2], std::string* err) {
  const size_t n_rows = en->X.walk_mod;
  const size_t words = n_rows / 32 + 1 + 2 * kTextPad;
  const uint32_t L = tmer_symbols(en);
  const size_t tmer_bytes = ((size_t)1 << (2 * L)) * sizeof(uint2);
  const size_t need = 4 * n_rows * sizeof(uint32_t) + words * sizeof(uint64_t) + 2 * tmer_bytes;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || need > free_b / 4) {
    cudaGetLastError();
    return 0;
  }
  bool ok = cudaMalloc(&en->d_text, words * sizeof(uint64_t)) == cudaSuccess;
  for (int d = 0; d < 2 && ok; ++d)
    ok = cudaMalloc(&en->d_sa[d], n_rows * 4) == cudaSuccess && cudaMalloc(&en->d_isa[d], n_rows * 4) == cudaSuccess;
  for (int d = 0; d < 2 && ok; ++d) ok = cudaMalloc(&en->d_tmer[d], tmer_bytes) == cudaSuccess;
  unsigned long long* bad = nullptr;
  ok = ok && cudaMalloc(&bad, 4 * sizeof(*bad)) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    cudaFree(bad);
    free_full_rows(en);
    return 0;
  }
  cudaMemset(en->d_text, 0, words * sizeof(uint64_t));
  cudaMemset(bad, 0, 4 * sizeof(*bad));
  for (int d = 0; d < 2; ++d) {
    // rows that no walk reaches (a corrupt index, refused below) must not hold garbage
    cudaMemset(en->d_sa[d], 0, n_rows * 4);
    cudaMemset(en->d_isa[d], 0, n_rows * 4);
    count_launches(1);
    full_rows_kernel<<<(unsigned)en->num_sms * 8, 256>>>(en->X, (uint32_t)d, n_samples[d], en->d_sa[d], en->d_isa[d],
                                                         en->d_text + kTextPad, bad + 2 * d);
  }
  unsigned long long h[4] = {0, 0, 0, 0};
  cudaError_t ce = cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost);
  cudaFree(bad);
  if (ce != cudaSuccess) {
    *err = std::string("full suffix arrays: ") + cudaGetErrorString(ce);
    return -1;
  }
  if (h[0] || h[2] || h[1] != n_rows || h[3] != n_rows) {  // not consistent: the sampled arrays serve this index
    free_full_rows(en);
    return 0;
  }
  for (uint32_t d = 0; d < 2; ++d) launch_build_kmer(en->X, d, L, en->d_tmer[d], 0);
  if ((ce = cudaDeviceSynchronize()) != cudaSuccess) {
    *err = std::string("full suffix arrays: ") + cudaGetErrorString(ce);
    return -1;
  }
  engine_set_full_rows(en, 1);
  return 0;
}

}  // namespace hpgbwt
