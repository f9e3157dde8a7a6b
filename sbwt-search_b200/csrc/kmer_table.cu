// The k-mer table of an index: every k-mer of the SBWT (k <= 31) -> its node,
// in an open-addressing hash table on the device.  It extends the presearch
// idea (a table lookup replaces the first p search steps) to the whole
// k-mer: a read k-mer that cannot be reached by a stream step from the
// previous k-mer costs one table lookup instead of a presearch lookup and
// k - p backward-search steps.  (A failed stream step still starts the
// absent-prefix probe, which proves a run of the following k-mers absent
// with one presearch lookup.)  Results are identical: the table holds exactly
// the k-mers of the SBWT with their nodes.
//
// Labels are recovered from the SBWT itself: the last char of node v is the
// c with C[c] <= v < C[c + 1] (node 0 is the root, all '$'), and its
// predecessor (the node whose marked c-edge reaches v) is the
// (v - C[c])-th set bit of vector c: the set bits of A, C, G and T, one vector
// after the other, are the predecessors of the nodes 1, 2, ...  A node's last m
// chars and the node m steps back give its last 2 m chars and the node 2 m
// steps back with one look at that node's own, so a label takes about
// 1.6 log2(k) passes over the nodes instead of k; a node whose chain reaches
// the root within k chars is a dummy ($-padded) and is not a k-mer.
//
// Table: 2^m slots of 16 bytes (key, value), value = the node, with the k-mer's
// position in the path cover (path_cover.cu) in the high half when the index
// has one; key = the k chars with the first char on top (2 bits each), empty
// = ~0; a key's probe sequence starts at an
// even slot (so a 32-byte sector holds the first two slots it probes) and
// moves one slot at a time; at most half of the slots are used.
//
// Filter: beside the table, a blocked Bloom filter of the same keys, 10 bits
// per k-mer, one 64-bit word per key with four of its bits set
// (kmer_filter_word / kmer_filter_bits).  It is 25x smaller than the table
// (144 MB for 115 M k-mers against 4 GiB), so a read k-mer that is absent
// -- most k-mers that a stream step cannot reach -- is answered from a
// structure inside the GPU's address-translation reach and mostly in L2,
// and only k-mers the filter passes pay a table lookup.  A filter answer of
// "absent" is exact (no false negatives), so results do not change.
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>

#include "index_internal.hpp"
#include "rank_blocks.cuh"
#include "table_budget.hpp"

namespace sbwt {

namespace {

// Word w of a bitvector, read from its rank blocks (three payload words per
// block, in order).
__device__ __forceinline__ uint64_t vec_word(const Block *blocks, uint64_t w) {
  const Block &b = blocks[w / 3];
  const uint32_t j = (uint32_t)(w % 3);
  return j == 0 ? b.w0 : (j == 1 ? b.w1 : b.w2);
}

// Set bits of each word of the four vectors, one vector after the other.
__global__ void word_ones_kernel(SbwtView s, uint64_t n_words, uint64_t *cnt) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < 4 * n_words; i += step)
    cnt[i] = __popcll(vec_word(s.blocks[i / n_words], i % n_words));
}

// prev[1 + i] = position of the i-th of these set bits (n nodes; prev[0] = 0).
template <class I>
__global__ void prev_kernel(SbwtView s, uint64_t n_words, const uint64_t *off, uint64_t n,
                            I *prev) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i0 == 0) prev[0] = 0;
  for (uint64_t i = i0; i < 4 * n_words; i += step) {
    const uint64_t w = i % n_words;
    uint64_t m = vec_word(s.blocks[i / n_words], w), o = 1 + off[i];
    for (; m && o < n; m &= m - 1) {
      const uint64_t at = w * 64 + __ffsll((long long)m) - 1;
      prev[o++] = at < n ? (I)at : 0;
    }
  }
}

// The last chars of a node (the last one in the low bits) and the node that
// many steps back.
template <class I>
struct __align__(16) Back {
  uint64_t chars;
  I node;
};

__device__ __forceinline__ uint64_t last_char(const SbwtView &s, uint64_t v) {
  return (v >= s.c_map[1]) + (v >= s.c_map[2]) + (v >= s.c_map[3]);  // 0 for the root
}

template <class I>
__global__ void back_one_kernel(SbwtView s, uint64_t n, const I *prev, Back<I> *out) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step)
    out[v] = Back<I>{last_char(s, v), prev[v]};
}
// m steps back -> 2 m steps back.
template <class I>
__global__ void back_double_kernel(uint64_t n, uint32_t m, const Back<I> *in, Back<I> *out) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    const Back<I> a = in[v], b = in[a.node];
    out[v] = Back<I>{a.chars | b.chars << (2 * m), b.node};
  }
}
// m steps back -> m + 1 steps back.
template <class I>
__global__ void back_next_kernel(SbwtView s, uint64_t n, uint32_t m, const I *prev,
                                 Back<I> *back) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    const Back<I> a = back[v];
    back[v] = Back<I>{a.chars | last_char(s, a.node) << (2 * m), prev[a.node]};
  }
}
// k - 1 steps back -> the label and whether the node is a k-mer.
template <class I>
__global__ void label_kernel(SbwtView s, uint64_t n, uint32_t k, const Back<I> *back,
                             uint64_t *key, uint8_t *alive) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    const Back<I> a = back[v];
    key[v] = a.chars | last_char(s, a.node) << (2 * (k - 1));
    alive[v] = a.node != 0;
  }
}

// k-mers (alive nodes), one atomic per warp
__global__ void count_alive_kernel(const uint8_t *alive, uint64_t n, unsigned long long *out) {
  unsigned long long c = 0;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step)
    c += alive[v];
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// pos: the k-mers' positions in the path cover (the high half of a slot's
// value), or nullptr.
__global__ void table_insert_kernel(const uint64_t *key, const uint8_t *alive, uint64_t n,
                                    const uint32_t *pos, uint64_t *table, uint64_t mask,
                                    uint32_t *err) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    if (!alive[v]) continue;
    const unsigned long long kk = key[v];
    uint64_t s = kmer_table_bucket(kk, mask);
    for (uint64_t tries = 0; tries <= mask; ++tries) {
      const unsigned long long old =
          atomicCAS((unsigned long long *)(table + 2 * s), ~0ULL, kk);
      if (old == ~0ULL) {
        table[2 * s + 1] = pos ? v | (uint64_t)pos[v] << 32 : v;
        break;
      }
      if (old == kk) {  // a k-mer twice: the SBWT is malformed
        atomicOr(err, 1u);
        break;
      }
      s = (s + 1) & mask;
    }
  }
}

__global__ void filter_insert_kernel(const uint64_t *key, const uint8_t *alive, uint64_t n,
                                     unsigned long long *filter, uint64_t n_words) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    if (!alive[v]) continue;
    const uint64_t z = kmer_mix(key[v]);
    atomicOr(filter + kmer_filter_word(z, n_words), (unsigned long long)kmer_filter_bits(z));
  }
}

unsigned grid_of(uint64_t n) {
  return (unsigned)std::max<uint64_t>(std::min<uint64_t>((n + 255) / 256, 148 * 32), 1);
}

}  // namespace

// Labels of all nodes; `prev` and the two arrays of n Back records are scratch,
// key and alive come to lie in one of the two arrays.
template <class I>
static void recover_labels(const SbwtView &s, u64 n, u32 k, I *prev, Back<I> *a, Back<I> *b,
                           u64 **key, u8 **alive) {
  const u64 nw = (n + 63) / 64;
  u64 *const cnt = reinterpret_cast<u64 *>(b);  // 4 nw + 1 words, before b is used
  DeviceBuffer tmp;
  size_t tb = 0;
  word_ones_kernel<<<grid_of(4 * nw), 256>>>(s, nw, cnt);
  SBWT_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, cnt, cnt, (int64_t)(4 * nw)));
  tmp.resize(std::max<size_t>(tb, 1));
  SBWT_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tb, cnt, cnt, (int64_t)(4 * nw)));
  SBWT_CUDA(cudaMemsetAsync(prev, 0, n * sizeof(I)));  // should the vectors lack bits
  prev_kernel<I><<<grid_of(4 * nw), 256>>>(s, nw, cnt, n, prev);
  back_one_kernel<I><<<grid_of(n), 256>>>(s, n, prev, a);
  // m from 1 to k - 1 by the bits of k - 1: double, and one more for a set bit
  u32 m = 1;
  int bit = 31 - __builtin_clz(k - 1);
  for (--bit; bit >= 0; --bit) {
    back_double_kernel<I><<<grid_of(n), 256>>>(n, m, a, b);
    std::swap(a, b);
    m *= 2;
    if (((k - 1) >> bit) & 1u) {
      back_next_kernel<I><<<grid_of(n), 256>>>(s, n, m, prev, a);
      ++m;
    }
  }
  *key = reinterpret_cast<u64 *>(b);
  *alive = reinterpret_cast<u8 *>(*key + n);
  label_kernel<I><<<grid_of(n), 256>>>(s, n, k, a, *key, *alive);
  SBWT_CUDA(cudaGetLastError());
  SBWT_CUDA(cudaDeviceSynchronize());  // tmp goes
}

// Builds the table from the index's rank blocks.  Returns false (and builds
// nothing) when k > 31, when the vectors' set bits are not one per node (no
// SBWT), or when the table would not fit in kKmerTableMaxBytes or
// kmer_table_budget of the free device memory.
bool IndexImpl::build_kmer_table() {
  DeviceGuard g(device);
  drop_kmer_table();
  if (k > 31 || k < 2 || c_map[4] != num_bits) return false;
  const u64 n = num_bits;
  size_t free_b = 0, total_b = 0;
  SBWT_CUDA(cudaMemGetInfo(&free_b, &total_b));
  const u64 budget = kmer_table_budget(free_b, n);
  // one allocation: two arrays of 16-byte records, and the predecessors
  const bool narrow = n < (1ULL << 32) - 1;
  const u64 rec_bytes = (n * 16 + 4096 + 255) / 256 * 256;
  DeviceBuffer arena;
  try {
    arena.resize(2 * rec_bytes + n * (narrow ? 4 : 8));
  } catch (const Error &e) {
    if (e.code != SBWT_E_OOM) throw;
    cudaGetLastError();
    return false;  // every search also works without the table
  }
  u8 *const rec[2] = {arena.get<u8>(), arena.get<u8>() + rec_bytes};
  u8 *const prev = arena.get<u8>() + 2 * rec_bytes;
  u64 *key = nullptr;
  u8 *alive = nullptr;
  if (narrow)
    recover_labels(view, n, k, reinterpret_cast<u32 *>(prev),
                   reinterpret_cast<Back<u32> *>(rec[0]), reinterpret_cast<Back<u32> *>(rec[1]),
                   &key, &alive);
  else
    recover_labels(view, n, k, reinterpret_cast<u64 *>(prev),
                   reinterpret_cast<Back<u64> *>(rec[0]), reinterpret_cast<Back<u64> *>(rec[1]),
                   &key, &alive);
  // the record array that does not hold the labels is free from here on
  u8 *const free_rec = reinterpret_cast<u8 *>(key) == rec[0] ? rec[1] : rec[0];
  // k-mer count -> table size (load <= 1/2)
  DeviceBuffer d_n(16);  // the count, an error word
  SBWT_CUDA(cudaMemset(d_n.get(), 0, 16));
  count_alive_kernel<<<grid_of(n), 256>>>(alive, n, d_n.get<unsigned long long>());
  SBWT_CUDA(cudaGetLastError());
  u64 n_kmers = 0;
  SBWT_CUDA(cudaMemcpy(&n_kmers, d_n.get(), 8, cudaMemcpyDeviceToHost));
  u64 slots = 2;
  while (slots < 2 * n_kmers) slots <<= 1;
  const u64 filter_words = std::max<u64>((n_kmers * kFilterBitsPerKmer + 63) / 64, 1);
  if (slots > (1ULL << 32) || slots * 16 > kKmerTableMaxBytes ||
      slots * 16 + filter_words * 8 > budget)
    return false;
  // the path cover first: the table's values hold its positions.  An index
  // that cannot have it (or no memory for it) keeps the table alone.
  u32 *pos = reinterpret_cast<u32 *>(prev);  // the predecessors are done with
  try {
    if (!narrow || !build_path_cover(key, alive, n_kmers, pos, free_rec, rec_bytes)) pos = nullptr;
  } catch (const Error &e) {
    if (e.code != SBWT_E_OOM) throw;
    cudaGetLastError();
    pos = nullptr;
    drop_path_cover();
  }
  try {
    kmer_table.resize(slots * 16);
    kmer_filter.resize(filter_words * 8);
  } catch (const Error &e) {  // no room beside the temporaries (see kmer_table_budget)
    if (e.code != SBWT_E_OOM) throw;
    cudaGetLastError();
    drop_kmer_table();
    return false;
  }
  SBWT_CUDA(cudaMemset(kmer_table.get(), 0xFF, slots * 16));
  table_insert_kernel<<<grid_of(n), 256>>>(key, alive, n, pos, kmer_table.get<u64>(), slots - 1,
                                           d_n.get<uint32_t>() + 2);
  SBWT_CUDA(cudaGetLastError());
  uint32_t e = 0;
  SBWT_CUDA(cudaMemcpy(&e, d_n.get<uint32_t>() + 2, 4, cudaMemcpyDeviceToHost));
  if (e) {
    drop_kmer_table();
    throw Error(SBWT_E_FORMAT, "an SBWT k-mer occurs twice");
  }
  SBWT_CUDA(cudaMemset(kmer_filter.get(), 0, filter_words * 8));
  filter_insert_kernel<<<grid_of(n), 256>>>(key, alive, n, kmer_filter.get<unsigned long long>(),
                                            filter_words);
  SBWT_CUDA(cudaGetLastError());
  view.kmer_table = kmer_table.get<u64>();
  view.kmer_table_mask = slots - 1;
  view.node_mask = view.path_node ? 0xFFFFFFFFULL : ~0ULL;
  view.kmer_filter = kmer_filter.get<u64>();
  view.filter_words = filter_words;
  table_kmers = n_kmers;
  return true;
}

void IndexImpl::drop_kmer_table() {
  DeviceGuard g(device);
  kmer_table.release();
  kmer_filter.release();
  drop_path_cover();
  view.kmer_table = nullptr;
  view.kmer_table_mask = 0;
  view.kmer_filter = nullptr;
  view.filter_words = 0;
  table_kmers = 0;
}

}  // namespace sbwt
