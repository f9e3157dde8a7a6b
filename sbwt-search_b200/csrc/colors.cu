// Colors step on the B200: per-read color counting and the tau threshold.
//
// Reference behaviour restated (SBWT-Search, paths in its src/):
//   d_color_search   ColorSearcher/ColorSearcher.cuh:68-206 (+ helpers :208-318)
//   d_post_process   ColorSearcher/ColorPostProcessor.cuh:21-43
//   threshold        ColorResultsPrinter/ContinuousColorResultsPrinter.hpp:235-263
//   .tcolors layout  ColorIndexBuilder/ColorIndexBuilder.cpp:23-86
//
// Semantics: count[r][c] = number of found k-mers of read r whose color set
// holds c.  The reference gets there with one thread per k-mer, a warp-wide
// loop over the color span and u8 per-(warp, color) partial counts summed by
// a second kernel into an R x C u64 matrix copied to the host.  Here one warp
// owns one read and one tile of 2048 colors (more colors -> more tiles per
// read): lane i owns colors [64 i, 64 i + 64) of the tile as bit-sliced
// counters in registers (plane j holds bit j of 64 counters).  K-mers in a
// row that share a color set count as one entry with their number; the rows
// of dense sets met once are added eight at a time through a carry-save tree,
// the others (and sparse sets, turned into row words in shared memory) with
// their weight.  The threshold is a bit-sliced comparison; only the passing
// color bits leave the kernel, and of those only the words that hold one.
// Each k-mer's set is one 8-byte record load from a per-node table when that
// table is resident (else rank over the key k-mer marks, color set index,
// record).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <type_traits>
#include <vector>

#include "colors_internal.hpp"
#include "common.hpp"
#include "formats.hpp"
#include "rank_blocks.cuh"

namespace sbwt {

constexpr int kColorWarps = 4;  // warps (reads in flight) per block

__device__ __forceinline__ uint64_t rec_start(uint64_t rec) { return rec >> (kRecLenBits + 1); }
__device__ __forceinline__ uint32_t rec_len(uint64_t rec) {
  return (uint32_t)(rec >> 1) & ((1u << kRecLenBits) - 1);
}

struct ColorsJob {
  const uint64_t *vals;     // SBWT indexes (markers allowed when counted)
  const uint64_t *offs;     // n_reads + 1
  const uint64_t *not_found;  // per read or nullptr
  const uint64_t *invalid;    // per read or nullptr
  uint64_t n_reads;
  const uint64_t *list;     // the reads to do (n_list of them), nullptr: all
  uint64_t n_list;
  double tau;
  uint32_t include_not_found, include_invalid;
  // mode 0: passing colors.  Of the row words of a (read, tile), those with a
  // passing color (bit i of word_mask[read * tiles + tile]: word i), in order
  // from pass_bits[read * row_words + 32 * tile].
  uint64_t *pass_bits;      // n_reads x row_words
  uint32_t *word_mask;      // n_reads x tiles
  uint32_t *pass_count;     // n_reads
  uint32_t *counts;         // n_reads x num_colors (mode 1)
};

__device__ __forceinline__ uint64_t rank_key(const ColorsView &cv, uint64_t i) {
  const uint64_t b = i / kBlockBits;
  const Block B = load_block(cv.key_blocks + b);
  return cv.key_l0[b >> kSuperchunkShift] + block_rank(B, (uint32_t)(i - b * kBlockBits));
}

// The packed set record of SBWT index v < key_bits: the set of key k-mer
// number rank(key_marks, v), as the reference's ColorSearcher resolves it
// (rank of v among the key k-mer marks, then color_set_idxs).  kRecNone when
// the rank is past the last key k-mer.  DIRECT reads the per-node table that
// holds exactly these values.
template <bool DIRECT>
__device__ __forceinline__ uint64_t set_record(const ColorsView &cv, uint64_t v) {
  if (DIRECT) return __ldg(cv.node_rec + v);
  const uint64_t j = rank_key(cv, v);
  if (j >= cv.n_keys) return kRecNone;
  const uint32_t s = __ldg(cv.csi + j);
  return s < cv.n_sets ? __ldg(cv.recs + s) : kRecNone;
}

// out[i] = entry i of an sdsl int vector of `width` bits per entry (LSB-first
// in 64-bit words); entries >= limit set *err and read as 0.
__global__ void unpack_set_indexes_kernel(const uint64_t *words, uint64_t n, uint32_t width,
                                          uint64_t limit, uint32_t *out, uint32_t *err) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t mask = width >= 64 ? ~0ULL : (1ULL << width) - 1;
  uint32_t bad = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += step) {
    const uint64_t bit = i * width, w = bit >> 6, o = bit & 63;
    uint64_t v = words[w] >> o;
    if (o + width > 64) v |= words[w + 1] << (64 - o);
    v &= mask;
    if (v >= limit) {
      bad = 1;
      v = 0;
    }
    out[i] = (uint32_t)v;
  }
  if (__any_sync(0xFFFFFFFFu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, 1u);
}

// node_rec[v] = set_record(v) for every v < key_bits.
__global__ void node_record_kernel(ColorsView cv, uint64_t *out) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < cv.key_bits; v += step)
    out[v] = set_record<false>(cv, v);
}

// Error bits of the colors kernel.
enum : uint32_t { kErrNode = 1, kErrLong = 2, kErrOffsets = 4 };

constexpr int kWindows = 4;                  // windows of 32 k-mers looked up together
constexpr int kChunk = 32 * kWindows;        // k-mers of one round
constexpr int kRows = 8;                     // dense rows of one carry-save tree
constexpr int kOthers = 4;                   // other rows loaded together
constexpr int kListSlots = kChunk + 16;      // runs of a round, padded at either end
static_assert(kRows + kOthers <= 16 && kListSlots * 16 >= 32 * 9 * 8, "list size");
// Counter planes of the kernels: reads of at most 255, 65535 and 2^40 - 1 k-mers.
constexpr int kPlanes[3] = {8, 16, 40};

// One run of k-mers that share a color set.
struct __align__(16) Run {
  unsigned long long start;  // of the set's words (dense) or ids (sparse)
  uint32_t len;              // words or ids, kSparse: ids
  uint32_t weight;           // k-mers
};
constexpr uint32_t kSparse = 1u << 31;

// s, c: sum and carry of three one-bit numbers, 64 at a time.
__device__ __forceinline__ uint64_t csa(uint64_t &s, uint64_t a, uint64_t b) {
  const uint64_t c = (s & a) | (s & b) | (a & b);
  s ^= a ^ b;
  return c;
}

// Adds x (one bit per color) at plane J0: ripple carry.  Warp-uniform control;
// above plane 8 it stops when no lane has a carry left.
template <int P, int J0>
__device__ __forceinline__ void add_at(uint64_t (&p)[P], uint64_t x) {
#pragma unroll
  for (int j = J0; j < P; ++j) {
    if (j >= 8 && !__any_sync(0xFFFFFFFFu, x != 0)) break;
    const uint64_t t = p[j] & x;
    p[j] ^= x;
    x = t;
  }
}

// Adds m (<= 32) copies of row word x.
template <int P>
__device__ __forceinline__ void add_weighted(uint64_t (&p)[P], uint64_t x, uint32_t m) {
  uint64_t c = 0;
#pragma unroll
  for (int j = 0; j < P; ++j) {
    if (j >= 8 && !__any_sync(0xFFFFFFFFu, c != 0)) break;
    const uint64_t a = j < 6 && ((m >> j) & 1u) ? x : 0;
    const uint64_t t = (p[j] & a) | (p[j] & c) | (a & c);
    p[j] ^= a ^ c;
    c = t;
  }
}

// Adds eight row words.
template <int P>
__device__ __forceinline__ void add_rows(uint64_t (&p)[P], const uint64_t (&x)[kRows]) {
  const uint64_t a = csa(p[0], x[0], x[1]), b = csa(p[0], x[2], x[3]);
  const uint64_t c = csa(p[1], a, b);
  const uint64_t d = csa(p[0], x[4], x[5]), e = csa(p[0], x[6], x[7]);
  const uint64_t f = csa(p[1], d, e);
  add_at<P, 3>(p, csa(p[2], c, f));
}

// This lane's row word of the sparse list ids[0, n) (n <= 32, id: the lane's
// one) for the row words [wbase, wbase + 32): each lane ORs its id's bit into
// the warp's 32 zeroed words of shared memory and takes its own word back.
__device__ __forceinline__ uint64_t sparse_word(uint64_t *stage, uint32_t lane, uint32_t id,
                                                bool in, uint32_t wbase) {
  const uint32_t local = (id >> 6) - wbase;  // wraps past 32 when below the tile
  if (in && local < 32) atomicOr((unsigned long long *)(stage + local), 1ULL << (id & 63));
  __syncwarp();
  const uint64_t x = stage[lane];
  if (x) stage[lane] = 0;
  __syncwarp();
  return x;
}

// 8 x 8 bit transpose: byte j of (hi, lo) holds bit j of eight counters; byte
// i of the result is counter i.
__device__ __forceinline__ uint64_t transpose8(uint64_t x) {
  uint64_t t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAULL;
  x ^= t ^ (t << 7);
  t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCULL;
  x ^= t ^ (t << 14);
  t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ULL;
  return x ^ t ^ (t << 28);
}

// Counters of planes [J0, J0 + 8) of this lane's colors 8 q .. 8 q + 7, a byte each.
template <int P, int J0>
__device__ __forceinline__ uint64_t counter_bytes(const uint64_t (&p)[P], int q) {
  uint64_t x = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (J0 + j < P) x |= ((p[J0 + j] >> (8 * q)) & 0xFF) << (8 * j);
  return transpose8(x);
}

// One warp per work item (read r, color tile): tile t covers row words
// [32 t, 32 t + 32), lane i owns word 32 t + i.  The k-mers are taken kChunk
// at a time: every lane loads the set records of kWindows k-mers together,
// equal records in a row become one run, and the runs are added from a list
// in shared memory: the dense ones of weight 1 from the front, kRows per
// carry-save tree, the others from the back.  Counts are sums, so the order
// and grouping of the adds does not change them.
// MODE 0: passing color words + count per read; MODE 1: full counts.  P: the
// counter planes; a read of 2^P or more k-mers sets kErrLong and is left out.
//
// What bounds it: instructions, 2,325 warp instructions per read of 120 k-mers
// with 2000 colors (ALU pipe 74 %), beside the rows (11 KB a read, 8.5 KB of them
// from DRAM).  Planes in shared memory with one ripple per row took 7,324 (8.3 ms
// for 1 M reads; now 3.2 ms, see ColorsImpl::launch).
template <int MODE, bool DIRECT, int P>
__global__ void __launch_bounds__(32 * kColorWarps, P <= 8 ? 8 : (P <= 16 ? 6 : 3))
    colors_kernel(ColorsView cv, ColorsJob job, uint32_t *err) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  __shared__ Run sh_run[kColorWarps][kListSlots];
  __shared__ uint64_t sh_stage[kColorWarps][32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5, below = (1u << lane) - 1u;
  const uint32_t T = cv.tiles;
  Run *const list = sh_run[wid];
  Run *const back = list + kListSlots - 1;  // the others, downwards
  uint64_t *const stage = sh_stage[wid];
  stage[lane] = 0;
  __syncwarp();
  const uint64_t warps = (uint64_t)gridDim.x * kColorWarps;
  const bool listed = P > kPlanes[0] && job.list;
  const uint64_t n_items = (listed ? job.n_list : job.n_reads) * T;
  const uint64_t n_vals_end = job.offs[job.n_reads];
  for (uint64_t item = blockIdx.x * (uint64_t)kColorWarps + wid; item < n_items; item += warps) {
    const uint64_t at = T == 1 ? item : item / T;
    const uint64_t r = listed ? __ldg(job.list + at) : at;
    const uint32_t tile = (uint32_t)(item - at * T), wbase = 32 * tile;
    uint64_t o0 = job.offs[r], o1 = job.offs[r + 1];
    if (o1 < o0 || o1 > n_vals_end || ((o1 - o0) >> P)) {
      if (lane == 0) atomicOr(err, o1 < o0 || o1 > n_vals_end ? kErrOffsets : kErrLong);
      o1 = o0;
    }
    uint64_t p[P];
#pragma unroll
    for (int j = 0; j < P; ++j) p[j] = 0;
    uint32_t found = 0, not_found = 0, invalid = 0;
    for (uint64_t base = o0; base < o1; base += kChunk) {
      // lookups: lane t classifies k-mers base + 32 l + t (l < kWindows)
      uint64_t v[kWindows], rec[kWindows];
      bool bad = false;
#pragma unroll
      for (int l = 0; l < kWindows; ++l) {
        const uint64_t t = base + 32 * l + lane;
        v[l] = t < o1 ? job.vals[t] : kRecNone - 2;  // past the read: neither marker
      }
#pragma unroll
      for (int l = 0; l < kWindows; ++l) {
        rec[l] = kRecNone;
        if (v[l] < cv.key_bits) {
          rec[l] = set_record<DIRECT>(cv, v[l]);
          ++found;
        } else if (v[l] == SBWT_NOT_FOUND) {
          ++not_found;
        } else if (v[l] == SBWT_INVALID) {
          ++invalid;
        } else if (base + 32 * l + lane < o1) {
          bad = true;
        }
      }
      uint32_t n_dense = 0, n_other = 0;
#pragma unroll
      for (int l = 0; l < kWindows; ++l) {
        const uint64_t x = rec[l];
        if (x == kRecNone && v[l] < cv.key_bits) bad = true;
        // runs of equal records
        const uint64_t before = __shfl_up_sync(FULL, x, 1);
        const bool head = lane == 0 || x != before;
        const uint32_t heads = __ballot_sync(FULL, head);
        const uint32_t next = heads & ~(below | (1u << lane));
        const uint32_t weight = (next ? (uint32_t)__ffs(next) - 1u : 32u) - lane;
        const bool run = head && x != kRecNone, single = (x & 1ULL) && weight == 1;
        const uint32_t md = __ballot_sync(FULL, run && single);
        const uint32_t mo = __ballot_sync(FULL, run && !single);
        if (run) {
          Run *const e = single ? list + n_dense + __popc(md & below)
                                : back - (n_other + __popc(mo & below));
          *e = Run{rec_start(x), rec_len(x) | (x & 1ULL ? 0u : kSparse), weight};
        }
        n_dense += __popc(md);
        n_other += __popc(mo);
      }
      if (bad) atomicOr(err, kErrNode);
      __syncwarp();
      // the lists hold at most kChunk runs, so neither pad reaches the other
      if (lane < kRows) list[n_dense + lane].len = 0;
      __syncwarp();
      for (uint32_t i = 0; i < n_dense; i += kRows) {
        uint64_t x[kRows];
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
          const Run e = list[i + u];
          x[u] = wbase + lane < e.len ? __ldg(cv.dense + e.start + (wbase + lane)) : 0;
        }
        add_rows<P>(p, x);
      }
      if (lane < kOthers) {
        (back - n_other - lane)->len = 0;
        (back - n_other - lane)->weight = 0;
      }
      __syncwarp();
      for (uint32_t i = 0; i < n_other; i += kOthers) {
        // the row word of a dense set, the first 32 ids of a sparse one
        uint64_t x[kOthers];
#pragma unroll
        for (int u = 0; u < kOthers; ++u) {
          const Run e = *(back - i - u);
          x[u] = 0;
          if (e.len & kSparse) {
            if (lane < (e.len & ~kSparse)) x[u] = __ldg(cv.sparse + e.start + lane);
          } else if (wbase + lane < e.len) {
            x[u] = __ldg(cv.dense + e.start + (wbase + lane));
          }
        }
#pragma unroll
        for (int u = 0; u < kOthers; ++u) {
          const Run e = *(back - i - u);
          if (e.weight == 0) break;
          uint64_t y = x[u];
          if (e.len & kSparse) {
            const uint32_t len = e.len & ~kSparse;
            y = 0;
            for (uint32_t c0 = 0; c0 < len; c0 += 32) {
              const bool in = c0 + lane < len;
              uint32_t id = (uint32_t)x[u];
              if (c0) id = in ? __ldg(cv.sparse + e.start + c0 + lane) : 0;
              if (T > 1 && cv.sparse_sorted) {  // ascending ids: only chunks in the tile
                const uint32_t last = min(32u, len - c0) - 1;
                if ((__shfl_sync(FULL, id, last) >> 6) < wbase) continue;
                if ((__shfl_sync(FULL, id, 0) >> 6) >= wbase + 32) break;
              }
              y |= sparse_word(stage, lane, id, in, wbase);
            }
          }
          if (__any_sync(FULL, y != 0)) add_weighted<P>(p, y, e.weight);
        }
      }
      __syncwarp();
    }
    // per-read sizes
    found = __reduce_add_sync(FULL, found);
    not_found = __reduce_add_sync(FULL, not_found);
    invalid = __reduce_add_sync(FULL, invalid);
    const uint32_t word = wbase + lane;
    if (MODE == 0) {
      if (job.not_found) not_found += (uint32_t)job.not_found[r];
      if (job.invalid) invalid += (uint32_t)job.invalid[r];
      const uint64_t size = (uint64_t)found + (job.include_not_found ? not_found : 0) +
                            (job.include_invalid ? invalid : 0);
      const uint64_t minimum = (uint64_t)ceil((double)size * job.tau);
      uint64_t ge = 0;
      if (minimum > 0 && word < cv.row_words && (minimum >> P) == 0) {
        uint64_t gt = 0, eq = ~0ULL;
#pragma unroll
        for (int j = P - 1; j >= 0; --j) {
          if ((minimum >> j) & 1ULL) {
            eq &= p[j];
          } else {
            gt |= eq & p[j];
            eq &= ~p[j];
          }
        }
        ge = gt | eq;
        const uint32_t rem = cv.num_colors - word * 64;
        if (rem < 64) ge &= (1ULL << rem) - 1ULL;
      }
      const uint32_t mask = __ballot_sync(FULL, ge != 0);
      if (ge) job.pass_bits[r * cv.row_words + wbase + __popc(mask & below)] = ge;
      const uint32_t passing = __reduce_add_sync(FULL, (uint32_t)__popcll(ge));
      if (lane == 0) {
        job.word_mask[r * T + tile] = mask;
        if (T == 1)
          job.pass_count[r] = passing;
        else if (passing)
          atomicAdd(job.pass_count + r, passing);  // zeroed before the launch
      }
    } else {
      // counters as bytes through shared memory (the list's, free by now; a
      // lane's 64 colors are 8 words, the row stride is odd), 4 colors a lane
      // and store
      uint64_t *const bytes = reinterpret_cast<uint64_t *>(list);  // 32 x 9 words <= the list
      const uint64_t row = r * cv.num_colors + (uint64_t)wbase * 64;
      const uint32_t n = min(2048u, cv.num_colors - wbase * 64);  // colors of the tile
      const bool vec = ((reinterpret_cast<uintptr_t>(job.counts) | (row * 4)) & 15) == 0;
      auto emit = [&](auto read) {  // read(c): count of color c of the tile
        if (vec) {
          for (uint32_t c = 4 * lane; c + 4 <= n; c += 128)
            __stcs(reinterpret_cast<uint4 *>(job.counts + row + c),
                   make_uint4(read(c), read(c + 1), read(c + 2), read(c + 3)));
          const uint32_t c = (n & ~3u) + lane;
          if (c < n) job.counts[row + c] = read(c);
        } else {
          for (uint32_t c = lane; c < n; c += 32) __stcs(job.counts + row + c, read(c));
        }
      };
      auto put = [&](auto J0) {
#pragma unroll
        for (int q = 0; q < 8; ++q) bytes[9 * lane + q] = counter_bytes<P, J0.value>(p, q);
        __syncwarp();
      };
      const uint8_t *const b = reinterpret_cast<const uint8_t *>(bytes);
      auto byte = [&](uint32_t c) -> uint32_t { return b[72 * (c >> 6) + (c & 63)]; };
      put(std::integral_constant<int, 0>{});
      emit(byte);
      if (P > 8) {  // the higher bytes on top of what is written
#pragma unroll 1
        for (int j0 = 8; j0 < P; j0 += 8) {
          __syncwarp();
          if (j0 == 8) put(std::integral_constant<int, (P > 8 ? 8 : 0)>{});
          if (j0 == 16) put(std::integral_constant<int, (P > 16 ? 16 : 0)>{});
          if (j0 == 24) put(std::integral_constant<int, (P > 24 ? 24 : 0)>{});
          if (j0 == 32) break;  // counts are 32 bits
          for (uint32_t c = lane; c < n; c += 32) {
            const uint32_t x = byte(c);
            if (x) atomicAdd(job.counts + row + c, x << j0);
          }
        }
      }
      __syncwarp();
    }
    __syncwarp();
  }
}

// Expands each read's passing words into ascending color ids at ids_off[r].
// One thread per read: the words with a passing color are few; a read with
// more ids than a thread should write alone is taken by its whole warp.
constexpr uint32_t kIdsPerThread = 64;
__global__ void emit_ids_kernel(const uint64_t *pass_bits, const uint32_t *word_mask,
                                uint32_t row_words, uint32_t tiles, const uint64_t *ids_off,
                                uint64_t n_reads, uint32_t *ids, uint64_t capacity) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  if (ids_off[n_reads] > capacity) return;
  for (uint64_t r0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ULL; r0 < n_reads;
       r0 += step) {
    const uint64_t r = r0 + lane;
    uint64_t out = 0, n = 0;
    if (r < n_reads) {
      out = ids_off[r];
      n = ids_off[r + 1] - out;
    }
    if (n && n <= kIdsPerThread) {
      for (uint32_t t = 0; t < tiles; ++t) {
        uint32_t mask = word_mask[r * tiles + t];
        const uint64_t *w = pass_bits + r * row_words + 32 * t;
        for (; mask; mask &= mask - 1, ++w) {
          const uint32_t c = (32 * t + __ffs(mask) - 1) * 64;
          for (uint64_t m = *w; m; m &= m - 1, ++out) ids[out] = c + __ffsll((long long)m) - 1;
        }
      }
    }
    for (unsigned big = __ballot_sync(0xFFFFFFFFu, n > kIdsPerThread); big; big &= big - 1) {
      const int q = __ffs(big) - 1;
      const uint64_t rq = r0 + q;
      uint64_t at = __shfl_sync(0xFFFFFFFFu, out, q);
      for (uint32_t t = 0; t < tiles; ++t) {
        const uint32_t mask = word_mask[rq * tiles + t];
        uint64_t m = 0;
        if ((mask >> lane) & 1u)
          m = pass_bits[rq * row_words + 32 * t + __popc(mask & ((1u << lane) - 1u))];
        const uint32_t cnt = __popcll(m);
        uint32_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        uint64_t pos = at + incl - cnt;
        for (; m; m &= m - 1, ++pos) ids[pos] = (32 * t + lane) * 64 + __ffsll((long long)m) - 1;
        at += __shfl_sync(0xFFFFFFFFu, incl, 31);
      }
    }
  }
}

// Exclusive scan of u32 counts into u64 offsets off[0..n] in three launches
// and no scratch: block b of the first launch leaves the total of counts
// [b * kScanSpan, (b + 1) * kScanSpan) in off[b * kScanSpan], one block
// scans those totals in place (and writes off[n]), and the last launch
// replaces every block's range with its offsets.
constexpr uint32_t kScanThreads = 1024, kScanPer = 4, kScanSpan = kScanThreads * kScanPer;

// Block-wide exclusive scan of one u64 per thread; the block total comes back
// through *total.  All threads of the block must call it.
__device__ __forceinline__ uint64_t block_exclusive_scan(uint64_t v, uint64_t *total) {
  __shared__ uint64_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint64_t s = lane < blockDim.x / 32 ? wsum[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
      if (lane >= (uint32_t)o) s += y;
    }
    wsum[lane] = s;
  }
  __syncthreads();
  const uint64_t ex = (wid ? wsum[wid - 1] : 0) + x - v;
  *total = wsum[blockDim.x / 32 - 1];
  __syncthreads();  // wsum is reused by the next call
  return ex;
}

__global__ void __launch_bounds__(kScanThreads) scan_totals_kernel(const uint32_t *cnt, uint64_t n,
                                                                   uint64_t *off) {
  const uint64_t b0 = blockIdx.x * (uint64_t)kScanSpan;
  uint64_t v = 0;
  for (uint32_t k = 0; k < kScanPer; ++k) {
    const uint64_t i = b0 + k * kScanThreads + threadIdx.x;
    if (i < n) v += cnt[i];
  }
  uint64_t total = 0;
  block_exclusive_scan(v, &total);
  if (threadIdx.x == 0) off[b0] = total;
}

// total: if set, receives off[n] too.
__global__ void __launch_bounds__(kScanThreads) scan_tops_kernel(uint64_t *off, uint64_t n,
                                                                 uint64_t n_blocks,
                                                                 uint64_t *total_out) {
  uint64_t carry = 0;
  for (uint64_t b = 0; b < n_blocks; b += kScanThreads) {
    const uint64_t i = b + threadIdx.x;
    const uint64_t v = i < n_blocks ? off[i * kScanSpan] : 0;
    uint64_t total = 0;
    const uint64_t ex = block_exclusive_scan(v, &total);
    if (i < n_blocks) off[i * kScanSpan] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) {
    off[n] = carry;
    if (total_out) *total_out = carry;
  }
}

__global__ void __launch_bounds__(kScanThreads) scan_write_kernel(const uint32_t *cnt, uint64_t n,
                                                                  uint64_t *off) {
  __shared__ uint64_t base;
  const uint64_t b0 = blockIdx.x * (uint64_t)kScanSpan;
  if (threadIdx.x == 0) base = off[b0];
  __syncthreads();
  const uint64_t i0 = b0 + (uint64_t)threadIdx.x * kScanPer;
  uint32_t c[kScanPer];
  uint64_t v = 0;
#pragma unroll
  for (uint32_t k = 0; k < kScanPer; ++k) {
    c[k] = i0 + k < n ? cnt[i0 + k] : 0;
    v += c[k];
  }
  uint64_t total = 0;
  uint64_t at = base + block_exclusive_scan(v, &total);
#pragma unroll
  for (uint32_t k = 0; k < kScanPer; ++k) {
    if (i0 + k < n) off[i0 + k] = at;
    at += c[k];
  }
}

static void enqueue_scan_counts(const uint32_t *d_cnt, uint64_t n, uint64_t *d_off,
                                uint64_t *d_total, cudaStream_t st) {
  if (n == 0) {
    SBWT_CUDA(cudaMemsetAsync(d_off, 0, 8, st));
    return;
  }
  const uint64_t nb = (n + kScanSpan - 1) / kScanSpan;
  scan_totals_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(d_cnt, n, d_off);
  scan_tops_kernel<<<1, kScanThreads, 0, st>>>(d_off, n, nb, d_total);
  scan_write_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(d_cnt, n, d_off);
  SBWT_CUDA(cudaGetLastError());
}

// The reads of at least `shortest` k-mers into list, their number into out[2];
// out[0] = the longest read's k-mers; out[1] = 1 when some offset decreases.  out
// is zeroed before the launch.
__global__ void long_reads_kernel(const uint64_t *offs, uint64_t n_reads, uint64_t shortest,
                                  uint64_t *list, unsigned long long *out) {
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long m = 0, bad = 0;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ULL; r0 < n_reads;
       r0 += step) {
    const uint64_t r = r0 + lane;
    uint64_t span = 0;
    if (r < n_reads) {
      const uint64_t a = offs[r], b = offs[r + 1];
      if (b < a)
        bad = 1;
      else
        span = b - a;
    }
    m = max(m, (unsigned long long)span);
    const uint32_t found = __ballot_sync(0xFFFFFFFFu, span >= shortest);
    if (!found) continue;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(out + 2, (unsigned long long)__popc(found));
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if ((found >> lane) & 1u) list[at + __popc(found & ((1u << lane) - 1u))] = r;
  }
  for (int o = 16; o; o >>= 1) {
    m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    bad |= __shfl_xor_sync(0xFFFFFFFFu, bad, o);
  }
  if (lane == 0) {
    if (m) atomicMax(out, m);
    if (bad) atomicOr(out + 1, bad);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
void build_rank_blocks_host(const u64 *words, u64 num_bits, std::vector<Block> &blocks,
                            std::vector<u64> &l0, u64 &total);

ColorsImpl::ColorsImpl(const TColorsFile &t, int device_) {
  device = device_;
  DeviceGuard g(device);
  num_colors = t.num_colors();
  if (num_colors == 0 || num_colors > (1u << 20))
    throw Error(SBWT_E_FORMAT, "number of colors out of range");
  const u64 n_sets = t.is_dense_marks.num_bits;
  const u64 n_keys = t.color_set_idxs.size();
  const HostColorSets h = prepare_color_sets(t);
  std::vector<Block> kb;
  std::vector<u64> kl0;
  u64 total_keys = 0;
  build_rank_blocks_host(t.key_kmer_marks.words.data(), t.key_kmer_marks.num_bits, kb, kl0,
                         total_keys);
  if (total_keys > n_keys)
    throw Error(SBWT_E_FORMAT, "more key k-mers than color set indexes");
  auto up = [&](DeviceBuffer &b, const void *src, size_t bytes) {
    b.resize(bytes);
    SBWT_CUDA(cudaMemcpy(b.get(), src, bytes, cudaMemcpyHostToDevice));
  };
  up(key_blocks, kb.data(), kb.size() * sizeof(Block));
  up(key_l0, kl0.data(), kl0.size() * 8);
  up(recs_buf, h.recs.data(), h.recs.size() * 8);
  up(dense_buf, h.dense_words.data(), h.dense_words.size() * 8);
  up(sparse_buf, h.sparse.data(), h.sparse.size() * 4);
  // color set indexes: the packed int vector goes up as it is and is widened
  // to u32 on the device
  csi_buf.resize(std::max<u64>(n_keys, 1) * 4);
  if (n_keys) {
    DeviceBuffer packed, err;
    up(packed, t.color_set_idxs.words.data(), t.color_set_idxs.words.size() * 8);
    err.resize(4);
    SBWT_CUDA(cudaMemset(err.get(), 0, 4));
    const u64 blocks = std::min<u64>((n_keys + 255) / 256, 148 * 16);
    unpack_set_indexes_kernel<<<(unsigned)blocks, 256>>>(
        packed.get<u64>(), n_keys, t.color_set_idxs.width, n_sets, csi_buf.get<uint32_t>(),
        err.get<uint32_t>());
    SBWT_CUDA(cudaGetLastError());
    uint32_t bad = 0;
    SBWT_CUDA(cudaMemcpy(&bad, err.get(), 4, cudaMemcpyDeviceToHost));
    if (bad) throw Error(SBWT_E_FORMAT, "color set index out of range");
  }
  view = ColorsView{};
  view.key_blocks = key_blocks.get<Block>();
  view.key_l0 = key_l0.get<u64>();
  view.key_bits = t.key_kmer_marks.num_bits;
  view.csi = csi_buf.get<uint32_t>();
  view.n_keys = n_keys;
  view.recs = recs_buf.get<u64>();
  view.n_sets = n_sets;
  view.dense = dense_buf.get<u64>();
  view.sparse = sparse_buf.get<uint32_t>();
  view.num_colors = (uint32_t)num_colors;
  view.row_words = (uint32_t)((num_colors + 63) / 64);
  view.tiles = (view.row_words + 31) / 32;  // 32 row words (2048 colors) per warp
  view.sparse_sorted = h.sparse_sorted ? 1 : 0;
  set_node_table(true);
}

u64 ColorsImpl::device_footprint() const {
  return key_blocks.size() + key_l0.size() + csi_buf.size() + recs_buf.size() +
         dense_buf.size() + sparse_buf.size() + node_buf.size();
}

// The per-node record table turns the k-mer -> color set lookup (rank block,
// color set index, set record: three dependent random loads) into one load.
// It costs 8 bytes per SBWT node and is only built when that stays within
// kNodeTableMaxBytes and half of the free device memory.
bool ColorsImpl::set_node_table(bool enable) {
  DeviceGuard g(device);
  view.node_rec = nullptr;
  node_buf.release();
  if (enable) {
    const u64 bytes = std::max<u64>(view.key_bits, 1) * 8;
    size_t free_b = 0, total_b = 0;
    SBWT_CUDA(cudaMemGetInfo(&free_b, &total_b));
    if (bytes <= kNodeTableMaxBytes && bytes <= free_b / 2) {
      node_buf.resize(bytes);
      const u64 blocks = std::min<u64>((view.key_bits + 255) / 256, 148 * 16);
      node_record_kernel<<<(unsigned)std::max<u64>(blocks, 1), 256>>>(view, node_buf.get<u64>());
      SBWT_CUDA(cudaGetLastError());
      SBWT_CUDA(cudaDeviceSynchronize());
      view.node_rec = node_buf.get<u64>();
    }
  }
  device_bytes = device_footprint();
  return view.node_rec != nullptr;
}

struct ColorsWorkspace {
  int device = -1;
  DeviceBuffer vals, offs, nf, inv, pass_bits, pass_count, ids_off, ids, counts, status, span, list;
  cudaStream_t stream = nullptr;
  u64 *status_host = nullptr;  // pinned: the error bits, the id count
  uint32_t *err() { return status.get<uint32_t>(); }
  u64 *total() { return status.get<u64>() + 1; }
  ~ColorsWorkspace() {
    if (stream) cudaStreamDestroy(stream);
    if (status_host) cudaFreeHost(status_host);
  }
};

static ColorsWorkspace &colors_workspace(int device) {
  thread_local std::unique_ptr<ColorsWorkspace> ws[16];
  if (device < 0 || device >= 16) throw Error(SBWT_E_INVALID, "device id out of range");
  auto &p = ws[device];
  if (!p) {
    p = std::make_unique<ColorsWorkspace>();
    p->device = device;
    SBWT_CUDA(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    SBWT_CUDA(cudaMallocHost(&p->status_host, 16));
    p->status.resize(16);
    SBWT_CUDA(cudaMemset(p->status.get(), 0, 16));
  }
  return *p;
}

// Counter planes of a batch whose reads have at most max_kmers k-mers.
static int planes_for(u64 max_kmers) {
  for (int P : kPlanes)
    if ((max_kmers >> P) == 0) return P;
  throw Error(SBWT_E_INVALID, "a read has too many k-mers");
}

// Runs the colors kernel on device-resident arrays.  mode 0 -> passing words
// + counts; mode 1 -> counts.  A read of 2^planes or more k-mers sets kErrLong
// in *d_err.  d_word_mask: n_reads x tiles.  d_list: if set, the n_list reads
// that are done (after a launch over all of them, with more planes).
// One B200, 1 M reads of 120 k-mers: 2000 colors 8.31 -> 3.20 ms.
void ColorsImpl::launch(const u64 *d_vals, const u64 *d_offs, const u64 *d_nf,
                        const u64 *d_inv, u64 n_reads, int planes, double tau,
                        u32 flags, int mode, u64 *d_pass_bits, uint32_t *d_word_mask,
                        uint32_t *d_pass_count, uint32_t *d_counts, uint32_t *d_err,
                        cudaStream_t st, const u64 *d_list, u64 n_list) const {
  if (n_reads == 0) return;
  ColorsJob job{};
  job.vals = d_vals;
  job.offs = d_offs;
  job.not_found = d_nf;
  job.invalid = d_inv;
  job.n_reads = n_reads;
  job.list = d_list;
  job.n_list = n_list;
  job.tau = tau;
  job.include_not_found = (flags & SBWT_INCLUDE_NOT_FOUND) ? 1 : 0;
  job.include_invalid = (flags & SBWT_INCLUDE_INVALID) ? 1 : 0;
  if (mode == 0 && view.tiles > 1 && !d_list)  // tiles of a read add their passing counts
    SBWT_CUDA(cudaMemsetAsync(d_pass_count, 0, n_reads * 4, st));
  job.pass_bits = d_pass_bits;
  job.word_mask = d_word_mask;
  job.pass_count = d_pass_count;
  job.counts = d_counts;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const u64 items = (d_list ? n_list : n_reads) * view.tiles;
  const u64 blocks = std::min<u64>((items + kColorWarps - 1) / kColorWarps, (u64)sms * 32);
  const bool direct = view.node_rec != nullptr;
  auto go = [&](auto kernel) {
    kernel<<<(unsigned)blocks, 32 * kColorWarps, 0, st>>>(view, job, d_err);
  };
#define SBWT_COLORS(M_, P_) (direct ? go(colors_kernel<M_, true, P_>) : go(colors_kernel<M_, false, P_>))
  if (mode == 0) {
    planes <= 8 ? SBWT_COLORS(0, 8) : planes <= 16 ? SBWT_COLORS(0, 16) : SBWT_COLORS(0, 40);
  } else {
    planes <= 8 ? SBWT_COLORS(1, 8) : planes <= 16 ? SBWT_COLORS(1, 16) : SBWT_COLORS(1, 40);
  }
#undef SBWT_COLORS
  SBWT_CUDA(cudaGetLastError());
}

void ColorsImpl::emit_ids(const u64 *d_pass_bits, const uint32_t *d_word_mask,
                          const u64 *d_ids_off, u64 n_reads, uint32_t *d_ids, u64 capacity,
                          cudaStream_t st) const {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  const u64 blocks = std::min<u64>((n_reads + 127) / 128, (u64)sms * 16);
  emit_ids_kernel<<<(unsigned)std::max<u64>(blocks, 1), 128, 0, st>>>(
      d_pass_bits, d_word_mask, view.row_words, view.tiles, d_ids_off, n_reads, d_ids, capacity);
  SBWT_CUDA(cudaGetLastError());
}

// The colors step of one device-resident batch without host synchronisation
// (capturable): per-read counting over `vals` (index-step results, -1/-2
// markers counted, not looked up) + threshold, scan of the per-read pass
// counts into d_ids_off (n_reads + 1), ids into d_ids (none when
// d_ids_off[n_reads], the required size, is more than ids_capacity).
// d_pass_count: n_reads counts, then n_reads x tiles word masks.
void ColorsImpl::enqueue_pseudoalign(const u64 *d_vals, const u64 *d_offs, u64 n_reads,
                                     u64 max_kmers, double tau, u32 flags, u64 *d_pass_bits,
                                     uint32_t *d_pass_count, u64 *d_ids_off, uint32_t *d_ids,
                                     u64 ids_capacity, uint32_t *d_err,
                                     cudaStream_t st) const {
  if (n_reads == 0) {
    SBWT_CUDA(cudaMemsetAsync(d_ids_off, 0, 8, st));
    return;
  }
  launch(d_vals, d_offs, nullptr, nullptr, n_reads, planes_for(max_kmers), tau, flags, 0,
         d_pass_bits, d_pass_count + n_reads, d_pass_count, nullptr, d_err, st);
  enqueue_scan_counts(d_pass_count, n_reads, d_ids_off, nullptr, st);
  emit_ids(d_pass_bits, d_pass_count + n_reads, d_ids_off, n_reads, d_ids, ids_capacity, st);
}

static u64 max_span(const u64 *offs, u64 n_reads) {
  u64 m = 0;
  for (u64 r = 0; r < n_reads; ++r) {
    if (offs[r + 1] < offs[r]) throw Error(SBWT_E_INVALID, "offsets must be non-decreasing");
    m = std::max(m, offs[r + 1] - offs[r]);
  }
  return m;
}

// The reads of device-resident offsets that the planes of short reads leave out,
// into ws.list (their number to *n_list); returns the longest one's k-mers.
static u64 list_long_reads(ColorsWorkspace &ws, const u64 *d_offs, u64 n_reads, cudaStream_t st,
                           u64 *n_list) {
  ws.span.ensure(24);
  ws.list.ensure(n_reads * 8);
  SBWT_CUDA(cudaMemsetAsync(ws.span.get(), 0, 24, st));
  const u64 blocks = std::min<u64>((n_reads + 255) / 256, 148 * 8);
  long_reads_kernel<<<(unsigned)std::max<u64>(blocks, 1), 256, 0, st>>>(
      d_offs, n_reads, 1ULL << kPlanes[0], ws.list.get<u64>(), ws.span.get<unsigned long long>());
  SBWT_CUDA(cudaGetLastError());
  unsigned long long h[3] = {0, 0, 0};
  SBWT_CUDA(cudaMemcpyAsync(h, ws.span.get(), 24, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  if (h[1]) throw Error(SBWT_E_INVALID, "offsets must be non-decreasing");
  *n_list = h[2];
  return h[0];
}

// Waits for the stream and reads the status words back: the error bits turn
// into exceptions, except kErrLong, which is returned.
static bool wait_status(ColorsWorkspace &ws, cudaStream_t st) {
  SBWT_CUDA(cudaMemcpyAsync(ws.status_host, ws.status.get(), 16, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  const uint32_t e = (uint32_t)*ws.status_host;
  if (!e) return false;
  SBWT_CUDA(cudaMemsetAsync(ws.status.get(), 0, 8, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  if (e & kErrOffsets) throw Error(SBWT_E_INVALID, "offsets must be non-decreasing");
  if (e & kErrNode)
    throw Error(SBWT_E_INVALID, "an SBWT index is not a key k-mer of this color index");
  return true;
}

// Device-resident batches: `run` with the planes of short reads first (the
// longest read is only known on the device), which leaves the longer ones out,
// then over those alone with the planes they need; each time the status is read
// back once.
// 2000 colors, 200 k reads of 120 k-mers and one of 300: 0.85 ms, 1.63 ms with all
// of them done again; 100 k reads of about 270: 0.97 against 1.52 ms.
template <class F>
static void run_planes(ColorsWorkspace &ws, const u64 *d_offs, u64 n_reads, cudaStream_t st,
                       F &&run) {
  run(kPlanes[0], nullptr, 0);
  if (!wait_status(ws, st)) return;
  u64 n_list = 0;
  const int planes = planes_for(list_long_reads(ws, d_offs, n_reads, st, &n_list));
  run(planes, ws.list.get<u64>(), n_list);
  wait_status(ws, st);
}

void ColorsImpl::counts(const u64 *vals, const u64 *offs, u64 n_reads, uint32_t *out,
                        u32 flags, cudaStream_t user_stream) const {
  DeviceGuard g(device);
  ColorsWorkspace &ws = colors_workspace(device);
  if (n_reads == 0) return;
  if (flags & SBWT_DEVICE_POINTERS) {
    run_planes(ws, offs, n_reads, user_stream, [&](int planes, const u64 *list, u64 n_list) {
      launch(vals, offs, nullptr, nullptr, n_reads, planes, 0.0, 0, 1, nullptr, nullptr, nullptr,
             out, ws.err(), user_stream, list, n_list);
    });
    return;
  }
  const u64 mk = max_span(offs, n_reads);
  const u64 n_vals = offs[n_reads] - offs[0];
  cudaStream_t st = ws.stream;
  ws.vals.ensure(std::max<u64>(n_vals, 1) * 8);
  ws.offs.ensure((n_reads + 1) * 8);
  ws.counts.ensure(n_reads * num_colors * 4);
  // offsets are rebased to the first value
  std::vector<u64> ro(n_reads + 1);
  for (u64 r = 0; r <= n_reads; ++r) ro[r] = offs[r] - offs[0];
  if (n_vals)
    SBWT_CUDA(cudaMemcpyAsync(ws.vals.get(), vals + offs[0], n_vals * 8,
                              cudaMemcpyHostToDevice, st));
  SBWT_CUDA(cudaMemcpyAsync(ws.offs.get(), ro.data(), (n_reads + 1) * 8,
                            cudaMemcpyHostToDevice, st));
  launch(ws.vals.get<u64>(), ws.offs.get<u64>(), nullptr, nullptr, n_reads, planes_for(mk), 0.0,
         0, 1, nullptr, nullptr, nullptr, ws.counts.get<uint32_t>(), ws.err(), st);
  SBWT_CUDA(cudaMemcpyAsync(out, ws.counts.get(), n_reads * num_colors * 4,
                            cudaMemcpyDeviceToHost, st));
  wait_status(ws, st);
}

void ColorsImpl::pseudoalign(const u64 *vals, const u64 *offs, const u64 *nf,
                             const u64 *inv, u64 n_reads, double tau, u32 flags,
                             uint32_t *ids, u64 capacity, u64 *ids_offsets,
                             cudaStream_t user_stream) const {
  DeviceGuard g(device);
  ColorsWorkspace &ws = colors_workspace(device);
  const bool dev = flags & SBWT_DEVICE_POINTERS;
  cudaStream_t st = dev ? user_stream : ws.stream;
  if (n_reads == 0) {
    if (dev) {
      SBWT_CUDA(cudaMemsetAsync(ids_offsets, 0, 8, st));
    } else {
      ids_offsets[0] = 0;
    }
    return;
  }
  ws.pass_bits.ensure(n_reads * view.row_words * 8);
  ws.pass_count.ensure(n_reads * 4 * (1 + (u64)view.tiles));
  u64 *d_bits = ws.pass_bits.get<u64>();
  uint32_t *d_count = ws.pass_count.get<uint32_t>(), *d_mask = d_count + n_reads;
  const u64 *d_nf = flags & SBWT_INCLUDE_NOT_FOUND ? nf : nullptr;
  const u64 *d_inv = flags & SBWT_INCLUDE_INVALID ? inv : nullptr;
  if (dev) {
    run_planes(ws, offs, n_reads, st, [&](int planes, const u64 *list, u64 n_list) {
      launch(vals, offs, d_nf, d_inv, n_reads, planes, tau, flags, 0, d_bits, d_mask, d_count,
             nullptr, ws.err(), st, list, n_list);
      enqueue_scan_counts(d_count, n_reads, ids_offsets, ws.total(), st);
      emit_ids(d_bits, d_mask, ids_offsets, n_reads, ids, capacity, st);
    });
    if (ws.status_host[1] > capacity) throw Error(SBWT_E_CAPACITY, "ids_capacity too small");
    return;
  }
  const u64 mk = max_span(offs, n_reads);
  const u64 n_vals = offs[n_reads] - offs[0];
  ws.vals.ensure(std::max<u64>(n_vals, 1) * 8);
  ws.offs.ensure((n_reads + 1) * 8);
  ws.ids_off.ensure((n_reads + 1) * 8);
  std::vector<u64> ro(n_reads + 1);
  for (u64 r = 0; r <= n_reads; ++r) ro[r] = offs[r] - offs[0];
  if (n_vals)
    SBWT_CUDA(cudaMemcpyAsync(ws.vals.get(), vals + offs[0], n_vals * 8,
                              cudaMemcpyHostToDevice, st));
  SBWT_CUDA(cudaMemcpyAsync(ws.offs.get(), ro.data(), (n_reads + 1) * 8,
                            cudaMemcpyHostToDevice, st));
  if (d_nf) {
    ws.nf.ensure(n_reads * 8);
    SBWT_CUDA(cudaMemcpyAsync(ws.nf.get(), nf, n_reads * 8, cudaMemcpyHostToDevice, st));
    d_nf = ws.nf.get<u64>();
  }
  if (d_inv) {
    ws.inv.ensure(n_reads * 8);
    SBWT_CUDA(cudaMemcpyAsync(ws.inv.get(), inv, n_reads * 8, cudaMemcpyHostToDevice, st));
    d_inv = ws.inv.get<u64>();
  }
  launch(ws.vals.get<u64>(), ws.offs.get<u64>(), d_nf, d_inv, n_reads, planes_for(mk), tau, flags,
         0, d_bits, d_mask, d_count, nullptr, ws.err(), st);
  enqueue_scan_counts(d_count, n_reads, ws.ids_off.get<u64>(), ws.total(), st);
  SBWT_CUDA(cudaMemcpyAsync(ids_offsets, ws.ids_off.get(), (n_reads + 1) * 8,
                            cudaMemcpyDeviceToHost, st));
  wait_status(ws, st);
  const u64 total = ws.status_host[1];
  if (total > capacity) throw Error(SBWT_E_CAPACITY, "ids_capacity too small");
  if (total == 0) return;
  ws.ids.ensure(total * 4);
  emit_ids(d_bits, d_mask, ws.ids_off.get<u64>(), n_reads, ws.ids.get<uint32_t>(), total, st);
  SBWT_CUDA(cudaMemcpyAsync(ids, ws.ids.get(), total * 4, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
}

}  // namespace sbwt
