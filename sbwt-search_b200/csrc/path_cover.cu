// Path cover of an index with a k-mer table: the k-mers of the SBWT laid out
// along its edges, so that the k-mers of a read are consecutive entries.
//
// A node's number says nothing about its successor's, so resolving a read
// k-mer by k-mer costs one random 32-byte sector per k-mer.  The cover puts
// every k-mer at one position p of an array such that p + 1 is, as often as
// the graph allows, a successor of p:
//   path_node[p]  : the node at p (u32);
//   path_entry    : its last char (2 bits), 32 positions per 16-byte entry
//                   beside their break bits (set: p does not follow p - 1)
//                   and branch bits (set: the k-mer at p - 1 has other edges).
// A read that reaches position p is then resolved by comparing its next
// chars with the cover's, 32 at a time, and its results are a run of path_node
// (search_paths_kernel).  The table maps a k-mer to node | position << 32.
//
// Nodes with the same last k - 1 chars form a suffix group and share their
// out-edges, so the k-mers of a group and the targets of its edges are a
// complete bipartite graph and min(members, edges) pairs is the best any
// cover can do there: pairing each group on its own gives a cover with the
// fewest paths.  Where a group leaves a choice (branching), the member whose
// unbranched history is shortest is paired with the target whose unbranched
// future is shortest: the shared sequence of related strains branches often,
// the variants of single strains hardly ever, so shared stays with shared
// and a read follows one path until it really leaves it.
//
// Positions are a list ranking of the pairs: every path head and one node in
// 64 (by hash) are splitters, one thread walks each splitter's stretch, the
// splitters are ranked by pointer jumping, and a second walk places the
// nodes.  Cycles are cut at their lowest splitter; cycles without a splitter
// (shorter than a few hundred k-mers) become paths of one k-mer each.
//
// L-mer filter: a blocked Bloom filter of every L-mer inside the SBWT's
// k-mers (L: see lmer_length).  An L-mer it rejects proves absent all
// k - L + 1 k-mers that hold it, so the k-mers around a read error cost two
// or three probes instead of a table lookup each.  Only the last L-mer of
// each k-mer is inserted, and all L-mers of the k-mers without a k-mer before
// them (the others' earlier L-mers are last ones of a predecessor).
#include <cuda_runtime.h>

#include <cub/cub.cuh>

#include <algorithm>

#include "index_internal.hpp"
#include "rank_blocks.cuh"

namespace sbwt {

namespace {

constexpr uint32_t NONE = ~0u;
constexpr uint32_t kLookAhead = 32;  // steps to the next branch that pairing looks at
constexpr uint32_t kMaxGroup = 8;    // nodes of a suffix group (at most 5: one per first char)

__device__ __forceinline__ bool group_bit(const uint64_t *sg, uint64_t v) {
  return (sg[v >> 6] >> (v & 63)) & 1ULL;
}

// The k-mer that group g's edge c leads to, or NONE.
__device__ __forceinline__ uint32_t edge_target(const SbwtView &s, const uint8_t *alive,
                                                uint64_t g, uint32_t c) {
  const uint64_t b = block_of(g);
  const Block B = load_block(s.blocks[c] + b);
  const uint32_t q = (uint32_t)(g - b * kBlockBits);
  if (!block_bit(B, q)) return NONE;
  const uint64_t t = s.c_map[c] + block_rank(B, q);
  return t < s.num_bits && alive[t] ? (uint32_t)t : NONE;
}

// One thread per suffix group: its k-mers (alive members) and the targets of
// its edges; every member gets the first target and its out-degree, every
// target the first member and its in-degree.
__global__ void degrees_kernel(SbwtView s, const uint8_t *alive, uint32_t *nxt, uint32_t *prv,
                               uint8_t *outd, uint8_t *ind) {
  const uint64_t n = s.num_bits, step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < n; g += step) {
    if (!group_bit(s.suffix_group_starts, g)) continue;
    uint32_t first = NONE, members = 0;
    uint64_t u = g;
    do {
      if (alive[u]) {
        if (first == NONE) first = (uint32_t)u;
        ++members;
      }
      ++u;
    } while (u < n && u < g + kMaxGroup && !group_bit(s.suffix_group_starts, u));
    if (!members) continue;
    uint32_t edges = 0, target = NONE;
    for (uint32_t c = 0; c < 4; ++c) {
      const uint32_t t = edge_target(s, alive, g, c);
      if (t == NONE) continue;
      if (target == NONE) target = t;
      prv[t] = first;
      ind[t] = (uint8_t)min(members, 255u);
      ++edges;
    }
    for (uint64_t x = g; x < u; ++x)
      if (alive[x]) {
        nxt[x] = target;
        outd[x] = (uint8_t)edges;
      }
  }
}

// Steps along unbranched edges from a target (forward) or a member (back)
// until the next branch.
__device__ __forceinline__ uint32_t ahead(const uint32_t *to, const uint8_t *deg, uint32_t x) {
  uint32_t d = 0;
  while (d < kLookAhead && deg[x] == 1) {
    x = to[x];
    ++d;
  }
  return deg[x] == 0 ? kLookAhead : d;
}

// The pairing of every group with more than one member or edge (the others'
// pair is already in pair_of, a copy of nxt).
__global__ void pair_kernel(SbwtView s, const uint8_t *alive, const uint32_t *nxt,
                            const uint32_t *prv, const uint8_t *outd, const uint8_t *ind,
                            uint32_t *pair_of) {
  const uint64_t n = s.num_bits, step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < n; g += step) {
    if (!group_bit(s.suffix_group_starts, g)) continue;
    uint32_t member[kMaxGroup], target[4], md[kMaxGroup], td[4], m = 0, t = 0;
    uint64_t u = g;
    do {
      if (alive[u]) member[m++] = (uint32_t)u;
      ++u;
    } while (u < n && u < g + kMaxGroup && !group_bit(s.suffix_group_starts, u));
    const uint32_t edges = m ? outd[member[0]] : 0;
    if (m == 0 || (m == 1 && edges <= 1)) continue;
    for (uint32_t c = 0; c < 4 && edges; ++c) {
      const uint32_t x = edge_target(s, alive, g, c);
      if (x != NONE) target[t++] = x;
    }
    for (uint32_t i = 0; i < m; ++i) md[i] = m > 1 ? ahead(prv, ind, member[i]) : 0;
    for (uint32_t i = 0; i < t; ++i) td[i] = t > 1 ? ahead(nxt, outd, target[i]) : 0;
    // the i-th nearest member gets the i-th nearest target (ties by number)
    for (uint32_t i = 0; i < m; ++i) {
      uint32_t mr = 0, to = NONE;
      for (uint32_t j = 0; j < m; ++j) mr += md[j] < md[i] || (md[j] == md[i] && j < i);
      for (uint32_t j = 0; j < t; ++j) {
        uint32_t tr = 0;
        for (uint32_t l = 0; l < t; ++l) tr += td[l] < td[j] || (td[l] == td[j] && l < j);
        if (tr == mr) to = target[j];
      }
      pair_of[member[i]] = to;
    }
  }
}

__global__ void has_prev_kernel(const uint8_t *alive, const uint32_t *pair_of, uint64_t n,
                                uint8_t *hp) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step)
    if (alive[v] && pair_of[v] != NONE) hp[pair_of[v]] = 1;
}

__global__ void splitters_kernel(const uint8_t *alive, const uint8_t *hp, uint64_t n,
                                 uint8_t *sp) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step)
    sp[v] = alive[v] && (!hp[v] || (kmer_mix(v) & 63) == 0);
}

__global__ void splitter_map_kernel(const uint32_t *list, uint32_t n, uint32_t *map) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) map[list[i]] = i;
}

// Length of each splitter's stretch and the splitter after it.
__global__ void stretch_kernel(const uint32_t *list, uint32_t n, const uint32_t *pair_of,
                               const uint8_t *sp, const uint32_t *map, uint32_t *len,
                               uint32_t *nxs, uint32_t *prs) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    uint32_t u = list[i], l = 1, to = NONE;
    while (true) {  // ends: the pairs are one-to-one, so a cycle returns to list[i]
      const uint32_t t = pair_of[u];
      if (t == NONE) break;
      if (sp[t]) {
        to = map[t];
        break;
      }
      u = t;
      ++l;
    }
    len[i] = l;
    nxs[i] = to;
    if (to != NONE) prs[to] = i;
  }
}

struct Jump {
  uint32_t ptr, off, root, low;
};

__global__ void jump_init_kernel(uint32_t n, const uint32_t *prs, const uint32_t *len, Jump *j) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    const uint32_t p = prs[i];
    j[i] = Jump{p, p == NONE ? 0u : len[p], p == NONE ? i : p, p == NONE ? i : min(i, p)};
  }
}

// One pointer-jumping round over the splitters: off = nodes before the
// splitter on its path, root = its path's head, low = the lowest splitter seen.
__global__ void jump_kernel(uint32_t n, const Jump *in, Jump *out) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    Jump a = in[i];
    if (a.ptr != NONE) {
      const Jump b = in[a.ptr];
      a.off += b.off;
      a.root = b.root;
      a.low = min(a.low, b.low);
      a.ptr = b.ptr;
    }
    out[i] = a;
  }
}

// Splitters still pointing somewhere after ceil(log2 n) rounds are on cycles:
// the lowest one of each becomes its path's head.
__global__ void cut_cycles_kernel(uint32_t n, const Jump *j, uint32_t *prs, uint32_t *cut) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
    if (j[i].ptr != NONE && j[i].low == i) {
      prs[i] = NONE;
      *cut = 1;
    }
}

// Path lengths, at the heads (the last splitter of a path knows its length).
__global__ void path_totals_kernel(uint32_t n, const uint32_t *nxs, const uint32_t *prs,
                                   const uint32_t *len, const Jump *j, uint32_t *total) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
    if (nxs[i] == NONE || prs[nxs[i]] != i) total[j[i].root] = j[i].off + len[i];
}

__global__ void place_kernel(const uint32_t *list, uint32_t n, const uint32_t *pair_of,
                             const uint32_t *len, const Jump *j, const uint32_t *base,
                             uint32_t *pos, uint32_t *path_node) {
  const uint32_t step = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    uint32_t u = list[i], p = base[j[i].root] + j[i].off;
    for (uint32_t l = 0; l < len[i]; ++l, ++p) {
      if (l) u = pair_of[u];
      pos[u] = p;
      path_node[p] = u;
    }
  }
}

// k-mers no splitter reached (short cycles): paths of one k-mer each.
__global__ void place_rest_kernel(const uint8_t *alive, uint64_t n, uint32_t *pos,
                                  uint32_t *path_node, uint32_t *next) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step)
    if (alive[v] && pos[v] == NONE) {
      const uint32_t p = atomicAdd(next, 1u);
      pos[v] = p;
      path_node[p] = (uint32_t)v;
    }
}

// Chars, break and branch bits, one thread per entry of 32 positions.
__global__ void path_chars_kernel(SbwtView s, const uint32_t *path_node, uint32_t len,
                                  const uint32_t *pair_of, const uint8_t *outd, PathEntry *out,
                                  uint64_t n_entries) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < n_entries; w += step) {
    uint64_t chars = 0;
    uint32_t brk = 0, branch = 0;
    uint32_t before = w && 32 * w <= len ? path_node[32 * w - 1] : NONE;
    for (uint32_t i = 0; i < 32; ++i) {
      const uint64_t p = 32 * w + i;
      const uint32_t v = p < len ? path_node[p] : NONE;
      if (v == NONE || before == NONE || pair_of[before] != v) brk |= 1u << i;
      if (before != NONE && outd[before] != 1) branch |= 1u << i;
      if (v != NONE) {
        uint32_t c = 0;
        while (c < 3 && v >= s.c_map[c + 1]) ++c;
        chars |= (uint64_t)c << (62 - 2 * i);
      }
      before = v;
    }
    out[w] = PathEntry{chars, brk, branch};
  }
}

__global__ void lmer_insert_kernel(const uint64_t *key, const uint8_t *alive, const uint32_t *prv,
                                   uint64_t n, uint32_t k, uint32_t L, unsigned long long *filter,
                                   uint32_t n_words) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += step) {
    if (!alive[v]) continue;
    const uint32_t more = prv[v] == NONE ? k - L : 0;
    for (uint32_t j = 0; j <= more; ++j) {
      const uint32_t z = lmer_hash((key[v] >> (2 * j)) & ((1ULL << (2 * L)) - 1));
      const uint2 b = lmer_bits(z);
      atomicOr(filter + lmer_word(z, n_words), (unsigned long long)b.y << 32 | b.x);
    }
  }
}

unsigned grid_of(uint64_t n) {
  return (unsigned)std::max<uint64_t>(std::min<uint64_t>((n + 255) / 256, 148 * 32), 1);
}

// Length of the filter's L-mers: short enough that an absent one rules out
// many k-mers, long enough that a random one is absent.  With l = ceil(log4
// k-mers): l + 2 (a random one is present at most once in 16) from k = l + 5
// on, else l + 1, or l where k is l + 1 (an L-mer of all k chars rules out one
// k-mer).  300 k random reads on 2 M nodes (l = 11), L = l / l + 1 / l + 2 / l +
// 3: k = 13 920 / 820 / 1182 / 1192 us, k = 14 753 / 554 / 636 / 1043, k = 16 527
// / 377 / 376 / 419; 1 M on 69 M nodes (l = 14), k = 15: 3.17 / 3.95 ms.
// 0, no filter: fewer than 8 possible k-mers for each of the SBWT's.  Most L-mers
// are in such a graph then, and the read search does not run over its cover.
uint32_t lmer_length(u64 n_kmers, u32 k) {
  u32 lg = 0;
  while (lg < 32 && (1ULL << (2 * lg)) < n_kmers) ++lg;
  if ((1ULL << (2 * k)) / 8 < n_kmers) return 0;
  return k >= lg + 5 ? std::max<u32>(lg + 2, 4) : std::min(lg + 1, k - 1);
}

}  // namespace

// Builds the path cover and the L-mer filter from the labels of the k-mer
// table's construction; pos[v] (u32 per node) receives each k-mer's position.
// scratch: at least 16 bytes per node.  Returns false (and builds nothing) for
// SBWTs without suffix-group words, of 64-bit nodes, or when device memory is
// short.
bool IndexImpl::build_path_cover(const u64 *key, const u8 *alive, u64 n_kmers, u32 *pos,
                                 u8 *scratch, u64 scratch_bytes) {
  const u64 n = num_bits;
  if (!view.suffix_group_starts || n >= (u64)kBlockBits << kSuperchunkShift || n_kmers == 0)
    return false;
  const u64 n_entries = n_kmers / 32 + 3;  // two entries of breaks past the end
  const u32 L = lmer_length(n_kmers, k);
  const u64 lm_words = L ? std::max<u64>((n_kmers * kLmerFilterBits + 63) / 64, 1) : 0;
  size_t free_b = 0, total_b = 0;
  SBWT_CUDA(cudaMemGetInfo(&free_b, &total_b));
  if (n_kmers * 4 + n_entries * 16 + lm_words * 8 > free_b / 2) return false;
  const unsigned gn = grid_of(n);

  // three u32 arrays and three byte arrays of n, 256-byte aligned
  const u64 a4 = (n * 4 + 255) / 256 * 256, a1 = (n + 255) / 256 * 256;
  if (3 * a4 + 3 * a1 > scratch_bytes) return false;
  u32 *const nxt = reinterpret_cast<u32 *>(scratch);
  u32 *const prv = reinterpret_cast<u32 *>(scratch + a4);
  u32 *const pair = reinterpret_cast<u32 *>(scratch + 2 * a4);
  u8 *const outd = scratch + 3 * a4, *const ind = outd + a1, *const hp = ind + a1;
  SBWT_CUDA(cudaMemsetAsync(nxt, 0xFF, 2 * a4));
  SBWT_CUDA(cudaMemsetAsync(outd, 0, 3 * a1));
  degrees_kernel<<<gn, 256>>>(view, alive, nxt, prv, outd, ind);
  SBWT_CUDA(cudaMemcpyAsync(pair, nxt, n * 4, cudaMemcpyDeviceToDevice));
  pair_kernel<<<gn, 256>>>(view, alive, nxt, prv, outd, ind, pair);
  SBWT_CUDA(cudaGetLastError());
  if (L) {
    lmer_filter.resize(lm_words * 8);
    SBWT_CUDA(cudaMemsetAsync(lmer_filter.get(), 0, lm_words * 8));
    lmer_insert_kernel<<<gn, 256>>>(key, alive, prv, n, k, L,
                                    lmer_filter.get<unsigned long long>(), (u32)lm_words);
  }
  // splitters: path heads and one k-mer in 64
  u8 *const sp = ind;  // the in-degrees are done with
  has_prev_kernel<<<gn, 256>>>(alive, pair, n, hp);
  splitters_kernel<<<gn, 256>>>(alive, hp, n, sp);
  SBWT_CUDA(cudaGetLastError());
  u32 *const list = nxt, *const map = prv;  // done with as well
  cub::CountingInputIterator<u32> ids(0);
  size_t tb = 0, tb2 = 0;
  SBWT_CUDA(cub::DeviceSelect::Flagged(nullptr, tb, ids, sp, list, list, (int64_t)n));
  SBWT_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb2, list, list, (int64_t)n));
  DeviceBuffer tmp(std::max<size_t>(std::max(tb, tb2), 1) + 256);
  u32 *const small = reinterpret_cast<u32 *>(tmp.get<u8>());  // a word before the rest
  void *const cub_tmp = tmp.get<u8>() + 256;
  SBWT_CUDA(cub::DeviceSelect::Flagged(cub_tmp, tb, ids, sp, list, small, (int64_t)n));
  u32 ns = 0;
  SBWT_CUDA(cudaMemcpy(&ns, small, 4, cudaMemcpyDeviceToHost));
  SBWT_CUDA(cudaMemsetAsync(pos, 0xFF, n * 4));
  path_nodes.resize(n_kmers * 4);
  path_entries.resize(n_entries * sizeof(PathEntry));
  u32 placed = 0;
  DeviceBuffer ranks;  // of the splitters
  if (ns) {
    const unsigned gs = grid_of(ns);
    const u64 s4 = ((ns + 1) * 4ULL + 255) / 256 * 256, sj = (ns * sizeof(Jump) + 255) / 256 * 256;
    ranks.resize(4 * s4 + 2 * sj);
    u8 *const r = ranks.get<u8>();
    u32 *const len = reinterpret_cast<u32 *>(r), *const nxs = reinterpret_cast<u32 *>(r + s4);
    u32 *const prs = reinterpret_cast<u32 *>(r + 2 * s4);
    u32 *const total = reinterpret_cast<u32 *>(r + 3 * s4);
    Jump *const jump[2] = {reinterpret_cast<Jump *>(r + 4 * s4),
                           reinterpret_cast<Jump *>(r + 4 * s4 + sj)};
    SBWT_CUDA(cudaMemsetAsync(prs, 0xFF, ns * 4ULL));
    SBWT_CUDA(cudaMemsetAsync(total, 0, (ns + 1) * 4ULL));
    splitter_map_kernel<<<gs, 256>>>(list, ns, map);
    stretch_kernel<<<gs, 256>>>(list, ns, pair, sp, map, len, nxs, prs);
    SBWT_CUDA(cudaGetLastError());
    u32 rounds = 1;
    while ((1ULL << rounds) < ns) ++rounds;
    Jump *j = nullptr;
    auto rank = [&] {
      jump_init_kernel<<<gs, 256>>>(ns, prs, len, jump[0]);
      int at = 0;
      for (u32 q = 0; q <= rounds; ++q, at ^= 1)
        jump_kernel<<<gs, 256>>>(ns, jump[at], jump[at ^ 1]);
      j = jump[at];
    };
    rank();
    u32 cut = 0;
    SBWT_CUDA(cudaMemsetAsync(small, 0, 4));
    cut_cycles_kernel<<<gs, 256>>>(ns, j, prs, small);
    SBWT_CUDA(cudaMemcpy(&cut, small, 4, cudaMemcpyDeviceToHost));
    if (cut) rank();
    path_totals_kernel<<<gs, 256>>>(ns, nxs, prs, len, j, total);
    SBWT_CUDA(cub::DeviceScan::ExclusiveSum(cub_tmp, tb2, total, total, (int64_t)ns + 1));
    SBWT_CUDA(cudaMemcpy(&placed, total + ns, 4, cudaMemcpyDeviceToHost));
    if (placed > n_kmers) throw Error(SBWT_E_FORMAT, "the SBWT's edges are not one-to-one");
    place_kernel<<<gs, 256>>>(list, ns, pair, len, j, total, pos, path_nodes.get<u32>());
    SBWT_CUDA(cudaGetLastError());
  }
  SBWT_CUDA(cudaMemcpyAsync(small, &placed, 4, cudaMemcpyHostToDevice));
  place_rest_kernel<<<gn, 256>>>(alive, n, pos, path_nodes.get<u32>(), small);
  path_chars_kernel<<<grid_of(n_entries), 256>>>(view, path_nodes.get<u32>(), (u32)n_kmers, pair,
                                                 outd, path_entries.get<PathEntry>(), n_entries);
  SBWT_CUDA(cudaGetLastError());
  view.path_node = path_nodes.get<u32>();
  view.path_entry = path_entries.get<PathEntry>();
  view.path_len = (u32)n_kmers;
  view.lmer_filter = L ? lmer_filter.get<u64>() : nullptr;
  view.lmer_words = (u32)lm_words;
  view.lmer_len = L;
  return true;
}

void IndexImpl::drop_path_cover() {
  path_nodes.release();
  path_entries.release();
  lmer_filter.release();
  view.path_node = nullptr;
  view.path_entry = nullptr;
  view.path_len = 0;
  view.lmer_filter = nullptr;
  view.lmer_words = 0;
  view.lmer_len = 0;
}

}  // namespace sbwt
