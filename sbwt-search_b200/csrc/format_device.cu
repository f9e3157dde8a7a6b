// Result formatting on the GPU: the bytes the reference's printers write,
// produced on the device so that the device->host copy carries final output.
//
// Index results (src/IndexResultsPrinter/: AsciiContinuousIndexResultsPrinter
// .cpp:50-55, BinaryContinuousIndexResultsPrinter, BoolContinuousIndexResults
// Printer): per read, ascii = decimal tokens ("-1" not found, "-2" invalid)
// separated by ' ' and ended by '\n'; binary = one u64 per k-mer then u64 -3;
// bool = '0' found / '1' not found / '2' invalid per k-mer then '\n'.
// Color results (src/ColorResultsPrinter/: AsciiContinuousColorResultsPrinter
// .cpp:74-79, Binary..., Csv...): per read, ascii = ids separated by ' ' and
// ended by '\n'; binary = one u64 per id then u64 -1; csv = one "0/1" per
// color separated by ',' and ended by '\n'.  Headers (and the csv title row)
// are written once per file by the host writers, not here.
//
// Ascii is written in tiles of kTile tokens, whatever the reads' lengths: a
// pass over the tokens sums each tile's bytes, a scan turns them into offsets,
// and one block per tile composes its bytes in shared memory and stores them
// 16 at a time.  Every token is followed by one ' ' or '\n', so the first pass
// needs nothing of the reads but the empty ones ('\n' each) of a tile.  The
// other formats have closed-form offsets.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <memory>

#include "common.hpp"

namespace sbwt {

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr uint32_t kScanThreads = 1024, kScanPer = 4, kScanSpan = kScanThreads * kScanPer;

// Decimal digits of v, v < 2^32: entry log2(v) of `table` holds, in its high
// half, the digits of 2^log2(v) plus a carry-in that adds one from the next
// power of ten on (Lemire, "Computing the number of digits of an integer even
// faster", 2021).
__device__ __forceinline__ uint32_t dec_len32(const uint64_t *table, uint32_t v) {
  return (uint32_t)((v + table[31 - __clz(v | 1)]) >> 32);
}
struct DecLenTable {
  uint64_t entry[32];
  constexpr DecLenTable() : entry() {
    for (int log2 = 0; log2 < 32; ++log2) {
      uint64_t n = 1, p = 10;  // digits of 2^log2, the first power of ten above it
      while (p <= (1ULL << log2)) {
        p *= 10;
        ++n;
      }
      entry[log2] = p < (2ULL << log2) ? ((n + 1) << 32) - p : n << 32;
    }
  }
};
__constant__ const DecLenTable kDecLen{};
__device__ uint32_t dec_len64(uint64_t v) {
  uint32_t n = 1;
  for (; v >= 10; v /= 10) ++n;
  return n;
}

// Four decimal digits of x < 10000 as ascii bytes, the first in the low byte.
__device__ __forceinline__ uint32_t dec4(uint32_t x) {
  const uint32_t q = (x * 5243u) >> 19;  // x / 100
  const uint32_t z = q | (x - 100 * q) << 16;
  const uint32_t t = ((z * 103u) >> 10) & 0x000F000Fu;  // each half / 10
  return (t | (z - 10 * t) << 8) + 0x30303030u;
}

// Tokens of the index results (u64, two markers) and of the color ids (u32).
__device__ __forceinline__ bool is_marker(uint64_t v) { return v >= SBWT_INVALID; }
__device__ __forceinline__ bool is_marker(uint32_t) { return false; }
template <class V>
__device__ __forceinline__ uint32_t token_len(const uint64_t *table, V v) {
  if (is_marker(v)) return 2;
  if (sizeof(V) == 4 || (uint64_t)v < (1ULL << 32)) return dec_len32(table, (uint32_t)v);
  return dec_len64((uint64_t)v);
}

// k-mers of read r (reads shorter than k have none), from the read ends.
__device__ __forceinline__ uint64_t kmers_of(const uint64_t *ends, uint64_t r, uint32_t k) {
  const uint64_t len = ends[r] - (r ? ends[r - 1] : 0);
  return len >= k ? len - k + 1 : 0;
}

__global__ void kmer_counts_kernel(const uint64_t *ends, uint64_t n_reads, uint32_t k,
                                   uint64_t *kmers) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n_reads; r += step)
    kmers[r] = kmers_of(ends, r, k);
}

__global__ void index_fixed_kernel(const uint64_t *res, const uint64_t *ends, uint64_t n_reads,
                                   uint32_t k, const uint64_t *kmer_off, int format,
                                   uint8_t *out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; r < n_reads;
       r += warps) {
    const uint64_t m = kmers_of(ends, r, k), t0 = kmer_off[r];
    if (format == 1) {  // binary: u64 per k-mer, then -3
      uint64_t *o = reinterpret_cast<uint64_t *>(out) + t0 + r;
      for (uint64_t j = lane; j < m; j += 32) o[j] = res[t0 + j];
      if (lane == 0) o[m] = (uint64_t)-3;
    } else {  // bool
      uint8_t *o = out + t0 + r;
      for (uint64_t j = lane; j < m; j += 32) {
        const uint64_t v = res[t0 + j];
        o[j] = v == SBWT_NOT_FOUND ? '1' : (v == SBWT_INVALID ? '2' : '0');
      }
      if (lane == 0) o[m] = '\n';
    }
  }
}

__global__ void color_binary_kernel(const uint32_t *ids, const uint64_t *ids_off,
                                    uint64_t n_reads, uint64_t *out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; r < n_reads;
       r += warps) {
    const uint64_t a = ids_off[r], b = ids_off[r + 1];
    uint64_t *o = out + a + r;
    for (uint64_t t = a + lane; t < b; t += 32) o[t - a] = ids[t];
    if (lane == 0) o[b - a] = ~0ULL;
  }
}

// csv: row r at r * 2C; '0' / ',' everywhere, then '1' at the ids.
__global__ void color_csv_kernel(const uint32_t *ids, const uint64_t *ids_off, uint64_t n_reads,
                                 uint64_t num_colors, uint8_t *out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t row = 2 * num_colors;
  for (uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; r < n_reads;
       r += warps) {
    uint8_t *o = out + r * row;
    for (uint64_t i = lane; i < row; i += 32)
      o[i] = (i & 1) ? (i + 1 == row ? '\n' : ',') : '0';
    __syncwarp();
    for (uint64_t t = ids_off[r] + lane; t < ids_off[r + 1]; t += 32) {
      const uint32_t c = ids[t];
      if (c < num_colors) o[2 * (uint64_t)c] = '1';
    }
  }
}

// Multi-block exclusive scan of u64 values in place (v[n] = total): block
// totals into tops[], one block scans tops, the last launch writes.
__device__ __forceinline__ uint64_t block_exclusive(uint64_t v, uint64_t *total) {
  __shared__ uint64_t wsum[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) wsum[wid] = x;
  __syncthreads();
  if (wid == 0) {
    uint64_t s = lane < blockDim.x / 32 ? wsum[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(FULL, s, o);
      if (lane >= (uint32_t)o) s += y;
    }
    wsum[lane] = s;
  }
  __syncthreads();
  const uint64_t ex = (wid ? wsum[wid - 1] : 0) + x - v;
  *total = wsum[blockDim.x / 32 - 1];
  __syncthreads();
  return ex;
}

__global__ void __launch_bounds__(kScanThreads) scan_tops_of_kernel(const uint64_t *v, uint64_t n,
                                                                    uint64_t *tops) {
  const uint64_t b0 = blockIdx.x * (uint64_t)kScanSpan;
  uint64_t s = 0;
  for (uint32_t q = 0; q < kScanPer; ++q) {
    const uint64_t i = b0 + q * kScanThreads + threadIdx.x;
    if (i < n) s += v[i];
  }
  uint64_t total;
  block_exclusive(s, &total);
  if (threadIdx.x == 0) tops[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) scan_tops_kernel(uint64_t *tops, uint64_t nb) {
  uint64_t carry = 0;
  for (uint64_t b = 0; b < nb; b += kScanThreads) {
    const uint64_t i = b + threadIdx.x;
    const uint64_t x = i < nb ? tops[i] : 0;
    uint64_t total;
    const uint64_t ex = block_exclusive(x, &total);
    if (i < nb) tops[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) tops[nb] = carry;
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(uint64_t *v, uint64_t n,
                                                                  const uint64_t *tops) {
  const uint64_t i0 = blockIdx.x * (uint64_t)kScanSpan + (uint64_t)threadIdx.x * kScanPer;
  uint64_t c[kScanPer], s = 0;
#pragma unroll
  for (uint32_t q = 0; q < kScanPer; ++q) {
    c[q] = i0 + q < n ? v[i0 + q] : 0;
    s += c[q];
  }
  uint64_t total;
  uint64_t at = tops[blockIdx.x] + block_exclusive(s, &total);
#pragma unroll
  for (uint32_t q = 0; q < kScanPer; ++q) {
    if (i0 + q < n) v[i0 + q] = at;
    at += c[q];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) v[n] = tops[gridDim.x];
}

// ---- ascii in tiles of tokens ------------------------------------------------
constexpr uint32_t kTileThreads = 256, kTokens = 8, kTile = kTileThreads * kTokens;
// Bytes of a tile that shared memory holds (16 per token).  A tile with more (tens
// of thousands of empty reads, or tokens of 16 and more digits) is a big one: it is
// filled with '\n' by many blocks, and its tokens go straight to their places.
constexpr uint32_t kTileBytes = 16 * kTile;

// What read r adds to a count of the empty reads in front of a token, mod 2^32: the
// last one of a stretch its end, the first one its start taken away, so that
// thousands of empty reads in a row are two additions.  before, a, b, after:
// off[r - 1] to off[r + 2], where they exist (all loaded at once).
__device__ __forceinline__ uint32_t empty_share(uint64_t r, uint64_t n_reads, uint64_t before,
                                                uint64_t a, uint64_t b, uint64_t after) {
  if (a != b) return 0;
  return (r + 1 == n_reads || after != a ? (uint32_t)r + 1 : 0u) -
         (r == 0 || before != a ? (uint32_t)r : 0u);
}

// One thread per read: first_read[t] = the first read r with off[r] - off[0]
// >= t * kTile (t <= n / kTile), the empty reads of each tile, and the bit of
// every read's last token in `ends` (both zeroed before).
// status: 0 (flags, set later), off[n_reads] - off[0], off[0], 0 (a count).  Tokens
// past max_n (< tiles * kTile) count as its last one.
__global__ void tile_lines_kernel(const uint64_t *off, uint64_t n_reads, uint64_t max_n,
                                  uint64_t *first_read, uint32_t *empty, uint32_t *ends,
                                  uint64_t *status) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x, base = off[0];
  const uint64_t n = min(off[n_reads] - base, max_n);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    status[0] = 0;
    status[1] = off[n_reads] - base;
    status[2] = base;
    status[3] = 0;
  }
  const uint32_t lane = threadIdx.x & 31;
  for (uint64_t r0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ULL; r0 <= n_reads;
       r0 += step) {
    const uint64_t r = r0 + lane;
    uint64_t a = 0;
    uint32_t share = 0;
    if (r <= n_reads) {
      const uint64_t o_before = r ? off[r - 1] : base, o = off[r];
      const uint64_t o_end = off[min(r + 1, n_reads)], o_after = off[min(r + 2, n_reads)];
      a = min(o - base, n);
      const uint64_t before = min(o_before - base, n);
      for (uint64_t t = r ? before / kTile + 1 : 0; t <= a / kTile; ++t) first_read[t] = r;
      if (r && a > before) atomicOr(ends + (a - 1) / 32, 1u << ((a - 1) & 31));
      if (r < n_reads) share = empty_share(r, n_reads, o_before, o, o_end, o_after);
    }
    const unsigned m = __ballot_sync(FULL, share != 0);
    if (!m) continue;
    const uint64_t t = a / kTile;
    // neighbours are in the same tile nearly always: one add for them
    const int lead = __ffs(m) - 1;
    const uint64_t t0 = __shfl_sync(FULL, t, lead);
    const uint32_t sum = __reduce_add_sync(FULL, t == t0 ? share : 0);
    if ((int)lane == lead && sum) atomicAdd(empty + t0, sum);
    if (t != t0 && share) atomicAdd(empty + t, share);
  }
}

// This thread's kTokens tokens of the tile from slot s0 (missing ones 0).
template <class V>
__device__ __forceinline__ void load_tokens(const V *tok, uint64_t s0, uint64_t n,
                                            V (&v)[kTokens]) {
  const uint64_t i = s0 + kTokens * threadIdx.x;
  if (i + kTokens <= n && ((uintptr_t)(tok + i) & 15) == 0) {
#pragma unroll
    for (uint32_t q = 0; q < kTokens; q += 16 / sizeof(V)) {
      if constexpr (sizeof(V) == 8) {
        const ulonglong2 a = __ldcs(reinterpret_cast<const ulonglong2 *>(tok + i + q));
        v[q] = (V)a.x;
        v[q + 1] = (V)a.y;
      } else {
        const uint4 a = __ldcs(reinterpret_cast<const uint4 *>(tok + i + q));
        v[q] = (V)a.x;
        v[q + 1] = (V)a.y;
        v[q + 2] = (V)a.z;
        v[q + 3] = (V)a.w;
      }
    }
    return;
  }
#pragma unroll
  for (uint32_t q = 0; q < kTokens; ++q) v[q] = i + q < n ? tok[i + q] : 0;
}

// bytes[t]: the tile's tokens and terminators plus its empty reads; *flags
// gets bit 0 when some tile has empty reads, and counts the big tiles from bit 1
// on; big[i]: the i-th of them, whose empty[t] becomes kBig | i (a store for every
// tile took 7 % longer).  kSumTiles tiles per block, all their loads in flight.
constexpr uint32_t kBig = 1u << 31;
constexpr uint32_t kSumTiles = 2;
constexpr uint64_t kFewTiles = 4 * kTileThreads;
template <class V>
__global__ void __launch_bounds__(kTileThreads) tile_bytes_kernel(const V *tok, uint64_t max_n,
                                                                  uint64_t tiles,
                                                                  uint32_t *empty,
                                                                  uint32_t *big,
                                                                  uint64_t *bytes,
                                                                  uint64_t *flags) {
  const uint64_t n = min(flags[1], max_n);  // tile_lines_kernel's status
  tok += flags[2];
  __shared__ uint64_t table[32];
  __shared__ uint32_t sums[kSumTiles][kTileThreads / 32];
  if (threadIdx.x < 32) table[threadIdx.x] = kDecLen.entry[threadIdx.x];
  const uint64_t t0 = blockIdx.x * (uint64_t)kSumTiles;
  V v[kSumTiles][kTokens];
#pragma unroll
  for (uint32_t i = 0; i < kSumTiles; ++i) load_tokens(tok, (t0 + i) * kTile, n, v[i]);
  __syncthreads();
#pragma unroll
  for (uint32_t i = 0; i < kSumTiles; ++i) {
    const uint64_t s0 = (t0 + i) * kTile + kTokens * threadIdx.x;
    uint32_t s = 0;
#pragma unroll
    for (uint32_t q = 0; q < kTokens; ++q)
      if (s0 + q < n) s += token_len(table, v[i][q]) + 1;
    s = __reduce_add_sync(FULL, s);
    if ((threadIdx.x & 31) == 0) sums[i][threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x < kSumTiles && t0 + threadIdx.x < tiles) {
    const uint64_t tile = t0 + threadIdx.x;
    const uint32_t e = empty[tile];
    uint64_t t = e;
    for (uint32_t w = 0; w < kTileThreads / 32; ++w) t += sums[threadIdx.x][w];
    bytes[tile] = t;
    if (e) atomicOr((unsigned long long *)flags, 1ULL);
    if (t > kTileBytes) {
      const uint32_t at = (uint32_t)(atomicAdd((unsigned long long *)flags, 2ULL) >> 1);
      big[at] = (uint32_t)tile;
      empty[tile] = kBig | at;
    }
  }
  if (tiles > kFewTiles) return;
  // few tiles: the last block to get here turns the bytes into offsets
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicAdd((unsigned long long *)flags + 3, 1ULL) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint64_t carry = 0;
  for (uint64_t i0 = 0; i0 < tiles; i0 += kTileThreads) {
    const uint64_t i = i0 + threadIdx.x;
    uint64_t total;
    const uint64_t ex = block_exclusive(i < tiles ? __ldcg(bytes + i) : 0, &total);
    if (i < tiles) bytes[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) bytes[tiles] = carry;
}

// ORs the bytes of w into the zeroed bytes at o.
__device__ __forceinline__ void put_bytes(uint32_t *buf, uint32_t o, uint64_t w) {
  const uint32_t g = 8 * (o & 3), lo = (uint32_t)w, hi = (uint32_t)(w >> 32);
  atomicOr(buf + (o >> 2), lo << g);
  const uint32_t u1 = __funnelshift_l(lo, hi, g), u2 = __funnelshift_l(hi, 0, g);
  if (u1) atomicOr(buf + (o >> 2) + 1, u1);
  if (u2) atomicOr(buf + (o >> 2) + 2, u2);
}

// The stretches of more than kFewLines '\n' (e from o on, in the zeroed buf) of a
// warp's threads, by the whole warp: whole words by plain stores, as no other
// token or line reaches into them.  (Kept out of write_tile's token loop, which
// it made 7 % longer for tiles with short stretches alone.)
constexpr uint32_t kFewLines = 64;
__device__ __forceinline__ void put_newlines(uint32_t *buf, uint32_t o, uint32_t e) {
  constexpr uint32_t kLines = 0x0A0A0A0Au;
  const uint32_t lane = threadIdx.x & 31;
  for (unsigned m = __ballot_sync(FULL, e > kFewLines); m; m &= m - 1) {
    const uint32_t a = __shfl_sync(FULL, o, __ffs(m) - 1);
    const uint32_t b = a + __shfl_sync(FULL, e, __ffs(m) - 1);
    for (uint32_t w = (a + 3) / 4 + lane; w < b / 4; w += 32) buf[w] = kLines;
    if (lane == 0 && (a & 3)) atomicOr(buf + a / 4, kLines << (8 * (a & 3)));
    if (lane == 1 && (b & 3)) atomicOr(buf + b / 4, kLines >> (8 * (4 - (b & 3))));
  }
}

// f(off[r], off[r + 1]) of all reads by the whole block, four reads' loads in
// flight per thread.
template <class F>
__device__ __forceinline__ void each_read(const uint64_t *off, uint64_t n_reads, F f) {
  constexpr uint32_t U = 4;
  for (uint64_t r = threadIdx.x; r < n_reads; r += U * kTileThreads) {
    uint64_t a[U], b[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint64_t x = min(r + u * kTileThreads, n_reads - 1);
      a[u] = __ldg(off + x);
      b[u] = __ldg(off + x + 1);
    }
#pragma unroll
    for (uint32_t u = 0; u < U; ++u)
      if (r + u * kTileThreads < n_reads) f(a[u], b[u]);
  }
}

// extra[i] = the empty reads before the token of slot i of the tile.  Slot n (in
// the last tile) stands for the end: it has no token, only the empty reads
// after the last one.  By the whole block; the caller waits for the counts.
__device__ __forceinline__ void count_extras(const uint64_t *off, uint64_t n_reads, uint64_t n,
                                             const uint64_t *first_read, uint64_t tile,
                                             uint32_t *extra) {
  const uint64_t base = off[0], s0 = tile * kTile;
  for (uint32_t i = threadIdx.x; i < kTile; i += kTileThreads) extra[i] = 0;
  __syncthreads();
  const uint64_t r_hi = s0 + kTile <= n ? first_read[tile + 1] : n_reads;
  for (uint64_t r = first_read[tile] + threadIdx.x; r < r_hi; r += kTileThreads) {
    const uint64_t a = off[r] - base;
    if (off[r + 1] - base == a && a - s0 < kTile) atomicAdd(&extra[a - s0], 1u);
  }
}

struct TileShared {
  uint64_t table[32];
  __align__(16) uint32_t buf[kTileBytes / 4 + 8];
  uint32_t sums[kTileThreads / 32];
};

// One block writes a tile of `bytes` <= kTileBytes bytes at dst.  A thread
// turns its tokens into bytes, eight digits at a time, and ORs them into shared
// memory at their offsets (a scan of the lengths); the block then stores the
// bytes 16 at a time, laid out as the output's own 16-byte lines.  left: tokens
// from the tile's first on; bits: which of this thread's tokens end a read;
// extra: see count_extras (EXTRAS: there are any).
template <class V, bool EXTRAS>
__device__ __forceinline__ void write_tile(TileShared &sh, const V (&v)[kTokens], uint32_t left,
                                           uint32_t bits, const uint32_t *extra, uint32_t bytes,
                                           uint8_t *dst) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t *const buf = sh.buf;
  const uint32_t shift = (uint32_t)((uintptr_t)dst & 15);  // the place in a 16-byte line
  const uint32_t stop = shift + bytes;
  for (uint32_t i = tid; 16 * i < stop; i += kTileThreads)
    reinterpret_cast<uint4 *>(buf)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  uint32_t len[kTokens], mine = 0, most = 0;
#pragma unroll
  for (uint32_t q = 0; q < kTokens; ++q) {
    len[q] = kTokens * tid + q < left ? token_len(sh.table, v[q]) + 1 : 0;
    mine += len[q];
    if (EXTRAS) {
      mine += extra[kTokens * tid + q];
      most = max(most, extra[kTokens * tid + q]);
    }
  }
  const bool many = EXTRAS && __any_sync(FULL, most > kFewLines);
  uint32_t x = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) sh.sums[wid] = x;
  __syncthreads();
  uint32_t o = shift + x - mine;
#pragma unroll
  for (uint32_t w = 0; w < kTileThreads / 32; ++w) o += w < wid ? sh.sums[w] : 0;
  if (EXTRAS && many) {
    uint32_t at = o;
#pragma unroll
    for (uint32_t q = 0; q < kTokens; ++q) {
      const uint32_t e = extra[kTokens * tid + q];
      put_newlines(buf, at, e);
      at += e + len[q];
    }
  }
  const uint32_t alone = many ? kFewLines : ~0u;
#pragma unroll
  for (uint32_t q = 0; q < kTokens; ++q) {
    if (EXTRAS) {
      uint32_t e = extra[kTokens * tid + q];
      if (e > alone) {
        o += e;
        e = 0;
      }
      for (; e; --e, ++o) atomicOr(buf + (o >> 2), (uint32_t)'\n' << (8 * (o & 3)));
    }
    if (!len[q]) continue;
    const uint32_t term = (bits >> q) & 1u ? '\n' : ' ', end = o + len[q];
    if (is_marker(v[q])) {
      put_bytes(buf, o, '-' | ((uint64_t)v[q] == SBWT_NOT_FOUND ? '1' : '2') << 8 | term << 16);
    } else {
      uint32_t m = len[q] - 1, b = (uint32_t)v[q];
      if (m > 8) {  // the digits before the last eight
        if (sizeof(V) == 4 || (uint64_t)v[q] < (1ULL << 32)) {  // one or two
          const uint32_t a = b / 100000000u, t = (a * 103u) >> 10;
          b -= a * 100000000u;
          const uint32_t two = (t | (a - 10 * t) << 8) + 0x3030u;
          put_bytes(buf, o, m == 9 ? two >> 8 : two);
        } else {
          uint64_t a = (uint64_t)v[q] / 100000000u;
          b = (uint32_t)((uint64_t)v[q] - a * 100000000u);
#pragma unroll 1
          for (uint32_t i = m - 8; i-- > 0; a /= 10)
            put_bytes(buf, o + i, '0' + (uint32_t)(a % 10));
        }
        m = 8;
      }
      const uint32_t c = b / 10000u, skip = 8 * (8 - m);
      const uint64_t d = (uint64_t)dec4(b - 10000u * c) << 32 | dec4(c);
      // the last m digits and, where it fits, the terminator
      uint64_t w = d >> skip;
      if (skip)
        w |= (uint64_t)term << (64 - skip);
      else
        atomicOr(buf + ((end - 1) >> 2), term << (8 * ((end - 1) & 3)));
      put_bytes(buf, end - 1 - m, w);
    }
    o = end;
  }
  __syncthreads();
  uint8_t *const line = dst - shift;
  for (uint32_t i = tid; 16 * i < stop; i += kTileThreads) {
    if (16 * i >= shift && 16 * i + 16 <= stop) {
      __stcs(reinterpret_cast<uint4 *>(line) + i, reinterpret_cast<const uint4 *>(buf)[i]);
    } else {  // the tile's first and last line
      const uint8_t *const from = reinterpret_cast<const uint8_t *>(buf);
      for (uint32_t p = max(16 * i, shift); p < min(16 * i + 16, stop); ++p) line[p] = from[p];
    }
  }
}

// One block per tile.  status: if set, the count and the tokens' place are
// read from there (tile_lines_kernel's), and nothing is written when the
// count is above n or the total above out_cap.
// What bounds it: instructions (about half for the digits and their places, a
// tenth for the stores) and the waits of a block's few steps, beside 17 bytes
// of DRAM traffic a token.  139 M tokens: 0.94 ms; one warp per read with byte
// stores took 1.94 ms, and its lengths pass 0.72 ms against 0.19 ms of
// tile_bytes_kernel.  4 tokens per thread: 0.99 ms; persistent blocks that
// load the next tile ahead: 1.16 ms (spills).  EXTRAS costs 0.09 ms, so it is
// left out of batches without an empty read.
template <class V, bool EXTRAS>
__global__ void __launch_bounds__(kTileThreads, 5)
    tile_ascii_kernel(const V *tok, uint64_t n, const uint64_t *off, uint64_t n_reads,
                      const uint64_t *first_read, const uint32_t *ends,
                      const uint64_t *tile_off, uint8_t *out, const uint64_t *status,
                      uint64_t out_cap) {
  __shared__ TileShared sh;
  __shared__ uint32_t extra[EXTRAS ? kTile : 1];
  if (status) {
    if (status[1] > n || tile_off[gridDim.x] > out_cap) return;
    n = status[1];
    tok += status[2];
  }
  const uint64_t s0 = blockIdx.x * (uint64_t)kTile;
  V v[kTokens];
  load_tokens(tok, s0, n, v);
  const uint64_t i0 = s0 + kTokens * threadIdx.x;
  const uint32_t bits = i0 < n ? __ldg(ends + i0 / 32) >> (i0 & 31) : 0;
  const uint64_t b0 = __ldg(tile_off + blockIdx.x), b1 = __ldg(tile_off + blockIdx.x + 1);
  if (b1 == b0 || b1 - b0 > kTileBytes) return;  // past the end; a big tile
  if (threadIdx.x < 32) sh.table[threadIdx.x] = kDecLen.entry[threadIdx.x];
  if (EXTRAS) count_extras(off, n_reads, n, first_read, blockIdx.x, extra);
  write_tile<V, EXTRAS>(sh, v, (uint32_t)min(n - s0, (uint64_t)kTile), bits, extra,
                        (uint32_t)(b1 - b0), out + b0);
}

// A small output in one launch and one block: the total, then, if it fits, the
// tiles one after the other.  result: the total, 1 when the block did its work
// (not when a tile is big or the tokens are more than the block takes), and the
// number of tokens.
// More reads than kSmallReads, or fewer for each of several tiles, are faster by
// many blocks, as this one looks at all of them for every tile.
constexpr uint64_t kSmallBytes = kTileBytes * 3 / 2;
constexpr uint64_t kSmallReads = 32768;
template <class V>
__global__ void __launch_bounds__(kTileThreads)
    small_ascii_kernel(const V *tok, const uint64_t *off, uint64_t n_reads, uint8_t *out,
                       uint64_t out_cap, uint64_t *result) {
  __shared__ TileShared sh;
  __shared__ uint32_t extra[kTile], ends[kTile / 32];
  const uint32_t tid = threadIdx.x;
  const uint64_t base = off[0], n = off[n_reads] - base;
  tok += base;
  if (tid < 32) sh.table[tid] = kDecLen.entry[tid];
  if (tid == 0) {
    result[1] = 0;
    result[2] = n;
  }
  if (n > kSmallBytes / 2 || (n / kTile + 1) * n_reads > kSmallReads) return;
  __syncthreads();
  uint32_t mine = 0;  // a total of at most 21 kSmallBytes
  for (uint64_t i = tid; i < n; i += kTileThreads) mine += token_len(sh.table, tok[i]) + 1;
  each_read(off, n_reads, [&](uint64_t a, uint64_t b) { mine += a == b; });
  uint64_t total;
  block_exclusive(mine, &total);
  if (tid == 0) {
    result[0] = total;
    result[1] = 1;
  }
  if (total > out_cap) return;
  for (uint64_t s0 = 0, at = 0; s0 <= n; s0 += kTile) {
    __syncthreads();
    for (uint32_t i = tid; i < kTile; i += kTileThreads) extra[i] = 0;
    if (tid < kTile / 32) ends[tid] = 0;
    V v[kTokens];
    load_tokens(tok, s0, n, v);
    __syncthreads();
    each_read(off, n_reads, [&](uint64_t a, uint64_t b) {
      a -= base;
      b -= base;
      if (a == b && a - s0 < kTile) atomicAdd(&extra[a - s0], 1u);
      if (a < b && b - 1 - s0 < kTile) atomicOr(&ends[(b - 1 - s0) / 32], 1u << ((b - 1) & 31));
    });
    __syncthreads();
    mine = 0;
#pragma unroll
    for (uint32_t q = 0; q < kTokens; ++q) {
      const uint32_t sl = kTokens * tid + q;
      mine += extra[sl] + (s0 + sl < n ? token_len(sh.table, v[q]) + 1 : 0);
    }
    uint64_t bytes;
    block_exclusive(mine, &bytes);
    if (bytes > kTileBytes) {  // the same for every thread
      if (tid == 0) result[1] = 0;
      return;
    }
    write_tile<V, true>(sh, v, (uint32_t)min(n - s0, (uint64_t)kTile),
                        ends[kTokens * tid / 32] >> (kTokens * tid % 32), extra, (uint32_t)bytes,
                        out + at);
    at += bytes;
  }
}

// ---- big tiles: any number of empty reads, tokens of any length ---------------
// extra[i * kTile + s]: the empty reads before slot s of big tile i (zeroed by
// big_fill_kernel).  One thread per read; empty: tile_bytes_kernel's.
__global__ void big_empties_kernel(const uint64_t *off, uint64_t n_reads, const uint32_t *empty,
                                   uint32_t *extra) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x, base = off[0];
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n_reads; r += step) {
    const uint64_t o = off[r], a = o - base;
    const uint32_t share = empty_share(r, n_reads, r ? off[r - 1] : o, o, off[r + 1],
                                       off[min(r + 2, n_reads)]);
    const uint32_t i = share ? __ldg(empty + a / kTile) : 0;
    if (i & kBig) atomicAdd(extra + (uint64_t)(i & ~kBig) * kTile + a % kTile, share);
  }
}

// '\n' into all bytes of the big tiles, 0 into extra.
__global__ void big_fill_kernel(const uint32_t *big, uint64_t n_big, const uint64_t *tile_off,
                                uint8_t *out, uint32_t *extra) {
  for (uint64_t i = blockIdx.y; i < n_big; i += gridDim.y) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < kTile; s += gridDim.x * blockDim.x)
      extra[i * kTile + s] = 0;
    uint8_t *const dst = out + tile_off[big[i]];
    const uint64_t shift = (uintptr_t)dst & 15;
    const uint64_t stop = shift + (tile_off[big[i] + 1] - tile_off[big[i]]);
    uint8_t *const line = dst - shift;
    const uint64_t step = 16ULL * gridDim.x * blockDim.x;
    for (uint64_t p = 16 * (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x); p < stop; p += step) {
      if (p >= shift && p + 16 <= stop) {
        *reinterpret_cast<uint4 *>(line + p) =
            make_uint4(0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au, 0x0A0A0A0Au);
      } else {
        for (uint64_t b = max(p, shift); b < min(p + 16, stop); ++b) line[b] = '\n';
      }
    }
  }
}

// One block per big tile: every token straight to its place.  extra: nullptr
// without empty reads.
template <class V>
__global__ void __launch_bounds__(kTileThreads)
    big_tokens_kernel(const V *tok, uint64_t n, const uint32_t *big, uint64_t n_big,
                      const uint32_t *extra, const uint32_t *ends, const uint64_t *tile_off,
                      uint8_t *out) {
  __shared__ uint64_t table[32], starts[kTile];
  const uint32_t tid = threadIdx.x;
  if (tid < 32) table[tid] = kDecLen.entry[tid];
  for (uint64_t i = blockIdx.x; i < n_big; i += gridDim.x) {
    const uint64_t s0 = big[i] * (uint64_t)kTile;
    const uint32_t left = (uint32_t)min(n - s0, (uint64_t)kTile);
    V v[kTokens];
    load_tokens(tok, s0, n, v);
    __syncthreads();
    uint64_t mine = 0, total;
    uint32_t len[kTokens], before[kTokens];
#pragma unroll
    for (uint32_t q = 0; q < kTokens; ++q) {
      const uint32_t sl = kTokens * tid + q;
      len[q] = sl < left ? token_len(table, v[q]) + 1 : 0;
      before[q] = extra ? __ldg(extra + i * kTile + sl) : 0;
      mine += before[q] + len[q];
    }
    uint64_t at = block_exclusive(mine, &total);
#pragma unroll
    for (uint32_t q = 0; q < kTokens; ++q) {
      starts[kTokens * tid + q] = at + before[q];
      at += before[q] + len[q];
    }
    __syncthreads();
    uint8_t *const dst = out + tile_off[big[i]];
    for (uint32_t sl = tid; sl < left; sl += kTileThreads) {  // neighbours by neighbours
      const V x = tok[s0 + sl];
      uint8_t *const p = dst + starts[sl];
      const uint32_t m = token_len(table, x);
      if (is_marker(x)) {
        p[0] = '-';
        p[1] = (uint64_t)x == SBWT_NOT_FOUND ? '1' : '2';
      } else {
        uint64_t y = (uint64_t)x;
        uint32_t d = m;
        for (; y >> 32; y /= 100000000u) {  // eight digits at a time
          uint32_t z = (uint32_t)(y % 100000000u);
          for (uint32_t e = 0; e < 8; ++e, z /= 10) p[--d] = (uint8_t)('0' + z % 10);
        }
        for (uint32_t z = (uint32_t)y; d; z /= 10) p[--d] = (uint8_t)('0' + z % 10);
      }
      p[m] = (ends[(s0 + sl) / 32] >> (sl & 31)) & 1u ? '\n' : ' ';
    }
    __syncthreads();
  }
}

// The same for n <= kScanSpan values, in one block.
__global__ void __launch_bounds__(kScanThreads) scan_one_kernel(uint64_t *v, uint64_t n) {
  const uint64_t i0 = (uint64_t)threadIdx.x * kScanPer;
  uint64_t c[kScanPer], s = 0;
#pragma unroll
  for (uint32_t q = 0; q < kScanPer; ++q) {
    c[q] = i0 + q < n ? v[i0 + q] : 0;
    s += c[q];
  }
  uint64_t total;
  uint64_t at = block_exclusive(s, &total);
#pragma unroll
  for (uint32_t q = 0; q < kScanPer; ++q) {
    if (i0 + q < n) v[i0 + q] = at;
    at += c[q];
  }
  if (threadIdx.x == 0) v[n] = total;
}

struct FormatWorkspace {
  DeviceBuffer kmer_off, tile_read, tile_bytes, line_bits, extra, tops, in_a, in_b, out;
  cudaStream_t stream = nullptr;
  u64 *host = nullptr;  // pinned: up to four counts
  ~FormatWorkspace() {
    if (stream) cudaStreamDestroy(stream);
    if (host) cudaFreeHost(host);
  }
};

FormatWorkspace &format_workspace(int device) {
  thread_local std::unique_ptr<FormatWorkspace> ws[16];
  if (device < 0 || device >= 16) throw Error(SBWT_E_INVALID, "device id out of range");
  auto &p = ws[device];
  if (!p) {
    p = std::make_unique<FormatWorkspace>();
    SBWT_CUDA(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    SBWT_CUDA(cudaMallocHost(&p->host, 32));
  }
  return *p;
}

// v[0..n) (n + 1 entries) -> exclusive offsets, v[n] = total.
void enqueue_scan(uint64_t *v, u64 n, FormatWorkspace &ws, cudaStream_t st) {
  if (n <= kScanSpan) {
    scan_one_kernel<<<1, kScanThreads, 0, st>>>(v, n);
  } else {
    const u64 nb = (n + kScanSpan - 1) / kScanSpan;
    ws.tops.ensure((nb + 1) * 8);
    uint64_t *tops = ws.tops.get<uint64_t>();
    scan_tops_of_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(v, n, tops);
    scan_tops_kernel<<<1, kScanThreads, 0, st>>>(tops, nb);
    scan_apply_kernel<<<(unsigned)nb, kScanThreads, 0, st>>>(v, n, tops);
  }
  SBWT_CUDA(cudaGetLastError());
}

// enqueue_scan, returning the total; the first `back` (1 to 4) entries from
// v[n] on come to ws.host.
u64 scan_inplace(uint64_t *v, u64 n, FormatWorkspace &ws, cudaStream_t st, int back = 1,
                 bool scanned = false) {
  if (!scanned) enqueue_scan(v, n, ws, st);
  SBWT_CUDA(cudaMemcpyAsync(ws.host, v + n, 8 * back, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  return ws.host[0];
}

unsigned warp_grid(u64 items) {
  return (unsigned)std::min<u64>(std::max<u64>((items + 7) / 8, 1), 148 * 64);
}

// The whole of format_tokens in one launch for a small output: false when that
// did not do (what it wrote is then written again); the number of tokens is in
// ws.host[2] either way.
// 100 reads of 2 color ids: 34 us a call against 47 us with a launch per step.
template <class V>
bool format_small(const V *tok, const uint64_t *off, u64 n_reads, uint8_t *out, u64 out_cap,
                  u64 *need, FormatWorkspace &ws, cudaStream_t st) {
  ws.tile_bytes.ensure(24);
  uint64_t *result = ws.tile_bytes.get<uint64_t>();
  small_ascii_kernel<V><<<1, kTileThreads, 0, st>>>(tok, off, n_reads, out, out_cap, result);
  SBWT_CUDA(cudaGetLastError());
  SBWT_CUDA(cudaMemcpyAsync(ws.host, result, 24, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  if (!ws.host[1]) return false;
  *need = ws.host[0];
  if (*need > out_cap) throw Error(SBWT_E_CAPACITY, "output capacity too small");
  return true;
}

// The big tiles, big[0, n_big), of format_tokens.  1 M reads without a token: 76
// us a call; 970 us with one block for all of a tile, 166 us with a warp per read
// and no tiles.
template <class V>
void format_big(const V *tok, u64 n, const uint64_t *off, u64 n_reads, bool empties,
                const uint32_t *big, u64 n_big, const uint32_t *empty, const uint32_t *ends,
                const uint64_t *tile_off, uint8_t *out, FormatWorkspace &ws, cudaStream_t st) {
  uint32_t *extra = nullptr;
  if (empties) {
    ws.extra.ensure(n_big * kTile * 4);
    extra = ws.extra.get<uint32_t>();
    big_fill_kernel<<<dim3(32, (unsigned)std::min<u64>(n_big, 148 * 4)), 256, 0, st>>>(
        big, n_big, tile_off, out, extra);
    big_empties_kernel<<<(unsigned)std::min<u64>(n_reads / 256 + 1, 148 * 16), 256, 0, st>>>(
        off, n_reads, empty, extra);
  }
  big_tokens_kernel<V><<<(unsigned)std::min<u64>(n_big, 148 * 16), kTileThreads, 0, st>>>(
      tok, n, big, n_big, extra, ends, tile_off, out);
  SBWT_CUDA(cudaGetLastError());
}

// The tokens tok[off[0], off[n_reads]) in lines (reads) of off as ascii, at
// most max_n of them; returns the bytes (*need set before the capacity is
// checked).  The count itself is read on the device, so the host waits once
// before the bytes are written, for the count, the total and the flags.
template <class V>
u64 format_tokens(const V *tok, u64 max_n, const uint64_t *off, u64 n_reads, uint8_t *out,
                  u64 out_cap, u64 *need, FormatWorkspace &ws, cudaStream_t st) {
  u64 tiles = max_n / kTile + 1;
  const u64 words = tiles * (kTile / 32);
  ws.tile_read.ensure(tiles * 12);           // first reads, big tiles
  ws.tile_bytes.ensure((tiles + 5) * 8);     // offsets, total, status
  ws.line_bits.ensure((tiles + words) * 4);  // empty reads of the tiles, end bits
  uint64_t *first = ws.tile_read.get<uint64_t>(), *bytes = ws.tile_bytes.get<uint64_t>();
  uint32_t *empty = ws.line_bits.get<uint32_t>(), *ends = empty + tiles;
  uint32_t *big = reinterpret_cast<uint32_t *>(first + tiles);
  SBWT_CUDA(cudaMemsetAsync(empty, 0, (tiles + words) * 4, st));
  tile_lines_kernel<<<(unsigned)std::min<u64>(n_reads / 256 + 1, 148 * 16), 256, 0, st>>>(
      off, n_reads, max_n, first, empty, ends, bytes + tiles + 1);
  tile_bytes_kernel<V><<<(unsigned)((tiles + kSumTiles - 1) / kSumTiles), kTileThreads, 0, st>>>(
      tok, max_n, tiles, empty, big, bytes, bytes + tiles + 1);
  const uint64_t *const status = bytes + tiles + 1;
  const bool few = tiles <= kFewTiles;  // written before the host knows the count
  if (few)
    tile_ascii_kernel<V, true><<<(unsigned)tiles, kTileThreads, 0, st>>>(
        tok, max_n, off, n_reads, first, ends, bytes, out, status, out_cap);
  const u64 total = scan_inplace(bytes, tiles, ws, st, 4, few);
  const u64 flags = ws.host[1], n = ws.host[2], base = ws.host[3];
  if (n > max_n) return format_tokens(tok, n, off, n_reads, out, out_cap, need, ws, st);
  if (need) *need = total;
  if (total > out_cap) throw Error(SBWT_E_CAPACITY, "output capacity too small");
  tok += base;
  tiles = n / kTile + 1;
  if (!few) {
    auto *const kernel = flags & 1 ? tile_ascii_kernel<V, true> : tile_ascii_kernel<V, false>;
    kernel<<<(unsigned)tiles, kTileThreads, 0, st>>>(tok, n, off, n_reads, first, ends, bytes,
                                                     out, nullptr, 0);
  }
  SBWT_CUDA(cudaGetLastError());
  if (flags >> 1)
    format_big(tok, n, off, n_reads, flags & 1, big, flags >> 1, empty, ends, bytes, out, ws, st);
  return total;
}

// The ascii of the tokens tok[off[0], off[n_reads]).  Their count is only known
// on the device: a small capacity is one launch, a medium one bounds the count
// (two bytes a token) for the tiles, and from `most` on the count is read back
// first (a wait of ~10 us, against tiles and end bits for many times the tokens).
// A few reads may well fill little of their room, so there `most` is smaller,
// and the launch for small outputs brings the count back (100 reads of 2 color
// ids into 16 / 64 MB: 75 / 87 us by the bound, 41 us so).
template <class V>
u64 format_ascii(const V *tok, const uint64_t *off, u64 n_reads, uint8_t *out, u64 out_cap,
                 u64 *need, FormatWorkspace &ws, cudaStream_t st) {
  u64 total = 0, max_n = out_cap / 2;
  const bool few = n_reads <= kSmallReads;
  const u64 most = few ? 4ULL << 20 : 64ULL << 20;
  const bool bound = out_cap > 0 && out_cap <= most;
  if (few && (!bound || out_cap <= kSmallBytes)) {
    if (format_small(tok, off, n_reads, out, out_cap, need ? need : &total, ws, st))
      return ws.host[0];
    max_n = ws.host[2];
  } else if (!bound) {
    SBWT_CUDA(cudaMemcpyAsync(ws.host, off, 8, cudaMemcpyDeviceToHost, st));
    SBWT_CUDA(cudaMemcpyAsync(ws.host + 1, off + n_reads, 8, cudaMemcpyDeviceToHost, st));
    SBWT_CUDA(cudaStreamSynchronize(st));
    max_n = ws.host[1] - ws.host[0];
  }
  return format_tokens(tok, max_n, off, n_reads, out, out_cap, need, ws, st);
}

// Device-resident index results -> formatted bytes (returns the byte count;
// SBWT_E_CAPACITY with *need set when out_cap is too small).
u64 format_index_device(const uint64_t *res, const uint64_t *ends, u64 n_reads, uint32_t k,
                        int format, uint8_t *out, u64 out_cap, u64 *need, FormatWorkspace &ws,
                        cudaStream_t st) {
  if (n_reads == 0) return 0;
  ws.kmer_off.ensure((n_reads + 1) * 8);
  uint64_t *koff = ws.kmer_off.get<uint64_t>();
  kmer_counts_kernel<<<(unsigned)std::min<u64>((n_reads + 255) / 256, 148 * 16), 256, 0, st>>>(
      ends, n_reads, k, koff);
  if (format == 0) {
    enqueue_scan(koff, n_reads, ws, st);
    return format_ascii(res, koff, n_reads, out, out_cap, need, ws, st);
  }
  const u64 n_kmers = scan_inplace(koff, n_reads, ws, st);
  const u64 bytes = format == 1 ? 8 * (n_kmers + n_reads) : n_kmers + n_reads;
  if (need) *need = bytes;
  if (bytes > out_cap) throw Error(SBWT_E_CAPACITY, "output capacity too small");
  index_fixed_kernel<<<warp_grid(n_reads), 256, 0, st>>>(res, ends, n_reads, k, koff, format,
                                                          out);
  SBWT_CUDA(cudaGetLastError());
  return bytes;
}

u64 format_colors_device(const uint32_t *ids, const uint64_t *ids_off, u64 n_reads,
                         u64 num_colors, int format, uint8_t *out, u64 out_cap, u64 *need,
                         FormatWorkspace &ws, cudaStream_t st) {
  if (n_reads == 0) return 0;
  u64 bytes = 0;
  if (format == 0) {
    bytes = format_ascii(ids, ids_off, n_reads, out, out_cap, need, ws, st);
  } else if (format == 1) {
    u64 n_ids = 0;
    SBWT_CUDA(cudaMemcpyAsync(&n_ids, ids_off + n_reads, 8, cudaMemcpyDeviceToHost, st));
    u64 first = 0;
    SBWT_CUDA(cudaMemcpyAsync(&first, ids_off, 8, cudaMemcpyDeviceToHost, st));
    SBWT_CUDA(cudaStreamSynchronize(st));
    if (first != 0) throw Error(SBWT_E_INVALID, "ids offsets must start at 0");
    bytes = 8 * (n_ids + n_reads);
    if (need) *need = bytes;
    if (bytes > out_cap) throw Error(SBWT_E_CAPACITY, "output capacity too small");
    color_binary_kernel<<<warp_grid(n_reads), 256, 0, st>>>(ids, ids_off, n_reads,
                                                             reinterpret_cast<uint64_t *>(out));
  } else {
    bytes = n_reads * 2 * num_colors;
    if (need) *need = bytes;
    if (bytes > out_cap) throw Error(SBWT_E_CAPACITY, "output capacity too small");
    color_csv_kernel<<<warp_grid(n_reads), 256, 0, st>>>(ids, ids_off, n_reads, num_colors, out);
  }
  SBWT_CUDA(cudaGetLastError());
  return bytes;
}

}  // namespace

}  // namespace sbwt

using namespace sbwt;

extern "C" int sbwt_format_index_results(const uint64_t *results, const uint64_t *read_ends,
                                         uint64_t n_reads, uint32_t k, int format, char *out,
                                         uint64_t out_capacity, uint64_t *out_bytes,
                                         uint32_t flags, int device, void *stream) {
  if (!out_bytes || (n_reads && !read_ends) || format < 0 || format > 2 || k == 0) {
    set_last_error("invalid argument");
    return SBWT_E_INVALID;
  }
  *out_bytes = 0;
  return guarded([&] {
    DeviceGuard g(device);
    FormatWorkspace &ws = format_workspace(device);
    const bool dev = flags & SBWT_DEVICE_POINTERS;
    cudaStream_t st = dev && stream ? (cudaStream_t)stream : ws.stream;
    if (dev) {
      if (format == 1 && ((uintptr_t)out & 7))
        throw Error(SBWT_E_INVALID, "binary output must be 8-byte aligned");
      *out_bytes = format_index_device(results, read_ends, n_reads, k, format, (uint8_t *)out,
                                       out_capacity, out_bytes, ws, st);
      SBWT_CUDA(cudaStreamSynchronize(st));
      return;
    }
    if (n_reads == 0) return;
    // host buffers: the k-mer count comes from the read ends
    u64 n_kmers = 0, prev = 0;
    for (u64 r = 0; r < n_reads; ++r) {
      if (read_ends[r] < prev) throw Error(SBWT_E_INVALID, "read ends must not decrease");
      const u64 len = read_ends[r] - prev;
      prev = read_ends[r];
      n_kmers += len >= k ? len - k + 1 : 0;
    }
    if (n_kmers && !results) throw Error(SBWT_E_INVALID, "null results");
    ws.in_a.ensure(std::max<u64>(n_kmers, 1) * 8);
    ws.in_b.ensure(n_reads * 8);
    if (n_kmers)
      SBWT_CUDA(cudaMemcpyAsync(ws.in_a.get(), results, n_kmers * 8, cudaMemcpyHostToDevice, st));
    SBWT_CUDA(cudaMemcpyAsync(ws.in_b.get(), read_ends, n_reads * 8, cudaMemcpyHostToDevice, st));
    const u64 cap = format == 0 ? n_kmers * 21 + n_reads
                                : (format == 1 ? 8 * (n_kmers + n_reads) : n_kmers + n_reads);
    ws.out.ensure(std::max<u64>(cap, 1));
    const u64 bytes = format_index_device(ws.in_a.get<uint64_t>(), ws.in_b.get<uint64_t>(),
                                          n_reads, k, format, ws.out.get<uint8_t>(), cap, nullptr,
                                          ws, st);
    *out_bytes = bytes;
    if (bytes > out_capacity) throw Error(SBWT_E_CAPACITY, "output capacity too small");
    if (!out) throw Error(SBWT_E_INVALID, "null output");
    SBWT_CUDA(cudaMemcpyAsync(out, ws.out.get(), bytes, cudaMemcpyDeviceToHost, st));
    SBWT_CUDA(cudaStreamSynchronize(st));
  });
}

extern "C" int sbwt_format_color_results(const uint32_t *ids, const uint64_t *ids_offsets,
                                         uint64_t n_reads, uint64_t num_colors, int format,
                                         char *out, uint64_t out_capacity, uint64_t *out_bytes,
                                         uint32_t flags, int device, void *stream) {
  if (!out_bytes || (n_reads && !ids_offsets) || format < 0 || format > 2 ||
      (format == 2 && num_colors == 0)) {
    set_last_error("invalid argument");
    return SBWT_E_INVALID;
  }
  *out_bytes = 0;
  return guarded([&] {
    DeviceGuard g(device);
    FormatWorkspace &ws = format_workspace(device);
    const bool dev = flags & SBWT_DEVICE_POINTERS;
    cudaStream_t st = dev && stream ? (cudaStream_t)stream : ws.stream;
    if (dev) {
      if (format == 1 && ((uintptr_t)out & 7))
        throw Error(SBWT_E_INVALID, "binary output must be 8-byte aligned");
      *out_bytes = format_colors_device(ids, ids_offsets, n_reads, num_colors, format,
                                        (uint8_t *)out, out_capacity, out_bytes, ws, st);
      SBWT_CUDA(cudaStreamSynchronize(st));
      return;
    }
    if (n_reads == 0) return;
    if (ids_offsets[0] != 0) throw Error(SBWT_E_INVALID, "ids offsets must start at 0");
    for (u64 r = 0; r < n_reads; ++r)
      if (ids_offsets[r + 1] < ids_offsets[r])
        throw Error(SBWT_E_INVALID, "ids offsets must not decrease");
    const u64 n_ids = ids_offsets[n_reads];
    if (n_ids && !ids) throw Error(SBWT_E_INVALID, "null ids");
    ws.in_a.ensure(std::max<u64>(n_ids, 1) * 4);
    ws.in_b.ensure((n_reads + 1) * 8);
    if (n_ids)
      SBWT_CUDA(cudaMemcpyAsync(ws.in_a.get(), ids, n_ids * 4, cudaMemcpyHostToDevice, st));
    SBWT_CUDA(cudaMemcpyAsync(ws.in_b.get(), ids_offsets, (n_reads + 1) * 8,
                              cudaMemcpyHostToDevice, st));
    const u64 cap = format == 0 ? n_ids * 11 + n_reads
                                : (format == 1 ? 8 * (n_ids + n_reads) : n_reads * 2 * num_colors);
    ws.out.ensure(std::max<u64>(cap, 1));
    const u64 bytes =
        format_colors_device(ws.in_a.get<uint32_t>(), ws.in_b.get<uint64_t>(), n_reads,
                             num_colors, format, ws.out.get<uint8_t>(), cap, nullptr, ws, st);
    *out_bytes = bytes;
    if (bytes > out_capacity) throw Error(SBWT_E_CAPACITY, "output capacity too small");
    if (!out) throw Error(SBWT_E_INVALID, "null output");
    SBWT_CUDA(cudaMemcpyAsync(out, ws.out.get(), bytes, cudaMemcpyDeviceToHost, st));
    SBWT_CUDA(cudaStreamSynchronize(st));
  });
}
