// FASTA/FASTQ text -> concatenated sequence chars + read ends, on the GPU.
//
// Record rules are the host reader's (fastx.cpp, itself kseq's as the
// reference uses them: src/SequenceFileParser/ContinuousSequenceFileParser.cpp
// :148-156): lines end at '\n' (one trailing '\r' is dropped when a '\n'
// follows it); lines before the first header ('>' or '@') are skipped; every
// header starts one read; the lines after it are sequence up to the next
// header or a '+' line; after '+', lines are quality until their lengths reach
// the sequence length; then lines are skipped up to the next header.
//
// The steps:
//   1. newline positions, 16 text bytes per load, with what the later steps
//      need of the text beside each (a '\r' before it, the class of the next
//      line's first char), so that only the sequence chars are read again;
//   2. the per-line state (searching | sequence of n chars | quality with r
//      chars still due) is sequential, so one thread runs kFewLines lines from
//      the "searching" state, and also says what the chunk does when entered
//      inside a sequence (its leading lines then are sequence up to the first
//      special line).  These two-way summaries compose, so a scan gives every
//      chunk its entering state and the chars, reads and sequence lines
//      before it;
//   3. the threads run their lines again from the true state and write the
//      read ends and a list of the sequence lines (output offset, text
//      position);
//   4. warps copy the chars by ranges of the output, 16 bytes per lane, each
//      lane finding its line in the list: long and short lines cost the same.
// A chunk that is entered inside quality, or inside a sequence and meets a '+'
// line first, has no such summary (multi-line FASTQ, or FASTQ whose records do
// not start on a chunk): then the roles come from chunks of kChunkLines,
// one warp per chunk, speculatively from "searching" too, and one warp walks
// the chunks in order with the true entering state: a chunk entered
// "searching" is right as it is; one entered inside a sequence whose first
// special line is a header (or that has none) only turns its leading lines
// into sequence lines; anything else is re-run line by line until the re-run
// and the speculation both see a header on the same line, after which both
// states are equal.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>
#include <vector>

#include "common.hpp"

namespace sbwt {

namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr uint32_t kWarpBytes = 4096;  // text bytes per warp in the newline passes
constexpr uint32_t kFewLines = 32;     // lines of a chunk that one thread runs
constexpr uint32_t kChunkLines = 1024;
constexpr int kPrefixLines = 8;

enum : uint8_t { R_SKIP = 0, R_HEADER = 1, R_SEQ = 2, R_PLUS = 3, R_QUAL = 4 };
enum : uint32_t { S_SEARCH = 0, S_SEQ = 1, S_QUAL = 2 };

// A '\n': its position << 3 | kCr (a '\r' before it) | the class of the first
// char after it.
constexpr uint64_t kCr = 4, kHeaderClass = 1, kPlusClass = 2;

struct Lines {
  const uint8_t *text;
  uint64_t n_bytes;
  const uint64_t *nl;  // the '\n' bytes
  uint64_t n_nl;
  uint64_t n_lines;    // n_nl, + 1 when the text does not end with '\n'
};

__device__ __forceinline__ uint64_t char_class(uint32_t c) {
  return c == '>' || c == '@' ? kHeaderClass : (c == '+' ? kPlusClass : 0);
}

// Line i: its first byte, its length (without the '\r' before its '\n') and
// its first char as far as it matters ('>' for a header, '+', '\n' for an
// empty line, else 'A').
// before, e: the entries of the newlines before and after it.
__device__ __forceinline__ void line_of(const Lines &L, uint64_t i, uint64_t before, uint64_t e,
                                        uint64_t &start, uint32_t &len, uint8_t &c0) {
  const uint64_t cls = i ? before & 3 : char_class(L.text[0]);
  start = i ? (before >> 3) + 1 : 0;
  uint64_t n = L.n_bytes - start;
  if (i < L.n_nl) {
    n = (e >> 3) - start;
    if (n > 0 && (e & kCr)) --n;
  }
  len = (uint32_t)min(n, (uint64_t)0xFFFFFFFFu);
  c0 = n == 0 ? '\n' : (cls == kHeaderClass ? '>' : (cls == kPlusClass ? '+' : 'A'));
}
__device__ __forceinline__ void line_at(const Lines &L, uint64_t i, uint64_t &start,
                                        uint32_t &len, uint8_t &c0) {
  line_of(L, i, i ? __ldg(L.nl + i - 1) : 0, i < L.n_nl ? __ldg(L.nl + i) : 0, start, len, c0);
}

// f(start, length, first char) of the lines [l0, l0 + n), l0 a multiple of 8:
// the entries of eight newlines are loaded together, those of the next eight
// while these lines are looked at.
template <class F>
__device__ __forceinline__ void each_line(const Lines &L, uint64_t l0, uint32_t n, F f) {
  uint64_t e[8], next[8];
  auto load = [&](uint64_t i, uint64_t (&x)[8]) {
    if (i + 8 <= L.n_nl) {
#pragma unroll
      for (int q = 0; q < 8; q += 2) {
        const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(L.nl + i + q));
        x[q] = v.x;
        x[q + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = i + q < L.n_nl ? __ldg(L.nl + i + q) : 0;
    }
  };
  uint64_t before = l0 ? __ldg(L.nl + l0 - 1) : 0;
  load(l0, next);
  for (uint32_t j = 0; j < n; j += 8) {
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = next[q];
    if (j + 8 < n) load(l0 + j + 8, next);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (j + q >= n) break;
      uint64_t start;
      uint32_t len;
      uint8_t c0;
      line_of(L, l0 + j + q, before, e[q], start, len, c0);
      before = e[q];
      f(start, len, c0);
    }
  }
}

// One line through the record state machine; returns its role.
__device__ __forceinline__ uint8_t step(uint32_t &mode, uint64_t &a, uint32_t len, uint8_t c0) {
  const bool hdr = len > 0 && (c0 == '>' || c0 == '@');
  if (mode == S_SEARCH) {
    if (!hdr) return R_SKIP;
    mode = S_SEQ;
    a = 0;
    return R_HEADER;
  }
  if (mode == S_SEQ) {
    if (hdr) {
      a = 0;
      return R_HEADER;
    }
    if (len > 0 && c0 == '+') {
      mode = a ? S_QUAL : S_SEARCH;  // a: the sequence length, now quality due
      return R_PLUS;
    }
    a += len;
    return R_SEQ;
  }
  a = a > len ? a - len : 0;  // quality
  if (a == 0) mode = S_SEARCH;
  return R_QUAL;
}

__device__ __forceinline__ bool is_special(uint32_t len, uint8_t c0) {
  return len > 0 && (c0 == '>' || c0 == '@' || c0 == '+');
}

struct ChunkInfo {
  uint64_t end_a;          // speculative end state
  uint64_t pre_len;        // sequence chars before the first special line
  uint64_t prefix[kPrefixLines];  // (len << 8) | c0 of the first lines
  uint32_t end_mode;
  uint32_t first_special;  // index in the chunk, n_in_chunk when none
  uint32_t n_in_chunk;
  uint32_t special_c0;     // first char of that line
  uint32_t seq_prefix;     // set by the fix-up: leading lines that are sequence
  uint32_t pad;
};

// 16 text bytes from position p (p may lie before or past the text: 0 there);
// aligned loads when all of them are text.
__device__ __forceinline__ uint4 text16(const uint8_t *text, uint64_t n, int64_t p) {
  uint4 x = make_uint4(0, 0, 0, 0);
  if (p >= 0 && (uint64_t)p + 16 <= n) return __ldcs(reinterpret_cast<const uint4 *>(text + p));
  if (p + 16 <= 0 || p >= (int64_t)n) return x;
  uint32_t *const w = &x.x;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (p + i >= 0 && p + i < (int64_t)n) w[i >> 2] |= (uint32_t)text[p + i] << (8 * (i & 3));
  return x;
}

// Bit i of the result: byte i of x is c (repeated in c4).
__device__ __forceinline__ uint32_t equal_bits(uint32_t x, uint32_t c4) {
  const uint32_t y = x ^ c4;
  const uint32_t z = ~(((y & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | y | 0x7F7F7F7Fu) >> 7;
  return (z * 0x10204080u) >> 28;
}
__device__ __forceinline__ uint32_t equal_bits16(const uint4 &x, uint32_t c) {
  const uint32_t c4 = c * 0x01010101u;
  return equal_bits(x.x, c4) | equal_bits(x.y, c4) << 4 | equal_bits(x.z, c4) << 8 |
         equal_bits(x.w, c4) << 12;
}

// A warp takes kWarpBytes bytes of the text in 16-byte lines of memory (the
// text may start inside one: `lead` bytes into it), kNlLoads per lane.
constexpr int kNlLoads = kWarpBytes / 512;

// marks: a bit per byte, a word of kNlLoads 16-bit masks per lane.
static_assert(kNlLoads == 8, "a lane's masks fill a uint4");
__global__ void nl_count_kernel(const uint8_t *text, uint64_t n, uint32_t lead,
                                uint64_t *warp_counts, uint64_t n_warps, uint4 *marks) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (w >= n_warps) return;
  const int64_t p0 = (int64_t)(w * kWarpBytes + 16 * lane) - lead;
  uint4 x[kNlLoads];
#pragma unroll
  for (int i = 0; i < kNlLoads; ++i) x[i] = text16(text, n, p0 + 512 * i);
  uint32_t m[kNlLoads / 2], cnt = 0;
#pragma unroll
  for (int i = 0; i < kNlLoads / 2; ++i) {
    m[i] = equal_bits16(x[2 * i], '\n') | equal_bits16(x[2 * i + 1], '\n') << 16;
    cnt += __popc(m[i]);
  }
  marks[w * 32 + lane] = make_uint4(m[0], m[1], m[2], m[3]);
  cnt = __reduce_add_sync(FULL, cnt);
  if (lane == 0) warp_counts[w] = cnt;
}

// The lanes collect the places of the warp's newlines in shared memory, then
// take one newline each (its neighbours from L1, whole lines of stores).
// What is left is the scan's instructions and the neighbours' sectors: 355 MB of
// FASTQ with 4 M lines in 66 us from nl_count_kernel's marks (44 MB, mostly in
// L2), 111 us when it read the text again, 200 us with a scan per load and the
// stores beside it, 370 us byte by byte; nl_count_kernel 62 us, the text at
// 5.7 TB/s, with or without the marks (190 us byte by byte).
constexpr uint32_t kNlList = 1024;  // places held before they are written
__global__ void __launch_bounds__(256)
    nl_write_kernel(const uint8_t *text, uint64_t n, uint32_t lead, const uint64_t *warp_off,
                    uint64_t n_warps, const uint4 *marks, uint64_t *nl) {
  __shared__ uint16_t sh_list[8][kNlList];
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (w >= n_warps) return;
  uint16_t *const list = sh_list[threadIdx.x >> 5];
  const int64_t w0 = (int64_t)(w * kWarpBytes) - lead;
  const uint4 mk = __ldcs(marks + w * 32 + lane);
  const uint32_t m2[kNlLoads / 2] = {mk.x, mk.y, mk.z, mk.w};
  uint32_t mask[kNlLoads];
  // counts of four loads per word, 16 bits each, scanned over the lanes
  uint64_t cnt[kNlLoads / 4], incl[kNlLoads / 4];
#pragma unroll
  for (int g = 0; g < kNlLoads / 4; ++g) {
    cnt[g] = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      mask[4 * g + i] = (m2[2 * g + i / 2] >> (16 * (i & 1))) & 0xFFFFu;
      cnt[g] |= (uint64_t)__popc(mask[4 * g + i]) << (16 * i);
    }
    incl[g] = cnt[g];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(FULL, incl[g], o);
      if (lane >= (uint32_t)o) incl[g] += y;
    }
  }
  uint64_t at = warp_off[w];
  uint32_t held = 0;  // places in the list
  auto flush = [&] {
    __syncwarp();
    for (uint32_t j = lane; j < held; j += 32) {
      const int64_t p = w0 + list[j];
      const uint32_t pv = p > 0 ? text[p - 1] : 0, nx = p + 1 < (int64_t)n ? text[p + 1] : 0;
      nl[at + j] = (uint64_t)p << 3 | (pv == '\r' ? kCr : 0) | char_class(nx);
    }
    at += held;
    held = 0;
    __syncwarp();
  };
#pragma unroll
  for (int i = 0; i < kNlLoads; ++i) {
    const uint32_t total =
        (uint32_t)(__shfl_sync(FULL, incl[i / 4], 31) >> (16 * (i % 4))) & 0xFFFF;
    if (held + total > kNlList) flush();
    uint32_t o = held + ((uint32_t)((incl[i / 4] - cnt[i / 4]) >> (16 * (i % 4))) & 0xFFFF);
    for (uint32_t m = mask[i]; m; m &= m - 1, ++o)
      list[o] = (uint16_t)(512 * i + 16 * lane + __ffs(m) - 1);
    held += total;
  }
  flush();
}

// In-place exclusive scan of v[0..n) by one block; v[n] = total.
__global__ void scan_small_kernel(uint64_t *v, uint64_t n) {
  __shared__ uint64_t wsum[32];
  __shared__ uint64_t carry;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint64_t b = 0; b < n; b += blockDim.x) {
    const uint64_t i = b + threadIdx.x;
    const uint64_t x0 = i < n ? v[i] : 0;
    uint64_t x = x0;
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
    const uint64_t ex = carry + (wid ? wsum[wid - 1] : 0) + x - x0;
    if (i < n) v[i] = ex;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = ex + x0;
    __syncthreads();
  }
  if (threadIdx.x == 0) v[n] = carry;
}

// The same in three launches for more values: block totals, their scan
// (scan_small_kernel), then every block adds its own.
constexpr uint32_t kScanSpan = 8192;
__global__ void __launch_bounds__(1024) scan_totals_kernel(const uint64_t *v, uint64_t n,
                                                           uint64_t *tops) {
  __shared__ uint64_t sums[32];
  const uint64_t b0 = blockIdx.x * (uint64_t)kScanSpan;
  uint64_t s = 0;
  for (uint32_t i = threadIdx.x; i < kScanSpan; i += 1024)
    if (b0 + i < n) s += v[b0 + i];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sums[threadIdx.x];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
    if (threadIdx.x == 0) tops[blockIdx.x] = s;
  }
}
__global__ void __launch_bounds__(1024) scan_apply_kernel(uint64_t *v, uint64_t n,
                                                          const uint64_t *tops) {
  __shared__ uint64_t sums[32];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint64_t i0 = blockIdx.x * (uint64_t)kScanSpan + threadIdx.x * 8ULL;
  uint64_t c[8], s = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    c[q] = i0 + q < n ? v[i0 + q] : 0;
    s += c[q];
  }
  uint64_t x = s;
  for (int o = 1; o < 32; o <<= 1) {
    const uint64_t y = __shfl_up_sync(FULL, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) sums[wid] = x;
  __syncthreads();
  uint64_t at = tops[blockIdx.x] + x - s;
  for (uint32_t w = 0; w < wid; ++w) at += sums[w];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (i0 + q < n) v[i0 + q] = at;
    at += c[q];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) v[n] = tops[gridDim.x];
}

// One warp per chunk: speculative roles (from "searching") + summaries.
__global__ void roles_kernel(Lines L, uint8_t *roles, ChunkInfo *ci, uint64_t n_chunks) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (c >= n_chunks) return;
  const uint64_t l0 = c * kChunkLines;
  const uint32_t n_in = (uint32_t)min((uint64_t)kChunkLines, L.n_lines - l0);
  uint32_t mode = S_SEARCH, first_special = n_in, special_c0 = 0;
  uint64_t a = 0, pre_len = 0;
  for (uint32_t r0 = 0; r0 < n_in; r0 += 32) {
    uint64_t start = 0;
    uint32_t len = 0;
    uint8_t c0 = '\n';
    if (r0 + lane < n_in) line_at(L, l0 + r0 + lane, start, len, c0);
    if (r0 == 0 && lane < kPrefixLines)
      ci[c].prefix[lane] = ((uint64_t)len << 8) | c0;
    // first special line and the chars before it
    if (first_special == n_in) {
      const uint32_t sp = __ballot_sync(FULL, r0 + lane < n_in && is_special(len, c0));
      const uint32_t upto = sp ? (1u << (__ffs(sp) - 1)) - 1 : FULL;
      uint64_t part = (upto >> lane) & 1u ? len : 0;
      for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
      pre_len += part;
      if (sp) {
        first_special = r0 + __ffs(sp) - 1;
        special_c0 = __shfl_sync(FULL, (uint32_t)c0, __ffs(sp) - 1);
      }
    }
    uint8_t my_role = R_SKIP;
    const uint32_t m = min(32u, n_in - r0);
    for (uint32_t q = 0; q < m; ++q) {
      const uint32_t lq = __shfl_sync(FULL, len, q);
      const uint8_t cq = (uint8_t)__shfl_sync(FULL, (uint32_t)c0, q);
      const uint8_t role = step(mode, a, lq, cq);
      if (lane == q) my_role = role;
    }
    if (r0 + lane < n_in) roles[l0 + r0 + lane] = my_role;
  }
  if (lane == 0) {
    ci[c].end_a = a;
    ci[c].end_mode = mode;
    ci[c].pre_len = pre_len;
    ci[c].first_special = first_special;
    ci[c].special_c0 = special_c0;
    ci[c].n_in_chunk = n_in;
    ci[c].seq_prefix = 0;
  }
}

// Re-runs chunk c line by line from the true entering state until the re-run
// and the speculation both see a header on the same line (then their states
// are equal and the speculative end state holds); corrects the roles on the
// way.  All lanes compute the same; lane 0 writes.  prefix, spec: the chunk's
// first kPrefixLines lines and roles; the lines after them come 32 at a time,
// one per lane.
__device__ void rerun_chunk(const Lines &L, uint8_t *roles, uint64_t c, uint32_t n_in,
                            uint32_t end_mode, uint64_t end_a, const uint64_t *prefix,
                            uint64_t spec, uint32_t &mode, uint64_t &a, uint32_t lane) {
  const uint64_t l0 = c * kChunkLines;
  auto line = [&](uint32_t j, uint32_t len, uint8_t c0, uint8_t was) {  // true: at a common header
    const uint8_t role = step(mode, a, len, c0);
    if (role == R_HEADER && was == R_HEADER) {
      mode = end_mode;
      a = end_a;
      return true;
    }
    if (lane == 0 && role != was) roles[l0 + j] = role;
    return false;
  };
  for (uint32_t j = 0; j < min(n_in, (uint32_t)kPrefixLines); ++j)
    if (line(j, (uint32_t)(prefix[j] >> 8), (uint8_t)prefix[j], (uint8_t)(spec >> (8 * j)))) return;
  for (uint32_t j0 = kPrefixLines; j0 < n_in; j0 += 32) {
    uint64_t start;
    uint32_t len = 0, was = R_SKIP;
    uint8_t c0 = '\n';
    if (j0 + lane < n_in) {
      line_at(L, l0 + j0 + lane, start, len, c0);
      was = roles[l0 + j0 + lane];
    }
    __syncwarp();
    const uint32_t m = min(32u, n_in - j0);
    for (uint32_t q = 0; q < m; ++q)
      if (line(j0 + q, __shfl_sync(FULL, len, q), (uint8_t)__shfl_sync(FULL, (uint32_t)c0, q),
               (uint8_t)__shfl_sync(FULL, was, q)))
        return;
    __syncwarp();
  }
}

// One warp walks the chunks in order with the true entering state; lanes
// fetch the summaries and first lines of 32 chunks at a time, the state steps
// through them by shuffles.
// What bounds it: the serial chain over the chunks.  With the first lines loaded
// chunk by chunk, 200 k records (800 k lines) one line off the chunks took 1.18
// ms a call, now 0.88 ms; wrapped sequences 1.40 -> 0.96 ms.
static_assert(kPrefixLines == 8, "a chunk's first roles are one word");
__global__ void fixup_kernel(Lines L, uint8_t *roles, ChunkInfo *ci, uint64_t n_chunks) {
  __shared__ uint64_t sh_prefix[32][kPrefixLines + 1];
  const uint32_t lane = threadIdx.x & 31;
  uint32_t mode = S_SEARCH;
  uint64_t a = 0;
  for (uint64_t c0 = 0; c0 < n_chunks; c0 += 32) {
    const uint64_t c = c0 + lane;
    uint32_t em = 0, fs = 0, nin = 0, sc = 0;
    uint64_t ea = 0, pl = 0, sr = 0;
    __syncwarp();
    if (c < n_chunks) {
      em = ci[c].end_mode;
      ea = ci[c].end_a;
      fs = ci[c].first_special;
      nin = ci[c].n_in_chunk;
      sc = ci[c].special_c0;
      pl = ci[c].pre_len;
      for (int j = 0; j < kPrefixLines; ++j) sh_prefix[lane][j] = ci[c].prefix[j];
      // (8 bytes past the last role belong to the buffer)
      sr = *reinterpret_cast<const uint64_t *>(roles + c * kChunkLines);
    }
    __syncwarp();
    const uint32_t m = (uint32_t)min((uint64_t)32, n_chunks - c0);
    for (uint32_t q = 0; q < m; ++q) {
      const uint32_t q_em = __shfl_sync(FULL, em, q), q_fs = __shfl_sync(FULL, fs, q);
      const uint32_t q_nin = __shfl_sync(FULL, nin, q), q_sc = __shfl_sync(FULL, sc, q);
      const uint64_t q_ea = __shfl_sync(FULL, ea, q), q_pl = __shfl_sync(FULL, pl, q);
      const uint64_t q_sr = __shfl_sync(FULL, sr, q);
      if (mode == S_SEARCH) {  // the speculation was right
        mode = q_em;
        a = q_ea;
      } else if (mode == S_SEQ && (q_fs == q_nin || q_sc != '+')) {
        // the leading lines continue the open sequence, then as speculated
        if (lane == 0) ci[c0 + q].seq_prefix = q_fs;
        if (q_fs == q_nin) {
          a += q_pl;
        } else {
          mode = q_em;
          a = q_ea;
        }
      } else {
        rerun_chunk(L, roles, c0 + q, q_nin, q_em, q_ea, sh_prefix[q], q_sr, mode, a, lane);
      }
    }
  }
}

__device__ __forceinline__ uint8_t final_role(const uint8_t *roles, const ChunkInfo &k,
                                              uint64_t l0, uint32_t j) {
  return j < k.seq_prefix ? R_SEQ : roles[l0 + j];
}

// Per chunk: sequence chars -> tot[c], headers -> tot[n_chunks + 1 + c].
__global__ void chunk_totals_kernel(Lines L, const uint8_t *roles, const ChunkInfo *ci,
                                    uint64_t n_chunks, uint64_t *chars_tot,
                                    uint64_t *hdr_tot) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (c >= n_chunks) return;
  const ChunkInfo &k = ci[c];
  const uint64_t l0 = c * kChunkLines;
  uint64_t chars = 0, hdrs = 0;
  for (uint32_t j = lane; j < k.n_in_chunk; j += 32) {
    const uint8_t role = final_role(roles, k, l0, j);
    if (role == R_SEQ) {
      uint64_t start;
      uint32_t len;
      uint8_t c0;
      line_at(L, l0 + j, start, len, c0);
      chars += len;
    }
    hdrs += role == R_HEADER;
  }
  for (int o = 16; o; o >>= 1) {
    chars += __shfl_xor_sync(FULL, chars, o);
    hdrs += __shfl_xor_sync(FULL, hdrs, o);
  }
  if (lane == 0) {
    chars_tot[c] = chars;
    hdr_tot[c] = hdrs;
  }
}

// One warp per chunk: sequence chars to out at their offsets; for the read
// opened by header h > 0, the end of read h - 1.
__global__ void emit_kernel(Lines L, const uint8_t *roles, const ChunkInfo *ci,
                            uint64_t n_chunks, const uint64_t *chars_off,
                            const uint64_t *hdr_off, uint8_t *out, uint64_t *ends) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t c = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  if (c >= n_chunks) return;
  const ChunkInfo &k = ci[c];
  const uint64_t l0 = c * kChunkLines;
  uint64_t at = chars_off[c], h = hdr_off[c];
  for (uint32_t r0 = 0; r0 < k.n_in_chunk; r0 += 32) {
    const uint32_t j = r0 + lane;
    uint8_t role = R_SKIP;
    uint64_t start = 0;
    uint32_t len = 0;
    uint8_t c0;
    if (j < k.n_in_chunk) {
      role = final_role(roles, k, l0, j);
      line_at(L, l0 + j, start, len, c0);
    }
    const uint64_t my_chars = role == R_SEQ ? len : 0;
    uint64_t x = my_chars;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(FULL, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    const uint64_t my_at = at + x - my_chars;
    const uint32_t hm = __ballot_sync(FULL, role == R_HEADER);
    const uint64_t my_h = h + __popc(hm & ((1u << lane) - 1));
    if (role == R_HEADER && my_h > 0) ends[my_h - 1] = my_at;
    const uint32_t sm = __ballot_sync(FULL, role == R_SEQ && len > 0);
    for (uint32_t m = sm; m; m &= m - 1) {
      const int q = __ffs(m) - 1;
      const uint64_t s = __shfl_sync(FULL, start, q);
      const uint64_t d = __shfl_sync(FULL, my_at, q);
      const uint32_t n = __shfl_sync(FULL, len, q);
      for (uint32_t i = lane; i < n; i += 32) out[d + i] = L.text[s + i];
    }
    at = __shfl_sync(FULL, my_at + my_chars, 31);
    h += __popc(hm);
  }
}

// ---- chunks of kFewLines lines -----------------------------------------------
// 4 M lines: few_lines_kernel 20 us, the scan 21 us, list_lines_kernel 23 us
// (latency of a thread's own lines: 40 and 47 us when each newline's entry was
// loaded as its line came up, instead of eight together and ahead); the roles
// by one warp per kChunkLines and the one-warp fix-up took 450 us.
// What a run of lines does when entered searching (0) or inside a sequence (1):
// the state after it (kQuality: inside quality) and the chars and non-empty
// sequence lines in it; its headers are the same either way.  kUnknown: some
// chunk of the run is entered inside quality, or inside a sequence and meets a
// '+' line first (how much quality is due depends on the chunks before it): the
// state, chars, lines and headers are not known.
constexpr uint32_t kQuality = 2, kUnknown = 3;
struct Trans {
  uint64_t chars[2], lines[2], headers;
  uint32_t to[2];
};
__device__ __forceinline__ Trans then(const Trans &a, const Trans &b) {
  Trans r;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t m = a.to[s];
    r.to[s] = m >= kQuality ? kUnknown : (m ? b.to[1] : b.to[0]);
    r.chars[s] = a.chars[s] + (m ? b.chars[1] : b.chars[0]);
    r.lines[s] = a.lines[s] + (m ? b.lines[1] : b.lines[0]);
  }
  r.headers = a.headers + b.headers;
  return r;
}
// The run of no lines.  To the right of a run it stands only where a chunk
// follows (which is then entered in that run's state) or past the last chunk.
__device__ __forceinline__ Trans no_lines() { return Trans{{0, 0}, {0, 0}, 0, {0, 1}}; }

// Where a chunk starts: its entering state and what is before it.
struct Entry {
  uint64_t chars, lines, headers;
  uint64_t state;
};

__global__ void __launch_bounds__(256) few_lines_kernel(Lines L, uint64_t n_chunks, Trans *out) {
  const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (c >= n_chunks) return;
  const uint64_t l0 = c * kFewLines;
  const uint32_t n_in = (uint32_t)min((uint64_t)kFewLines, L.n_lines - l0);
  Trans t = no_lines();
  uint64_t pre_chars = 0, pre_lines = 0, a = 0;
  uint32_t mode = S_SEARCH;
  bool before_special = true, plus_first = false;
  each_line(L, l0, n_in, [&](uint64_t, uint32_t len, uint8_t c0) {
    if (before_special) {
      if (is_special(len, c0)) {
        before_special = false;
        plus_first = c0 == '+';
      } else {
        pre_chars += len;
        pre_lines += len > 0;
      }
    }
    const uint8_t role = step(mode, a, len, c0);
    if (role == R_SEQ) {
      t.chars[0] += len;
      t.lines[0] += len > 0;
    }
    t.headers += role == R_HEADER;
  });
  t.to[0] = mode == S_SEARCH ? 0 : (mode == S_SEQ ? 1 : kQuality);
  t.to[1] = before_special ? 1 : (plus_first ? kUnknown : t.to[0]);
  t.chars[1] = pre_chars + t.chars[0];
  t.lines[1] = pre_lines + t.lines[0];
  out[c] = t;
}

// Exclusive composition over the threads of a block; *total: of all.
__device__ __forceinline__ Trans block_before(const Trans &mine, Trans *sh, Trans *total) {
  const uint32_t t = threadIdx.x;
  sh[t] = mine;
  __syncthreads();
  Trans x = mine;
  for (uint32_t o = 1; o < blockDim.x; o <<= 1) {
    Trans y = no_lines();
    if (t >= o) y = sh[t - o];
    __syncthreads();
    if (t >= o) {
      x = then(y, x);
      sh[t] = x;
    }
    __syncthreads();
  }
  *total = sh[blockDim.x - 1];
  const Trans before = t ? sh[t - 1] : no_lines();
  __syncthreads();
  return before;
}

constexpr uint32_t kScanBlock = 256, kPerThread = 4, kBlockChunks = kScanBlock * kPerThread;

__device__ __forceinline__ Trans thread_trans(const Trans *t, uint64_t c0, uint64_t n) {
  Trans x = no_lines();
  for (uint32_t q = 0; q < kPerThread; ++q)
    if (c0 + q < n) x = then(x, t[c0 + q]);
  return x;
}

// Block totals, for more chunks than one block scans.
__global__ void __launch_bounds__(kScanBlock) trans_totals_kernel(const Trans *t, uint64_t n,
                                                                  Trans *tops) {
  __shared__ Trans sh[kScanBlock];
  Trans total;
  const uint64_t c0 = blockIdx.x * (uint64_t)kBlockChunks + threadIdx.x * kPerThread;
  block_before(thread_trans(t, c0, n), sh, &total);
  if (threadIdx.x == 0) tops[blockIdx.x] = total;
}
// tops[b] = the composition of the blocks before b.
__global__ void __launch_bounds__(kScanBlock) trans_tops_kernel(Trans *tops, uint64_t n_blocks) {
  __shared__ Trans sh[kScanBlock];
  Trans carry = no_lines();
  for (uint64_t b0 = 0; b0 < n_blocks; b0 += kScanBlock) {
    const uint64_t b = b0 + threadIdx.x;
    Trans total;
    const Trans before = block_before(b < n_blocks ? tops[b] : no_lines(), sh, &total);
    if (b < n_blocks) tops[b] = then(carry, before);
    carry = then(carry, total);
  }
}
// Every chunk's entry; status: chars, reads, sequence lines of the text, and 1
// when they are not known.
__global__ void __launch_bounds__(kScanBlock) trans_apply_kernel(const Trans *t, uint64_t n,
                                                                 const Trans *tops, Entry *entry,
                                                                 uint64_t *status) {
  __shared__ Trans sh[kScanBlock];
  Trans total;
  const uint64_t c0 = blockIdx.x * (uint64_t)kBlockChunks + threadIdx.x * kPerThread;
  Trans x = block_before(thread_trans(t, c0, n), sh, &total);
  if (tops) x = then(tops[blockIdx.x], x);
  for (uint32_t q = 0; q < kPerThread && c0 + q < n; ++q) {
    entry[c0 + q] = Entry{x.chars[0], x.lines[0], x.headers, x.to[0]};
    x = then(x, t[c0 + q]);
    if (c0 + q == n - 1) {  // (a text may end inside quality)
      status[3] = x.to[0] == kUnknown;
      status[0] = x.chars[0];
      status[1] = x.headers;
      status[2] = x.lines[0];
    }
  }
}

// Read ends, and the sequence lines: line_off (n_lines + 1), and line_src, the
// lines' places in the text minus line_off.
__global__ void __launch_bounds__(256)
    list_lines_kernel(Lines L, uint64_t n_chunks, const Entry *entry, const uint64_t *status,
                      uint64_t *ends, uint64_t *line_off, uint64_t *line_src) {
  const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (c >= n_chunks) return;
  const Entry e = entry[c];
  const uint64_t l0 = c * kFewLines;
  const uint32_t n_in = (uint32_t)min((uint64_t)kFewLines, L.n_lines - l0);
  uint64_t at = e.chars, line = e.lines, h = e.headers, a = 0;
  uint32_t mode = e.state ? S_SEQ : S_SEARCH;
  each_line(L, l0, n_in, [&](uint64_t start, uint32_t len, uint8_t c0) {
    const uint8_t role = step(mode, a, len, c0);
    if (role == R_HEADER) {
      if (h) ends[h - 1] = at;
      ++h;
    } else if (role == R_SEQ && len) {
      line_off[line] = at;
      line_src[line] = start - at;
      ++line;
      at += len;
    }
  });
  if (c == n_chunks - 1) {
    line_off[status[2]] = status[0];
    if (status[1]) ends[status[1] - 1] = status[0];
  }
}

// 16 text bytes at p (p may start before the text or end past it by up to 20
// bytes; what is outside is arbitrary), from aligned words.
__device__ __forceinline__ void bytes16(const uint8_t *text, uint64_t n_bytes, intptr_t p,
                                        uint32_t (&v)[4]) {
  const intptr_t lo = (intptr_t)text & ~(intptr_t)3, hi = ((intptr_t)text + (intptr_t)n_bytes - 1) & ~(intptr_t)3;
  const intptr_t s0 = p & ~(intptr_t)3;
  uint32_t x[5];
  if (s0 >= lo && s0 + 16 <= hi) {
#pragma unroll
    for (int u = 0; u < 5; ++u) x[u] = __ldg(reinterpret_cast<const uint32_t *>(s0) + u);
  } else {
#pragma unroll
    for (int u = 0; u < 5; ++u)
      x[u] = __ldg(reinterpret_cast<const uint32_t *>(min(max(s0 + 4 * u, lo), hi)));
  }
  const uint32_t f = 8 * (uint32_t)(p & 3);
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = __funnelshift_r(x[u], x[u + 1], f);
}

// Copies the sequence lines to out, a warp per `span` output bytes (a multiple
// of 512), in 16-byte lines of the output's memory (`lead`: the output's first
// byte in its line).  line_src[i]: where line i starts in the text, minus
// line_off[i].
// What bounds it: instructions (~270 per 512 bytes), at 2.7 TB/s of text and
// output: 128 us for 170 MB of reads of 150 chars; a warp per line with byte
// loads and stores took 367 us, and a line per chunk serialised long lines.
__global__ void __launch_bounds__(256)
    copy_lines_kernel(const uint8_t *text, uint64_t n_bytes, const uint64_t *line_off,
                      const uint64_t *line_src, uint64_t n_lines, uint64_t n_chars, uint32_t lead,
                      uint32_t span, uint8_t *out) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t first = (int64_t)(w * span) - lead, end = (int64_t)n_chars;
  if (first >= end) return;
  // the line of the warp's first byte: the last one with line_off <= it
  uint64_t lo = 0, hi = n_lines;  // line_off[lo] <= pos < line_off[hi]
  const uint64_t pos = first > 0 ? (uint64_t)first : 0;
  while (hi - lo > 1) {  // 32 probes a step
    const uint64_t step = (hi - lo + 31) / 32, p = lo + step * lane;
    const unsigned le = __ballot_sync(FULL, p < hi && __ldg(line_off + p) <= pos);
    const uint32_t k = 31 - __clz(le);  // lane 0 always holds
    hi = min(hi, lo + step * (k + 1));
    lo += step * k;
  }
  for (uint32_t i = 0; i < span; i += 512) {
    const int64_t c0 = first + i;  // the warp's 512 bytes
    if (c0 >= end) break;
    // where the next 32 lines start, from c0 on (far: beyond the 512 bytes)
    const uint64_t idx = min(lo + 1 + lane, n_lines);
    const int32_t rel = (int32_t)min((int64_t)__ldg(line_off + idx) - c0, (int64_t)0x7FFFFFFF);
    // this lane's bytes [j0, j1) of the 16 from o = c0 + 16 lane on
    const int64_t o = c0 + 16 * lane;
    const int32_t at = 16 * (int32_t)lane;
    const int32_t j0 = c0 < 0 && lane == 0 ? (int32_t)-c0 : 0;
    const int32_t j1 = (int32_t)min(end - c0, (int64_t)1024) - at;  // 16 and more: all
    uint32_t k = 0;  // lines lo + 1 .. lo + k start at or before byte j0
#pragma unroll
    for (uint32_t s = 16; s; s >>= 1)
      if (__shfl_sync(FULL, rel, k + s - 1) <= at + j0) k += s;
    int32_t stop = __shfl_sync(FULL, rel, k) - at;  // where the line ends
    uint64_t line = lo + k;
    if (j0 < j1) {
      if (stop <= j0) {  // 32 or more lines in 512 bytes: search on
        do {
          ++line;
        } while ((int64_t)__ldg(line_off + line + 1) <= o + j0);
        stop = (int32_t)min((int64_t)__ldg(line_off + line + 1) - o, (int64_t)16);
      }
      uint32_t v[4];
      bytes16(text, n_bytes, (intptr_t)text + o + (intptr_t)__ldg(line_src + line), v);
      while (stop < min(j1, 16)) {  // the next line's bytes from `stop` on
        ++line;
        uint32_t y[4];
        bytes16(text, n_bytes, (intptr_t)text + o + (intptr_t)__ldg(line_src + line), y);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int32_t from = stop - 4 * u;  // the first byte of word u to take
          const uint32_t keep = from <= 0 ? 0u : (from >= 4 ? ~0u : (1u << (8 * from)) - 1u);
          v[u] = (v[u] & keep) | (y[u] & ~keep);
        }
        stop = (int32_t)min((int64_t)__ldg(line_off + line + 1) - o, (int64_t)16);
      }
      if (j0 == 0 && j1 >= 16) {
        *reinterpret_cast<uint4 *>(out + o) = make_uint4(v[0], v[1], v[2], v[3]);
      } else {  // the output's first or last line
        for (int32_t j = j0; j < min(j1, 16); ++j)
          out[o + j] = (uint8_t)(v[j >> 2] >> (8 * (j & 3)));
      }
    }
    // the line of the next 512 bytes' first byte
    const bool past = rel <= 512 && idx < n_lines;
    const unsigned pm = __ballot_sync(FULL, past);
    lo += __popc(pm);
    if (pm >> 31)  // more lines than were looked at
      while (lo + 1 < n_lines && (int64_t)__ldg(line_off + lo + 1) <= c0 + 512) ++lo;
  }
}

__global__ void set_u64_kernel(uint64_t *p, const uint64_t *value) { *p = *value; }

struct FastxWorkspace {
  DeviceBuffer text, warp_counts, nl, roles, chunks, chars_tot, hdr_tot, stats, chars, ends;
  DeviceBuffer trans, tops, entries, line_off, line_src, marks;
  cudaStream_t stream = nullptr;
  u64 *host = nullptr;  // pinned: four counts
  ~FastxWorkspace() {
    if (stream) cudaStreamDestroy(stream);
    if (host) cudaFreeHost(host);
  }
};

FastxWorkspace &fastx_workspace(int device) {
  thread_local std::unique_ptr<FastxWorkspace> ws[16];
  if (device < 0 || device >= 16) throw Error(SBWT_E_INVALID, "device id out of range");
  auto &p = ws[device];
  if (!p) {
    p = std::make_unique<FastxWorkspace>();
    SBWT_CUDA(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
    SBWT_CUDA(cudaMallocHost(&p->host, 32));
  }
  return *p;
}

unsigned grid_for_warps(uint64_t warps) {
  return (unsigned)std::max<uint64_t>((warps + 7) / 8, 1);  // 256 threads per block
}

// v[0..n) (n + 1 entries) -> exclusive offsets, v[n] = total.
void enqueue_scan(u64 *v, u64 n, FastxWorkspace &ws, cudaStream_t st) {
  if (n <= kScanSpan) {
    scan_small_kernel<<<1, 1024, 0, st>>>(v, n);
  } else {
    const u64 nb = (n + kScanSpan - 1) / kScanSpan;
    ws.tops.ensure((nb + 1) * 8);
    u64 *tops = ws.tops.get<u64>();
    scan_totals_kernel<<<(unsigned)nb, 1024, 0, st>>>(v, n, tops);
    scan_small_kernel<<<1, 1024, 0, st>>>(tops, nb);
    scan_apply_kernel<<<(unsigned)nb, 1024, 0, st>>>(v, n, tops);
  }
  SBWT_CUDA(cudaGetLastError());
}

}  // namespace

// Device-resident text through newline positions, line states and totals
// (fastx_count), then the chars and read ends (fastx_emit).
struct ParsePlan {
  Lines L{};
  bool few = false;  // chunks of kFewLines, else of kChunkLines (see the top)
  u64 n_chunks = 0, n_chars = 0, n_reads = 0, n_seq_lines = 0;
};

// The totals of the steps for texts whose chunks of kFewLines have summaries;
// false when some chunk has none.
static bool count_few(ParsePlan &P, cudaStream_t st, FastxWorkspace &ws) {
  P.n_chunks = (P.L.n_lines + kFewLines - 1) / kFewLines;
  const u64 nb = (P.n_chunks + kBlockChunks - 1) / kBlockChunks;
  ws.trans.ensure(P.n_chunks * sizeof(Trans));
  ws.entries.ensure(P.n_chunks * sizeof(Entry));
  ws.stats.ensure(32);
  Trans *t = ws.trans.get<Trans>(), *tops = nullptr;
  u64 *status = ws.stats.get<u64>();
  SBWT_CUDA(cudaMemsetAsync(status, 0, 32, st));
  few_lines_kernel<<<(unsigned)((P.n_chunks + 255) / 256), 256, 0, st>>>(P.L, P.n_chunks, t);
  if (nb > 1) {
    ws.tops.ensure(nb * sizeof(Trans));
    tops = ws.tops.get<Trans>();
    trans_totals_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(t, P.n_chunks, tops);
    trans_tops_kernel<<<1, kScanBlock, 0, st>>>(tops, nb);
  }
  trans_apply_kernel<<<(unsigned)nb, kScanBlock, 0, st>>>(t, P.n_chunks, tops,
                                                          ws.entries.get<Entry>(), status);
  SBWT_CUDA(cudaGetLastError());
  SBWT_CUDA(cudaMemcpyAsync(ws.host, status, 32, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  if (ws.host[3]) return false;
  P.few = true;
  P.n_chars = ws.host[0];
  P.n_reads = ws.host[1];
  P.n_seq_lines = ws.host[2];
  return true;
}

ParsePlan fastx_count(const uint8_t *d_text, u64 n_bytes, cudaStream_t st, FastxWorkspace &ws) {
  ParsePlan P;
  if (n_bytes == 0) return P;
  const uint32_t lead = (uint32_t)((uintptr_t)d_text & 15);
  const u64 n_warps = (lead + n_bytes + kWarpBytes - 1) / kWarpBytes;
  ws.warp_counts.ensure((n_warps + 1) * 8);
  u64 *wc = ws.warp_counts.get<u64>();
  ws.marks.ensure(n_warps * 32 * sizeof(uint4));
  uint4 *marks = ws.marks.get<uint4>();
  nl_count_kernel<<<grid_for_warps(n_warps), 256, 0, st>>>(d_text, n_bytes, lead, wc, n_warps,
                                                           marks);
  enqueue_scan(wc, n_warps, ws, st);
  SBWT_CUDA(cudaMemcpyAsync(ws.host, wc + n_warps, 8, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaMemcpyAsync(ws.host + 1, d_text + n_bytes - 1, 1, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  const u64 n_nl = ws.host[0];
  const uint8_t last = *reinterpret_cast<const uint8_t *>(ws.host + 1);
  ws.nl.ensure(std::max<u64>(n_nl, 1) * 8);
  nl_write_kernel<<<grid_for_warps(n_warps), 256, 0, st>>>(d_text, n_bytes, lead, wc, n_warps,
                                                            marks, ws.nl.get<u64>());
  SBWT_CUDA(cudaGetLastError());
  P.L = Lines{d_text, n_bytes, ws.nl.get<u64>(), n_nl, n_nl + (last != '\n' ? 1 : 0)};
  if (count_few(P, st, ws)) return P;
  P.n_chunks = (P.L.n_lines + kChunkLines - 1) / kChunkLines;
  ws.roles.ensure(P.L.n_lines + 8);
  ws.chunks.ensure(std::max<u64>(P.n_chunks, 1) * sizeof(ChunkInfo));
  ws.chars_tot.ensure((P.n_chunks + 1) * 8);
  ws.hdr_tot.ensure((P.n_chunks + 1) * 8);
  uint8_t *roles = ws.roles.get<uint8_t>();
  ChunkInfo *ci = ws.chunks.get<ChunkInfo>();
  u64 *ct = ws.chars_tot.get<u64>(), *ht = ws.hdr_tot.get<u64>();
  roles_kernel<<<grid_for_warps(P.n_chunks), 256, 0, st>>>(P.L, roles, ci, P.n_chunks);
  fixup_kernel<<<1, 32, 0, st>>>(P.L, roles, ci, P.n_chunks);
  chunk_totals_kernel<<<grid_for_warps(P.n_chunks), 256, 0, st>>>(P.L, roles, ci, P.n_chunks,
                                                                    ct, ht);
  enqueue_scan(ct, P.n_chunks, ws, st);
  enqueue_scan(ht, P.n_chunks, ws, st);
  SBWT_CUDA(cudaMemcpyAsync(ws.host, ct + P.n_chunks, 8, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaMemcpyAsync(ws.host + 1, ht + P.n_chunks, 8, cudaMemcpyDeviceToHost, st));
  SBWT_CUDA(cudaStreamSynchronize(st));
  P.n_chars = ws.host[0];
  P.n_reads = ws.host[1];
  return P;
}

void fastx_emit(const ParsePlan &P, uint8_t *d_chars, u64 *d_ends, cudaStream_t st,
                FastxWorkspace &ws) {
  if (P.n_chunks == 0) return;
  if (!P.few) {
    u64 *ct = ws.chars_tot.get<u64>(), *ht = ws.hdr_tot.get<u64>();
    emit_kernel<<<grid_for_warps(P.n_chunks), 256, 0, st>>>(
        P.L, ws.roles.get<uint8_t>(), ws.chunks.get<ChunkInfo>(), P.n_chunks, ct, ht, d_chars,
        d_ends);
    if (P.n_reads) set_u64_kernel<<<1, 1, 0, st>>>(d_ends + P.n_reads - 1, ct + P.n_chunks);
    SBWT_CUDA(cudaGetLastError());
    return;
  }
  ws.line_off.ensure((P.n_seq_lines + 1) * 8);
  ws.line_src.ensure((P.n_seq_lines + 1) * 8);
  u64 *off = ws.line_off.get<u64>(), *src = ws.line_src.get<u64>();
  list_lines_kernel<<<(unsigned)((P.n_chunks + 255) / 256), 256, 0, st>>>(
      P.L, P.n_chunks, ws.entries.get<Entry>(), ws.stats.get<u64>(), d_ends, off, src);
  if (P.n_chars) {
    // 8 KB per warp, less when the output does not fill the GPU's warps with it
    const u64 span = std::min<u64>(std::max<u64>(P.n_chars / (148 * 64) / 512, 1), 16) * 512;
    const uint32_t lead = (uint32_t)((uintptr_t)d_chars & 15);
    copy_lines_kernel<<<grid_for_warps((lead + P.n_chars + span - 1) / span), 256, 0, st>>>(
        P.L.text, P.L.n_bytes, off, src, P.n_seq_lines, P.n_chars, lead, (uint32_t)span, d_chars);
  }
  SBWT_CUDA(cudaGetLastError());
}

}  // namespace sbwt

using namespace sbwt;

extern "C" int sbwt_fastx_parse(const char *text, uint64_t n_bytes, char *chars,
                                uint64_t chars_capacity, uint64_t *read_ends,
                                uint64_t ends_capacity, uint64_t *n_chars, uint64_t *n_reads,
                                uint32_t flags, int device, void *stream) {
  if (!n_chars || !n_reads || (n_bytes && !text)) {
    set_last_error("null argument");
    return SBWT_E_INVALID;
  }
  return guarded([&] {
    DeviceGuard g(device);
    FastxWorkspace &ws = fastx_workspace(device);
    const bool dev = flags & SBWT_DEVICE_POINTERS;
    cudaStream_t st = dev && stream ? (cudaStream_t)stream : ws.stream;
    const uint8_t *d_text = (const uint8_t *)text;
    if (!dev) {
      ws.text.ensure(std::max<u64>(n_bytes, 1));
      if (n_bytes)
        SBWT_CUDA(cudaMemcpyAsync(ws.text.get(), text, n_bytes, cudaMemcpyHostToDevice, st));
      d_text = ws.text.get<uint8_t>();
    }
    const ParsePlan P = fastx_count(d_text, n_bytes, st, ws);
    *n_chars = P.n_chars;
    *n_reads = P.n_reads;
    if (P.n_chars > chars_capacity || P.n_reads > ends_capacity)
      throw Error(SBWT_E_CAPACITY, "chars or read ends capacity too small");
    if ((P.n_chars && !chars) || (P.n_reads && !read_ends))
      throw Error(SBWT_E_INVALID, "null output buffer");
    if (dev) {
      fastx_emit(P, (uint8_t *)chars, read_ends, st, ws);
    } else {
      ws.chars.ensure(std::max<u64>(P.n_chars, 1));
      ws.ends.ensure(std::max<u64>(P.n_reads, 1) * 8);
      fastx_emit(P, ws.chars.get<uint8_t>(), ws.ends.get<u64>(), st, ws);
      if (P.n_chars)
        SBWT_CUDA(cudaMemcpyAsync(chars, ws.chars.get(), P.n_chars, cudaMemcpyDeviceToHost, st));
      if (P.n_reads)
        SBWT_CUDA(cudaMemcpyAsync(read_ends, ws.ends.get(), P.n_reads * 8,
                                  cudaMemcpyDeviceToHost, st));
    }
    SBWT_CUDA(cudaStreamSynchronize(st));
  });
}
