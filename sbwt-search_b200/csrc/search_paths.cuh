// Read search over the path cover (path_cover.cu): included by index.cu after
// ReadsView.
#pragma once

namespace sbwt {

// Read search of an index with its path cover and L-mer filter (the automatic
// choice as resolve_kernel_mode says; the conditions of the walks kernel, whose
// tiles, work queue and -1/-2 rules it shares).  A lane resolves runs of k-mers instead of k-mers:
//   P_SEED : the k-mer at pos by one table lookup: its position on the cover;
//   P_EXT  : the read's next chars against the cover's, 32 at a time: as long
//            as they agree (and the path does not break) the k-mers are the
//            next positions of the cover;
//   P_MISS : a k-mer that is absent (the table does not have it, or its first
//            k - 1 chars end a k-mer without another edge): L-mer filter
//            probes prove the k-mers around a read error absent;
//   P_FILT : a k-mer not looked up yet, after proven absent ones: probed first;
//   P_SYNC : past a char that disagreed with the path, its k-mers proven
//            absent: the path is tried again k positions on (a substitution
//            leaves the read on it), which spares the table lookup.
// Each iteration yields at most one run per lane (of cover positions, of -1,
// or of -2); the warp writes the runs, one run of consecutive results per
// store, kRunsInFlight runs' loads in flight.
//
// A run is exact: consecutive positions without a break are joined by an edge
// of the SBWT whose char is the later one's, and a k-mer has one node; an
// L-mer the filter rejects is in no k-mer of the SBWT.
//
// What bounds it: on a large index DRAM, by random 64-byte accesses: about 24
// bytes a k-mer (8 of results, 7 of nodes in runs that are not aligned, 3 each
// of table, cover and filter), on a small one the instructions (~3 per k-mer
// and warp against ~17 of the walks kernel, which takes one dependent random
// sector per k-mer besides).  Kernel time against the walks or k-mers kernel:
// 420 M k-mers of ragged reads on a 115 M-node index 2.83 against 7.20 ms, 140
// M k-mers with 5 % substitutions 1.45 against 4.29 ms, 12 M k-mers on a 2
// M-node index 92 against 147 us.
enum : uint32_t { P_NEW = 0, P_SEED = 1, P_EXT = 2, P_SYNC = 3, P_FILT = 4, P_MISS = 5,
                  P_DONE = 6 };

// 256-thread blocks per SM the register budget targets (64 registers; the
// grid is one wave).  More blocks (and 4 runs in flight) are slower on a large
// index, whose random DRAM accesses then queue: 3.30 ms with 5 against 2.96 ms
// with 4 and 2.79 ms with 3 on 420 M k-mers; on an index that stays in L2 it
// is 88 us with 5, 92 us with 4 and 93 us with 3 (12 M k-mers).
constexpr int kPathsBlocksPerSm = 4;

// 32 chars from offset j (0 <= j < 32) of the 64-char window (hi, lo).
__device__ __forceinline__ uint64_t window_at(uint64_t hi, uint64_t lo, uint32_t j) {
  return (hi << (2 * j)) | ((lo >> 1) >> (63 - 2 * j));
}

__device__ __forceinline__ PathEntry load_path_entry(const PathEntry *p) {
  const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
  return PathEntry{((unsigned long long)v.y << 32) | v.x, v.z, v.w};
}

constexpr int kRunsInFlight = 8;
constexpr int kRunSlots = 32 + kRunsInFlight;  // a list is padded to whole batches
constexpr uint32_t kTileReserve = 32;  // tiles a warp takes from the queue at a time

// O32: 32-bit results into rv.out32.
template <bool COUNT, int KC, bool O32>
__global__ void __launch_bounds__(256, kPathsBlocksPerSm)
    search_paths_kernel(SbwtView s, ReadsView rv, const uint64_t *__restrict__ tile_start,
                        unsigned long long *counters) {
  using I = uint32_t;
  constexpr I NONE = ~I(0);
  constexpr I INVALID = NONE - 1;
  // two lists of runs per warp (slot, position or marker, length, high word
  // of a marker's results): one being made, one being written
  __shared__ uint4 sh_run[8][2][kRunSlots];
  const uint32_t k = KC ? (uint32_t)KC : s.k;
  const uint32_t L = s.lmer_len, D = k - L;  // an absent L-mer rules out D + 1 k-mers
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  uint4 *runs = sh_run[threadIdx.x >> 5][0], *last = sh_run[threadIdx.x >> 5][1];
  const PathEntry *const reads = rv.entries;
  const I n_kmers = (I)(rv.n_kmers_dev ? *rv.n_kmers_dev : rv.n_kmers);
  const I tsize = (I)rv.tile;
  const I n_tiles = (n_kmers + tsize - 1) / tsize;
  const I base = (I)rv.base;
  const I out_cap = (I)min(rv.out_capacity, (uint64_t)NONE);
  const uint64_t pol_last = l2_policy_evict_last(), pol_first = l2_policy_evict_first();
  uint64_t n_table = 0, n_entry = 0, n_filter = 0, n_iter = 0, n_known = 0, n_found = 0,
           n_runs = 0;
  // the warp's tiles [res, res_end): the first ones by its number, then
  // kTileReserve at a time from the queue
  const I warps = gridDim.x * (blockDim.x >> 5);
  I res = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kTileReserve;
  I res_end = min(res + kTileReserve, n_tiles);
  const I queued = warps * kTileReserve;  // tiles handed out by number
  // slot, pos: the next k-mer; send: end of its read or tile; tend: of the tile
  I slot = 0, send = 0, tend = 0, r = 0, pos = 0;
  I pp = 0;               // cover position of k-mer pos - 1 (P_EXT)
  I alt = NONE, apos = 0; // cover position whose char disagreed; the k-mer start past it
  uint32_t mode = P_NEW;
  // Writing the last iteration's runs: the nodes of a batch are loaded before
  // the state machine waits for a load of its own and stored after it, so
  // their round trips overlap.
  uint32_t n_last = 0, val[kRunsInFlight];
  auto fetch = [&](uint32_t i) {
    if (i >= n_last) return;
#pragma unroll
    for (int u = 0; u < kRunsInFlight; ++u) {
      const uint4 q = last[i + u];
      val[u] = q.y;
      if (lane < q.z && q.y < INVALID) val[u] = load_u32_nc(s.path_node + (q.y + lane));
    }
  };
  auto store = [&](uint32_t i) {
    if (i >= n_last) return;
#pragma unroll
    for (int u = 0; u < kRunsInFlight; ++u) {
      const uint4 q = last[i + u];
      if (lane >= q.z) continue;
      if (O32)
        __stcs(rv.out32 + (q.x + lane), val[u]);
      else
        __stcs(reinterpret_cast<uint2 *>(rv.out) + (q.x + lane), make_uint2(val[u], q.w));
    }
  };
  while (true) {
    // ---- tiles: lanes in order take consecutive ones of the warp's
    const bool need = mode == P_NEW && slot >= tend;
    const unsigned nm = __ballot_sync(0xFFFFFFFFu, need);
    I tile = NONE;
    if (nm) {
      const I want = __popc(nm), t = res + __popc(nm & below);
      if (need && t < res_end) tile = t;
      const I got = res < res_end ? min(want, res_end - res) : 0;
      res += got;
      if (got < want) {
        unsigned long long qb = n_tiles;
        if (queued < n_tiles && res < n_tiles) {
          if (lane == 0) qb = atomicAdd(rv.queue, (unsigned long long)kTileReserve) + queued;
          qb = __shfl_sync(0xFFFFFFFFu, qb, 0);
        }
        res = (I)min(qb, (unsigned long long)n_tiles);
        res_end = (I)min(qb + kTileReserve, (unsigned long long)n_tiles);
        const I t2 = res + __popc(nm & below) - got;
        if (need && tile == NONE) {
          if (t2 < res_end)
            tile = t2;
          else
            mode = P_DONE;
        }
        res = min(res + want - got, res_end);
      }
      if (__all_sync(0xFFFFFFFFu, mode == P_DONE)) break;
    }
    fetch(0);
    if (mode == P_NEW) {
      if (tile != NONE) {
        const uint64_t e = __ldg(tile_start + tile);
        r = (I)e;
        pos = (I)(e >> 32);
        slot = tile * tsize;
        tend = min(slot + tsize, n_kmers);
      } else {  // the next read
        pos = (I)__ldg(rv.ends + r) - base;
        ++r;
      }
      I kend = (I)__ldg(rv.kmer_off + r + 1);
      if (kend == slot) {  // reads without k-mers
        do {
          kend = (I)__ldg(rv.kmer_off + (++r) + 1);
        } while (kend == slot);
        pos = (I)__ldg(rv.ends + r - 1) - base;
      }
      send = min(tend, kend);
      alt = NONE;
      mode = P_SEED;
    }
    // ---- the chars: 64 from pos (P_EXT: 32 from the next k-mer's last char)
    uint64_t hi = 0, lo = 0, inv = 0;
    if (mode != P_DONE) {
      const I at = mode == P_EXT ? pos + k - 1 : pos;
      const PathEntry *e = reads + (at >> 5);
      const uint32_t off = at & 31;
      const PathEntry a = load_path_entry(e), b = load_path_entry(e + 1);
      hi = window_at(a.chars, b.chars, off);
      inv = __funnelshift_r(a.brk, b.brk, off);
      if (mode != P_EXT) {
        const PathEntry c = load_path_entry(e + 2);
        lo = window_at(b.chars, c.chars, off);
        inv |= (uint64_t)__funnelshift_r(b.brk, c.brk, off) << 32;
      }
    }
    store(0);
    fetch(kRunsInFlight);
    I run_slot = slot, run_at = NONE;
    uint32_t run_n = 0;
    bool filt = mode == P_FILT || mode == P_MISS;
    const bool sync = mode == P_SYNC;
    // ---- invalid chars in the k-mer: -2 up to the last of them
    if (mode == P_SEED || filt) {
      const uint64_t m = inv & low_mask(k);
      if (m) {
        run_n = min(min(64u - (uint32_t)__clzll(m), send - slot), 32u);
        run_at = INVALID;
        if (COUNT) n_known += run_n;
        filt = false;
        mode = P_SEED;
      }
    }
    // ---- the k-mer's table lookup
    if (mode == P_SEED && run_n == 0) {
      const uint64_t key = hi >> (64 - 2 * k);
      uint64_t hs = kmer_table_bucket(key, s.kmer_table_mask);
      I found = NONE;
      while (true) {
        const Block A =
            load_block_hint(reinterpret_cast<const Block *>(s.kmer_table + 2 * hs), pol_first);
        if (COUNT) ++n_table;
        if (A.w0 == key) {
          found = (I)(A.w1 >> 32);
          break;
        }
        if (A.w2 == key) {
          found = (I)(A.w3 >> 32);
          break;
        }
        if (A.w0 == ~0ULL || A.w2 == ~0ULL) break;  // an empty slot: absent
        hs = (hs + 2) & s.kmer_table_mask;
      }
      if (found != NONE) {
        pp = run_at = found;
        run_n = 1;
        alt = NONE;
        mode = P_EXT;
        hi = window_at(hi, lo, k);  // the chars after the k-mer
        inv >>= k;
      } else {
        mode = P_MISS;
        filt = true;
      }
    }
    store(kRunsInFlight);
    fetch(2 * kRunsInFlight);
    // ---- filter probes of a k-mer that may be or is absent
    if (filt) {
      // an error at the k-mer's last char (where a path shows it) is in the
      // k-mer's last L-mer and in the L-mer that starts there; one further
      // left is looked for at two smaller offsets
      const bool at_end = alt != NONE && apos == pos + k;
      const uint32_t o[4] = {D >> 2, D >> 1, D, min(2 * D + 1, k - 1)};
      uint32_t z[4], cov = mode == P_MISS ? 1u : 0u;
      uint2 f[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f[i] = make_uint2(~0u, ~0u);
        z[i] = 0;
        if (i >= 2 || !at_end) {
          z[i] = lmer_hash(window_at(hi, lo, o[i]) >> (64 - 2 * L));
          f[i] = load_uint2_hint(s.lmer_filter + lmer_word(z[i], s.lmer_words), pol_last);
          if (COUNT) ++n_filter;
        }
      }
      bool hit = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint2 b = lmer_bits(z[i]);
        if (((f[i].x & b.x) != b.x || (f[i].y & b.y) != b.y) && o[i] <= cov + D) {
          cov = o[i] + 1;
          hit = true;
        }
      }
      // not past the read or tile, nor to a k-mer with an invalid char
      const uint64_t m = inv >> k;
      if (m) cov = min(cov, (uint32_t)__ffsll((long long)m));
      run_n = min(min(cov, send - slot), 32u);
      mode = hit ? P_FILT : P_SEED;
    }
    if (mode != P_EXT) {  // (P_SYNC: run_n is 0)
      slot += run_n;
      pos += run_n;
      if (run_n) mode = slot == send ? P_NEW : (alt != NONE && pos == apos ? P_SYNC : mode);
    }
    // ---- the cover's next chars
    if (mode == P_EXT || sync) {
      const I b = (sync ? alt : pp) + 1;
      const PathEntry e0 = load_path_entry(s.path_entry + (b >> 5));
      const PathEntry e1 = load_path_entry(s.path_entry + (b >> 5) + 1);
      if (COUNT) n_entry += 2;
      const uint32_t off = b & 31;
      const uint64_t x = hi ^ window_at(e0.chars, e1.chars, off);
      const uint32_t brk = __funnelshift_r(e0.brk, e1.brk, off);
      const uint64_t mm = (x | (x >> 1)) & 0x5555555555555555ULL;
      // first char that disagrees or is invalid; first break (32: none)
      const uint32_t stop = min((uint32_t)__clzll(mm) >> 1,
                                (uint32_t)__clz(__brev((uint32_t)inv)));
      const uint32_t end = (uint32_t)__clz(__brev(brk));
      const uint32_t m = min(stop, end);
      uint32_t n;
      if (sync) {
        n = m >= k ? min(m - k + 1, send - slot) : 0;
        run_at = alt + k;
        pp = run_at + n - 1;
        alt = NONE;
        mode = n ? P_EXT : P_SEED;
      } else {
        if (run_n == 0) run_at = b;
        const uint32_t lim = min(send - slot, 32u) - run_n;
        n = min(m, lim);
        pp += n;
        if (m < lim) {
          mode = P_SEED;
          if (stop < end) {  // a char that disagrees (no break up to it)
            alt = pp + 1;
            apos = pos + run_n + n + k;
            // the k-mer before it has no other edge: absent
            const uint32_t more = __funnelshift_r(e0.branch, e1.branch, off) | (uint32_t)inv;
            if (!((more >> m) & 1u)) mode = P_MISS;
          }
        }
      }
      run_n += n;
      slot += run_n;
      pos += run_n;
      if (slot == send) mode = P_NEW;
    }
    store(2 * kRunsInFlight);
    for (uint32_t i = 3 * kRunsInFlight; i < n_last; i += kRunsInFlight) {
      fetch(i);
      store(i);
    }
    // ---- this iteration's runs
    if (COUNT) {
      n_iter += lane == 0;
      n_runs += run_n != 0;
      n_found += run_at < INVALID ? run_n : 0;
    }
    run_n = run_slot < out_cap ? min(run_n, out_cap - run_slot) : 0;
    const unsigned rm = __ballot_sync(0xFFFFFFFFu, run_n != 0);
    n_last = __popc(rm);
    if (run_n)
      runs[__popc(rm & below)] = make_uint4(run_slot, run_at, run_n, run_at < INVALID ? 0u : ~0u);
    if (lane < kRunsInFlight) runs[n_last + lane].z = 0;
    uint4 *const t = runs;
    runs = last;
    last = t;
    __syncwarp();
  }
  for (uint32_t i = 0; i < n_last; i += kRunsInFlight) {
    fetch(i);
    store(i);
  }
  if (COUNT) {
    atomicAdd(counters + 0, (unsigned long long)n_table);
    atomicAdd(counters + 1, (unsigned long long)n_entry);   // cover entries
    atomicAdd(counters + 2, (unsigned long long)((n_found + 7) / 8));  // node sectors
    atomicAdd(counters + 3, (unsigned long long)n_filter);
    atomicAdd(counters + 4, (unsigned long long)n_iter);
    atomicAdd(counters + 5, (unsigned long long)n_runs);
    atomicAdd(counters + 6, (unsigned long long)n_known);
    atomicAdd(counters + 7, (unsigned long long)n_found);
    atomicAdd(counters + 9, (unsigned long long)n_filter);  // filter words
    atomicAdd(counters + 12, (unsigned long long)n_table);  // table lookups
  }
}

// The reference seam of an index with its k-mer table (k <= 31): a k-mer is a
// table lookup (32 bytes) instead of a presearch entry and k - p steps.
// Positions usually come from reads, so consecutive entries are consecutive
// positions: a warp takes 32 entries, and in kLeadRounds rounds the first
// unresolved entry of every stretch of consecutive positions is looked up and
// the entries behind it follow the path cover as far as their chars agree
// with it; what is left is looked up entry by entry, all together.
// What bounds it: the lookups' random DRAM sectors and the round trips of a
// round.  4 M positions on a 20 M-node index, a third of them absent: whole
// call 392 us with presearch and steps, 98 us here (two leading rounds 105 us,
// none 115 us; one round is the best or near it with no and with many absent
// k-mers).  32 registers, so that 64 warps per SM hide the round trips: 100 us
// against 107 us at 40.
constexpr int kLeadRounds = 1;
__global__ void __launch_bounds__(256, 8) search_positions_table_kernel(
    SbwtView s, const uint64_t *__restrict__ packed, uint64_t n_chars_cap,
    const uint64_t *__restrict__ positions, uint64_t n, uint64_t *__restrict__ out,
    uint32_t move_to_key, uint32_t *err) {
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  const uint32_t k = s.k, lane = threadIdx.x & 31;
  const uint64_t pol_first = l2_policy_evict_first();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t0 = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ULL; t0 < n;
       t0 += step) {
    const uint64_t t = t0 + lane;
    const uint64_t pos = t < n ? __ldg(positions + t) : 0;
    uint64_t v = SBWT_NOT_FOUND;
    const bool in = t < n && pos <= n_chars_cap && n_chars_cap - pos >= k;
    if (t < n && !in) atomicOr(err, 2u);  // a k-mer past bit_seqs
    bool open = in;
    const uint64_t before = __shfl_up_sync(FULL, pos, 1);
    const bool joined = lane > 0 && pos == before + 1;
    for (int round = s.path_node ? 0 : kLeadRounds; round <= kLeadRounds; ++round) {
      const unsigned om = __ballot_sync(FULL, open);
      if (!om) break;
      const bool last_round = round == kLeadRounds;
      // a leader: an open entry that does not continue an open one
      const bool lead = open && (last_round || !joined || !((om >> (lane - 1)) & 1u));
      const unsigned lm = __ballot_sync(FULL, lead);
      // open entries that join on behind this leader
      const unsigned stop = ~(om & ~lm) & ~((2u << lane) - 1u);
      const uint32_t behind = lead ? (stop ? (uint32_t)__ffs(stop) - 1u : 32u) - lane - 1 : 0;
      uint32_t at = ~0u, follow = 0;
      if (lead) {
        const uint64_t w = pos >> 5;
        const uint32_t off = (uint32_t)(pos & 31);
        uint64_t key = __ldg(packed + w) << (2 * off);
        if (off + k > 32) key |= __ldg(packed + w + 1) >> (64 - 2 * off);
        key >>= 64 - 2 * k;
        uint64_t hs = kmer_table_bucket(key, s.kmer_table_mask);
        while (true) {
          const Block A =
              load_block_hint(reinterpret_cast<const Block *>(s.kmer_table + 2 * hs), pol_first);
          if (A.w0 == key || A.w2 == key) {
            const uint64_t value = A.w0 == key ? A.w1 : A.w3;
            v = value & s.node_mask;
            at = (uint32_t)(value >> 32);
            break;
          }
          if (A.w0 == ~0ULL || A.w2 == ~0ULL) break;  // an empty slot: absent
          hs = (hs + 2) & s.kmer_table_mask;
        }
        open = false;
        if (behind && v != SBWT_NOT_FOUND) {
          // the chars of the entries behind (their words are inside bit_seqs)
          const uint64_t c = pos + k, cw = c >> 5;
          const uint32_t co = (uint32_t)(c & 31);
          uint64_t x = __ldg(packed + cw) << (2 * co);
          if (co + behind > 32) x |= __ldg(packed + cw + 1) >> (64 - 2 * co);
          const uint32_t b = at + 1, bo = b & 31;
          const PathEntry e0 = load_path_entry(s.path_entry + (b >> 5));
          const PathEntry e1 = load_path_entry(s.path_entry + (b >> 5) + 1);
          x ^= window_at(e0.chars, e1.chars, bo);
          const uint64_t mm = (x | (x >> 1)) & 0x5555555555555555ULL;
          const uint32_t brk = __funnelshift_r(e0.brk, e1.brk, bo);
          follow = min(min((uint32_t)__clzll(mm) >> 1, (uint32_t)__clz(__brev(brk))), behind);
        }
      }
      if (last_round) break;
      // entries behind a leader take its next positions
      const unsigned mine = lm & ((2u << lane) - 1u);
      const int q = mine ? 31 - __clz(mine) : 0;
      const uint32_t q_at = __shfl_sync(FULL, at, q), q_follow = __shfl_sync(FULL, follow, q);
      if (open && mine && lane - q <= q_follow) {
        v = __ldg(s.path_node + q_at + (lane - q));
        open = false;
      }
    }
    if (t < n) {
      if (move_to_key && v != SBWT_NOT_FOUND) v = key_walk(s, v, err);
      __stcs(out + t, (unsigned long long)v);
    }
  }
}

}  // namespace sbwt
