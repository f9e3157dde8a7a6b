// Device memory that the k-mer table and its filter may take.
#pragma once

#include <cstdint>

namespace sbwt {

// A quarter of what is free (`free_bytes`: before the construction of the table
// starts) beside a label of 8 bytes and a flag for each of n nodes.  The
// construction's temporaries, 36 to 40 bytes a node, are given back when it
// ends, so they do not lessen the budget; while they are held the table and a
// path cover of at most 5.5 bytes a k-mer fit beside them from 53 free bytes a
// node on (41.5 n + (free - 9 n) / 4 <= free), and an index with a k-mer per
// node needs 137 for a table of at least 32 bytes a k-mer.
inline uint64_t kmer_table_budget(uint64_t free_bytes, uint64_t n) {
  return free_bytes / 9 > n ? (free_bytes - 9 * n) / 4 : 0;
}

}  // namespace sbwt
