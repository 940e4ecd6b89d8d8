// SG as a breadth-first search over pairs (dl_pairs.cu).
#pragma once

#include "dl_engine_detail.h"

namespace dl {
namespace detail {

// Pairs of one search, in the order found: level 0 = the base rule's, level k =
// iteration k's new ones.
struct PairSearch {
    std::vector<u64> bound;  // level k holds words [bound[k], bound[k + 1])
    std::vector<u64> rows;   // rows[k]: pairs of level k whose two nodes have out-edges
    // With the joins counted, of level k's join in two steps (x, b), then (x, y):
    std::vector<u64> first;   // rows of the first one
    std::vector<u64> middle;  // distinct ones
    std::vector<u64> second;  // rows of the second one
    bool complete = false;   // the last level found nothing (or max_levels ended the search)
    u64 n_words() const { return bound.empty() ? 0 : bound.back(); }
};

// Out-edges of ranks [lo, hi).
struct PairDegrees {
    u64 most = 0;     // the largest
    u64 edges = 0;    // all
    u64 squares = 0;  // sum of their squares: the rows of the base rule's join
    // A pair's expansion is shared by 32 lanes at most.
    bool fits() const;
    // Mean out-edges of an edge's source (1 more than a node's mean where degrees are random).
    double of_sources() const { return edges ? (double) squares / (double) edges : 0.0; }
};
PairDegrees pair_degrees(Context &ctx, const Csr &csr, u64 lo, u64 hi);
// Whether sorted runs are the faster form for graphs of `n_ids` nodes each (see dl_pairs.cu).
bool pair_search_outrun(const PairDegrees &d, const std::vector<u64> &n_ids);

struct PairOptions {
    u64 max_levels = 0;    // the level to stop after (0: at the fixpoint)
    bool handover = false; // stop where a matrix is the faster form (see dl_pairs.cu)
    u64 limit = ~0ull;     // bytes of the list and the set
    bool joins = false;    // count the rows of the joins in two steps, as the sorted runs do
    PairDegrees deg;       // of the ranks, for `handover` and `joins`
};
// The search from the base rule of ranks [lo, hi) of the CSR; words (x << bits) | y
// in ws.jbuf[0], unsorted. It is not complete, and its last level may lack words, where
// it stopped for `handover`, for `limit` or half of the free memory, or because a level's first
// join did not fit the table that counts it.
PairSearch pair_search(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const PairOptions &opt);
// counts[instance * levels + k] = words of level k of each instance (instance of
// a word: the last one whose first rank is at most its key rank).
void pair_level_counts(Context &ctx, const PairSearch &ps, int bits, const u64 *inst_lo, u64 n_inst, u64 *counts);

}  // namespace detail
}  // namespace dl
