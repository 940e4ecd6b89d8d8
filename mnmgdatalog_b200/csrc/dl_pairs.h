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
    bool complete = false;   // the last level found nothing (or max_levels ended the search)
    u64 n_words() const { return bound.empty() ? 0 : bound.back(); }
};

// Out-edges of ranks [lo, hi): the largest degree and the ranks that have any.
struct PairDegrees {
    u32 most = 0;
    u64 sources = 0;
    // A pair's expansion is shared by 32 lanes at most.
    bool fits() const;
};
PairDegrees pair_degrees(Context &ctx, const Csr &csr, u64 lo, u64 hi);
// Whether sorted runs are the faster form for a session's instances of `n_ids` nodes
// each, with `edges` between them (see dl_pairs.cu).
bool pair_search_outrun(const PairDegrees &d, u64 edges, const std::vector<u64> &n_ids);
// The search from the base rule of ranks [lo, hi) of the CSR; words (x << bits) | y
// in ws.jbuf[0], unsorted. Stops after level max_levels (0: at the fixpoint). The
// search is not complete, and its last level may lack words,
//  * with most != 0 (the caller has another form for many pairs): once more than
//    `most` words are found or the first set is outgrown;
//  * once the list and the set would need more than `limit` bytes, or more than half
//    of the free memory.
PairSearch pair_search(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, u64 max_levels, u64 most, u64 limit);
// counts[instance * levels + k] = words of level k of each instance (instance of
// a word: the last one whose first rank is at most its key rank).
void pair_level_counts(Context &ctx, const PairSearch &ps, int bits, const u64 *inst_lo, u64 n_inst, u64 *counts);

}  // namespace detail
}  // namespace dl
