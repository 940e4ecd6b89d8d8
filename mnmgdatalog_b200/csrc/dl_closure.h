// Transitive closure as one breadth-first search per source (dl_closure.cu).
#pragma once

#include "dl_engine_detail.h"

namespace dl {
namespace detail {

// Levels a searched source may have; level d of a source = its targets at
// distance d (Delta_{d-1}: level 1 is the edge relation).
constexpr u32 CL_LEVELS = 4096;

// What the searches of one call found.
struct ClosureLight {
    u64 n_words = 0;      // (z << bits) | x words of the finished sources, unsorted, in ws.jbuf[0]
    u32 levels = 0;       // largest level of a finished source
    u64 n_heavy = 0;      // sources left over: ranks as u64 words, unsorted, in ws.cl_heavy
};

// Searches from every source in [lo, hi). Level counts go to
// cnt[instance * stride + d] (and the sum of the out-degrees of the level's
// targets to deg[...] when not null), instance k being the last one whose first
// rank inst_lo[k] is at most the source (one instance when inst_lo is null);
// [k0, k1): the sources' edges and all edges that can be reached from them;
// stride: above the levels an instance can have, or CL_LEVELS + 1. Sources
// whose reach or work outgrows the searches' shared memory are left over for
// the caller. max_level: 0 = no limit.
ClosureLight closure_search(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const u64 *inst_lo, u64 n_inst,
                            u64 k0, u64 k1, u64 stride, u64 max_level, u64 *cnt, u64 *deg);

// The words of a search's finished sources (all sources of the call, nothing
// appended since) sorted; ranks below 2^used_bits. The words of a source are equal
// below `bits`, so that lining the sources up replaces the passes over that field:
// a scan and one copy for about half the passes. Result in ws.jbuf[0] or [1].
u64 *closure_order(Context &ctx, u64 n_sources, u64 n_words, int bits, int used_bits);

// The closure of `h` heavy sources (ascending ranks `src`, device) over ranks
// [0, n) as bit rows: bit c of row z of `t` is set when source c reaches z.
// `cols`: rank of every column (padded to whole words with all ones), followed
// by room for n more words.
struct ClosureHeavy {
    u64 h = 0;
    u64 words = 0;                // words of a row (a multiple of 32)
    std::vector<u64> cnt, deg;    // per level (index d, [0] unused)
};
// Device bytes closure_pull needs for h sources over n ranks.
u64 closure_pull_bytes(u64 n, u64 h);
ClosureHeavy closure_pull(Context &ctx, const Csr &csr, const u64 *edges, u64 ne, int bits, u64 n, const u64 *src,
                          u64 h, u64 max_level, DevBuf &t, DevBuf &cols);

// The result of a run as bit rows (r.bm_t, r.cl_cols, the `n_light` light pairs
// in r.words): rows of every target (counts) and of its chunks (r.cl_start), the
// light pairs' place (r.cl_loff).
void bit_rows_count(Context &ctx, Run &r, u64 n, u64 words, u64 n_light, int bits, const u32 *place, u64 *counts);
// Then the first row of every target from the counts; returns the number of rows.
u64 bit_rows_finish(Context &ctx, Run &r, u64 n, u64 words, const u64 *counts);

// The pairs of heavy sources `src` (ascending, host) of one instance with ranks
// [lo, hi) of the CSR: appended as (z << bits) | x words to ws.jbuf[0] (n_words
// of it are kept and counted on), their levels added to cnt (index d, grown as
// needed).
void closure_heavy_words(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const std::vector<u64> &src,
                         u64 max_level, std::vector<u64> &cnt, u64 &n_words);

// SG as bit rows (dl_sgrows.cu) over the CSR and its sorted edge words; false
// when the rows do not fit.
bool sg_rows(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt, PhaseTimer &pt,
             u64 &nfull);

// single_join (dl_selfjoin.cu): rows (x, z) with x -> b -> z for some b, over the
// in-neighbour CSR (off[z]: the y with y -> z), as bit rows; `total`: join rows
// before dedup. False (nothing done) when the bit rows are not worth it or do
// not fit; the join and the sort of its output are the better form then.
bool self_join_rows(Context &ctx, Run &r, const Csr &in, u64 total, PhaseTimer &pt, u64 &rows);
// Edge words by one field, ascending, as words by the other, in a or b. Those of equal second field
// come in the order of the first already, so half the passes do, and no duplicates are left to
// drop (single_join of 1M rows of ids that are ranked by a sort, 1.44 -> 1.28 ms for the whole run;
// packing and sorting the rows a second time had made it slower than the two sorts of
// the rows side by side, 1.29; TC of a tree of 4M nodes, three children each, 13.4 -> 12.3
// with it and the row writer's shorter walk).
u64 *edges_by_other(Context &ctx, const u64 *edges, u64 ne, int bits, DevBuf &a, DevBuf &b);
// Sum over the edges y -> z of y's in-degree: the join rows of the self-join.
u64 self_join_total(Context &ctx, const Csr &in);

// TC of one graph by searches and pulls; false when its buffers do not fit
// (the workspace's join buffers are overwritten then, the CSR is not).
// `edges`: sorted (x, y) words.
bool tc_closure(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt,
                PhaseTimer &pt, u64 &nfull);

}  // namespace detail

// Result rows of targets [z0, z1) of a closure run into `out` (all rows' base).
void closure_extract_rows(Context &ctx, const Run &r, int32_t *out, u64 z0, u64 z1);

}  // namespace dl
