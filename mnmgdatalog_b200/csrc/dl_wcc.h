// WCC as level-synchronous min-label propagation (dl_wcc.cu).
#pragma once

#include "dl_engine_detail.h"

namespace dl {
namespace detail {

// The iterations of every instance: its |delta| per iteration, up to its own stop.
struct WccRun {
    std::vector<std::vector<i64>> deltas;
    std::vector<i64> joins;  // edges walked per iteration, all instances together
};

// Propagates labels over ranks [lo, hi) of a symmetric CSR whose lists ascend.
// Instance k holds the ranks from inst_lo[k] (ascending, inst_lo[0] = lo) up to the
// next one's, n_ids[k] of them. Final labels go to label[r - lo].
WccRun wcc_propagate(Context &ctx, const Csr &csr, u64 lo, u64 hi, const std::vector<u64> &inst_lo,
                     const std::vector<u64> &n_ids, int stop_rule, int max_iterations, u32 *label);

// counts[label[i] - base] += 1 (a warp's equal labels in one atomic).
void wcc_label_counts(Context &ctx, const u32 *label, u64 n, u32 base, u32 *counts);

}  // namespace detail
}  // namespace dl
