// Level-synchronous work on bit rows, shared by TC's heavy sources
// (dl_closure.cu) and SG (dl_sgrows.cu): rows in chunks of 1024 columns with
// activity tags, the list of the next level's rows, and the walk over the edges
// of a warp's rows.
#pragma once

#include "dl_engine_detail.h"

namespace dl {
namespace detail {
namespace {

constexpr u32 EMPTY = 0xFFFFFFFFu;  // ranks are below 2^32 - 1
constexpr int PU_THREADS = 256;

// Walks the edge targets of up to 32 rows (beg, deg of this lane's row; deg 0:
// none) in windows of 32: f(w, have) per window, all lanes; f returns false
// to stop. Returns the rows' edges. A window's rows are the bits of a
// start mask, a word's row the number of rows started up to its position.
template <class F>
__device__ __forceinline__ u32 walk_rows(u32 *wbeg, u32 *wpre, u32 beg, u32 deg, const u32 *__restrict__ val,
                                         u32 lane, u32 lt, u32 le, u32 limit, F f) {
    const u32 nz = __ballot_sync(0xffffffffu, deg != 0);
    if (!nz) return 0;
    const u32 incl = warp_inclusive_sum(deg);
    const u32 total = __shfl_sync(0xffffffffu, incl, 31);
    if (total > limit) return total;
    const u32 rk = __popc(nz & lt);
    if (deg) {
        wbeg[rk] = beg;
        wpre[rk] = incl - deg;
    }
    __syncwarp();
    const u32 nrows = __popc(nz);
    const u32 cb = lane < nrows ? wbeg[lane] : 0u;
    const u32 pre = lane < nrows ? wpre[lane] : 0xFFFFFFFFu;
    __syncwarp();
    int base = -1;  // last row started before the window
    auto load = [&](u32 i0) -> u32 {
        const u32 st = (pre - i0) < 32u ? 1u << (pre - i0) : 0u;
        const u32 starts = __reduce_or_sync(0xffffffffu, st);
        const int o = base + __popc(starts & le);
        base += __popc(starts);
        const u32 ob = __shfl_sync(0xffffffffu, cb, o);
        const u32 op = __shfl_sync(0xffffffffu, pre, o);
        return i0 + lane < total ? __ldg(val + ob + (i0 + lane - op)) : 0u;
    };
    u32 w = load(0);
    for (u32 i0 = 0; i0 < total; i0 += 32) {
        const u32 wn = i0 + 32 < total ? load(i0 + 32) : 0u;  // the next window's load is in flight
        if (!f(w, i0 + lane < total)) break;
        w = wn;
    }
    return total;
}

// Bit rows: chunks of 1024 columns (a 128-byte line), 2^shift
// of which share one activity bit, so that a row's activity is one word
// whatever the number of columns.
struct PullShape {
    u64 n;      // targets
    u32 words;  // words of a row
    u32 shift;
};

// One level's view of the state: row y of `cur` is valid when tag[y] is
// (activity, level - 1); todo[w] = activity of w's in-neighbours (zero: w is not
// in the list).
struct PullLevel {
    u32 level;
    const u32 *cur;
    u32 *nxt;
    const uint2 *tag;
    uint2 *tag_next;
    u32 *todo, *todo_next;
    const u32 *list;
    u32 *list_next;
    unsigned long long *count;  // [level]: targets in the level's list
    unsigned long long *cnt;    // [level]: new pairs
    unsigned long long *deg;    // [level]: sum of their targets' out-degrees
};

// Puts the targets of the newly active nodes on the next level's list: a
// thread per edge (x, y), sorted by x, so a node's out-degree does not matter
// (a warp per active node spent half a level on the few nodes with thousands
// of out-edges).
static __global__ void __launch_bounds__(PU_THREADS)
closure_push_kernel(PullLevel st, const u64 *__restrict__ edges, u64 ne, int bits) {
    if (st.level && st.count[st.level] == 0) return;  // the fixpoint was reached earlier
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u64 mask = (1ull << bits) - 1;
    for (u64 k0 = (u64) blockIdx.x * PU_THREADS + (threadIdx.x & ~31u); k0 < ne; k0 += (u64) gridDim.x * PU_THREADS) {
        bool fresh = false;
        u32 y = 0;
        if (k0 + lane < ne) {
            const u64 e = __ldg(edges + k0 + lane);
            const uint2 tg = st.tag_next[e >> bits];
            if (tg.y == st.level) {
                y = (u32) (e & mask);
                fresh = atomicOr(&st.todo_next[y], tg.x) == 0u;
            }
        }
        const u32 fm = __ballot_sync(0xffffffffu, fresh);
        if (!fm) continue;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(st.count + st.level + 1, (unsigned long long) __popc(fm));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (fresh) st.list_next[at + __popc(fm & lt)] = y;
    }
}

// off[k] = first word whose key (word >> bits) is at least k, k in [0, n].
template <class T>
__global__ void key_offsets_kernel(const u64 *__restrict__ w, u64 nw, int bits, u64 n, T *__restrict__ off) {
    for (u64 k = (u64) blockIdx.x * blockDim.x + threadIdx.x; k <= n; k += (u64) gridDim.x * blockDim.x) {
        const u64 target = k << bits;
        u64 l = 0, h = nw;
        while (l < h) {
            const u64 m = (l + h) >> 1;
            if (w[m] < target) l = m + 1;
            else h = m;
        }
        off[k] = (T) l;
    }
}

static __global__ void low_field_kernel(const u64 *__restrict__ w, u64 n, u64 mask, u32 *__restrict__ out) {
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x)
        out[i] = (u32) (w[i] & mask);
}

// Edge words (x, y) -> (y, x).
static __global__ void pull_swap_kernel(const u64 *__restrict__ e, u64 ne, int bits, u64 *__restrict__ out) {
    const u64 mask = (1ull << bits) - 1;
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += (u64) gridDim.x * blockDim.x) {
        const u64 w = e[i];
        out[i] = ((w & mask) << bits) | (w >> bits);
    }
}

}  // namespace
}  // namespace detail
}  // namespace dl
