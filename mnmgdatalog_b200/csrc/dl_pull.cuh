// Level-synchronous work on bit rows, shared by TC's heavy sources
// (dl_closure.cu) and SG (dl_sgrows.cu): rows in chunks of 1024 columns with
// activity tags, the list of the next level's rows, the targets with many in-edges, and
// the walk over the edges of a warp's rows.
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

// A target with more in-edges than lanes ("hub") is gathered in segments of 32
// in-edges by as many warps: one warp alone would walk them long after the
// others are done (at 256 in-edges a warp, 46 % of a level's time was that tail).
constexpr u32 PU_SEG = 32;

// Hubs: hub_at[w] = accumulator row of hub w, seg[...] = (w, first in-edge of a
// segment); found[0] = hubs, found[1] = segments.
static __global__ void pull_hubs_kernel(const u32 *__restrict__ roff, u64 n, u32 *__restrict__ hub_at,
                                        uint2 *__restrict__ seg, unsigned long long *__restrict__ found) {
    for (u64 w = (u64) blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (u64) gridDim.x * blockDim.x) {
        const u32 b = roff[w], d = roff[w + 1] - b;
        if (d <= PU_SEG) continue;
        hub_at[w] = (u32) atomicAdd(found, 1ull);
        const u32 k = (d + PU_SEG - 1) / PU_SEG;
        const unsigned long long at = atomicAdd(found + 1, (unsigned long long) k);
        for (u32 i = 0; i < k; ++i) seg[at + i] = make_uint2((u32) w, b + i * PU_SEG);
    }
}

// A warp works on K * 128 words of a row at a time: lane l holds words
// base + 128 k + 4 l .. + 3 (k < K), 16 bytes each, eight lanes to a chunk.
// Activity bit of the lane's k-th piece.
template <int K>
__device__ __forceinline__ u32 piece_bit(const PullShape &sh, u32 base, int k, u32 lane) {
    return 1u << (((base >> 5) + 4 * k + (lane >> 3)) >> sh.shift);
}

// ORs the newest words of a group of up to 32 in-neighbours (node y, activity
// a in the neighbour's lane) into acc: two neighbours' pieces in flight. The
// pieces whose bit of `need` is clear are not loaded.
template <int K>
__device__ __forceinline__ void or_neighbours(const PullShape &sh, const u32 *__restrict__ cur, u32 base, u32 y, u32 a,
                                              u32 need, u32 lane, uint4 (&acc)[K]) {
    u32 all = __ballot_sync(0xffffffffu, a != 0);
    const u32 *mine = cur + base + lane * 4;
    u32 bit[K];
#pragma unroll
    for (int k = 0; k < K; ++k) bit[k] = (need >> k) & 1u ? piece_bit<K>(sh, base, k, lane) : 0u;
    while (all) {
        uint4 v[2][K];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const u32 j = (__ffs(all) - 1) & 31;
            u32 aj = __shfl_sync(0xffffffffu, a, j);
            if (all == 0) aj = 0;
            all &= all - 1;
            const uint4 *src = reinterpret_cast<const uint4 *>(mine + (u64) __shfl_sync(0xffffffffu, y, j) * sh.words);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                v[q][k] = make_uint4(0, 0, 0, 0);
                if (aj & bit[k]) v[q][k] = __ldg(src + 32 * k);
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            acc[k].x |= v[0][k].x | v[1][k].x;
            acc[k].y |= v[0][k].y | v[1][k].y;
            acc[k].z |= v[0][k].z | v[1][k].z;
            acc[k].w |= v[0][k].w | v[1][k].w;
        }
    }
}

// Hub targets: a warp ORs the newest words of PU_SEG in-neighbours, K * 128
// words of the row, into the hub's accumulator (zero before the level).
template <int K>
__global__ void __launch_bounds__(PU_THREADS)
closure_pull_hub_kernel(PullShape sh, PullLevel st, const u32 *__restrict__ roff, const u32 *__restrict__ rval,
                        const uint2 *__restrict__ seg, u64 n_seg, const u32 *__restrict__ hub_at,
                        u32 *__restrict__ hub_acc) {
    if (st.count[st.level] == 0) return;  // the fixpoint was reached earlier
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64) gridDim.x * (PU_THREADS / 32);
    const u32 passes = (sh.words + K * 128 - 1) / (K * 128);
    for (u64 it = ((u64) blockIdx.x * PU_THREADS + threadIdx.x) / 32; it < n_seg * passes; it += warps) {
        const u32 base = (u32) (it % passes) * K * 128;
        const uint2 sg = seg[it / passes];
        if (st.todo[sg.x] == 0) continue;
        const u32 i = sg.y + lane;
        u32 y = 0, a = 0;
        if (i < roff[sg.x + 1]) {
            y = rval[i];
            const uint2 tg = st.tag[y];
            a = tg.y == st.level - 1 ? tg.x : 0u;
        }
        uint4 acc[K];
        u32 need = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            acc[k] = make_uint4(0, 0, 0, 0);
            if (base + 128 * k + lane * 4 < sh.words) need |= 1u << k;
        }
        or_neighbours<K>(sh, st.cur, base, y, a, need, lane, acc);
        u32 *dst = hub_acc + (u64) hub_at[sg.x] * sh.words + base + lane * 4;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (acc[k].x) atomicOr(dst + 128 * k, acc[k].x);
            if (acc[k].y) atomicOr(dst + 128 * k + 1, acc[k].y);
            if (acc[k].z) atomicOr(dst + 128 * k + 2, acc[k].z);
            if (acc[k].w) atomicOr(dst + 128 * k + 3, acc[k].w);
        }
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
