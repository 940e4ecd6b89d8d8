// WCC: min-label propagation from the changed nodes (wcc.cu:255-387).
//
// The reference's iteration joins the changed nodes' labels with the edges and
// keeps the smallest label per node. An iteration reads the labels as they were
// before it, so two label arrays take turns: iteration k lowers array k & 1, and
// a node that changed in iteration k - 1 has its label of then in the other one,
// where iteration k does not write. (A node's label is the smaller of its two
// entries.) That leaves one launch per iteration for the walk over the changed
// nodes' edges and one for the long lists, with the stop rule evaluated on the
// device: iterations are launched eight at a time between two host waits.
// The first iteration needs no walk: a node's smallest neighbour is the first
// entry of its ascending list.
//
// Bound by launches and host waits on small graphs: an iteration moves 36 bytes
// per edge of the changed nodes. Measured on B200 against four launches and two host
// waits per iteration (count, scan, balanced emit, rebuild): 20K edges from and
// to host memory 0.93 -> 0.53 ms for the whole run, 1.05M edges on the device 2.22 ->
// 1.28, 48 instances of 1K to 200K edges in one union 11.3 -> 3.7
// (they iterate on the device alone, not step by step).
#include "dl_wcc.h"
#include "dl_pull.cuh"

namespace dl {
namespace detail {
namespace {

constexpr int WC_THREADS = 256;
constexpr int WC_WARPS = WC_THREADS / 32;
constexpr u32 WC_LONG = 128;   // longer lists are cut into pieces of this many edges for as many warps
constexpr u32 WC_TAKE = 4;     // nodes a warp takes at least
constexpr u64 WC_LEVELS = 8;   // iterations launched between two host waits

struct WccState {
    u64 lo;                      // first rank; the arrays below start there
    u32 *lab[2];
    u32 *tag;                    // last iteration that changed the node
    u32 *list[2];                // ranks changed in an iteration, by its parity
    uint4 *piece;                // pieces of long lists: first edge, edges, label
    unsigned long long *pieces;  // their number [iteration - batch]
    unsigned long long *cnt;     // changed nodes [iteration - batch]
    unsigned long long *join;    // edges walked [iteration - batch]
    u32 *icnt;                   // changed nodes per instance [(iteration - batch) * n_inst + instance]
    const u64 *inst_lo;
    u32 n_inst;
    u32 *iprev;                  // per instance: changed nodes of the iteration before
    u32 *istop;                  // per instance: the iteration after which it stopped (0: running)
    u32 *stop;                   // no instance runs any more
    u32 *done;                   // blocks of the current launch that are through
};

__device__ __forceinline__ u32 wcc_instance(const WccState &st, u64 r) {
    if (st.n_inst == 1) return 0;
    u32 a = 0, b = st.n_inst;
    while (a < b) {
        const u32 m = (a + b) >> 1;
        if (st.inst_lo[m] <= r) a = m + 1;
        else b = m;
    }
    return a - 1;
}

// A warp's lowered ranks on their way to the iteration's list: 32 at a time, since
// one atomic per window of edges on the list's length would be the longest queue.
struct WccOut {
    u32 *buf;  // 64 words of shared memory
    u32 held;
};

__device__ __forceinline__ void wcc_flush(const WccState &st, u32 level, u32 at, WccOut &o, u32 n, u32 lane) {
    const bool have = lane < n;
    const u32 r = have ? o.buf[lane] : 0u;
    unsigned long long p = 0;
    if (lane == 0) p = atomicAdd(st.cnt + at, (unsigned long long) n);
    p = __shfl_sync(0xffffffffu, p, 0) + lane;
    if (have) st.list[level & 1][p] = r;
    if (st.n_inst > 1) {
        const u32 inst = have ? wcc_instance(st, r) : EMPTY;
        const u32 same = __match_any_sync(0xffffffffu, inst);
        if (have && lane == (u32) __ffs(same) - 1) atomicAdd(st.icnt + (u64) at * st.n_inst + inst, __popc(same));
    }
}

// Ranks lowered in iteration `level` by this warp's lanes (all lanes call).
__device__ __forceinline__ void wcc_append(const WccState &st, u32 level, u32 at, WccOut &o, u32 r, bool fresh, u32 lane,
                                           u32 lt) {
    const u32 fm = __ballot_sync(0xffffffffu, fresh);
    if (!fm) return;
    if (fresh) o.buf[o.held + __popc(fm & lt)] = r;
    o.held += __popc(fm);
    __syncwarp();
    if (o.held < 32) return;
    wcc_flush(st, level, at, o, 32, lane);
    o.held -= 32;
    const u32 x = lane < o.held ? o.buf[32 + lane] : 0u;
    __syncwarp();
    if (lane < o.held) o.buf[lane] = x;
    __syncwarp();
}

__device__ __forceinline__ void wcc_finish(const WccState &st, u32 level, u32 at, WccOut &o, u32 lane) {
    if (o.held) wcc_flush(st, level, at, o, o.held, lane);
}

// Iteration 1.
__global__ void __launch_bounds__(WC_THREADS)
wcc_first_kernel(WccState st, const u32 *__restrict__ off, const u32 *__restrict__ val, u64 hi) {
    __shared__ u32 buf[WC_WARPS][64];
    WccOut o{buf[threadIdx.x >> 5], 0};
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u64 step = (u64) gridDim.x * WC_THREADS;
    for (u64 r0 = st.lo + (u64) blockIdx.x * WC_THREADS + (threadIdx.x & ~31u); r0 < hi; r0 += step) {
        const u64 r = r0 + lane;
        bool low = false;
        if (r < hi) {
            const u32 b = off[r];
            u32 m = (u32) r;
            if (off[r + 1] > b) m = min(m, val[b]);
            low = m < (u32) r;
            st.lab[0][r - st.lo] = (u32) r;
            st.lab[1][r - st.lo] = m;
            st.tag[r - st.lo] = low ? 1u : 0u;
        }
        wcc_append(st, 1, 0, o, (u32) r, low, lane, lt);
    }
    wcc_finish(st, 1, 0, o, lane);
}

// Edge targets w of changed nodes with label l: lower array level & 1.
__device__ __forceinline__ void wcc_lower(const WccState &st, u32 level, u32 at, WccOut &o, u32 w, u32 l, bool have,
                                          u32 lane, u32 lt) {
    bool fresh = false;
    if (have) {
        const u64 i = w - st.lo;
        if (l < __ldcg(&st.lab[(level + 1) & 1][i])) {
            u32 *p = &st.lab[level & 1][i];
            if (l < *reinterpret_cast<volatile u32 *>(p)) {
                const u32 old = atomicMin(p, l);
                fresh = l < old && atomicExch(&st.tag[i], level) != level;
            }
        }
    }
    wcc_append(st, level, at, o, w, fresh, lane, lt);
}

// Iteration `level` (2 and up; `at` = its place in the batch's counters; `n_prev`
// = where the number of nodes changed before it is): a warp takes 4 to 32 of them, so
// that all warps have some, and walks their edges 32 at a time; long lists go to the
// next launch in pieces. (Lists of up to 1024 edges in takes of 32 left single warps
// with thousands of edges: 1.22 ms of 1.92 on 1.05M edges of skewed degrees.)
__global__ void __launch_bounds__(WC_THREADS)
wcc_level_kernel(WccState st, const u32 *__restrict__ off, const u32 *__restrict__ val, u32 level, u32 at,
                 const unsigned long long *__restrict__ n_prev) {
    if (*st.stop) return;
    __shared__ u32 wbeg[WC_WARPS][32], wpre[WC_WARPS][32], wlab[WC_WARPS][32], buf[WC_WARPS][64];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 lt = lanemask_lt(), le = lane == 31 ? ~0u : (2u << lane) - 1;
    const u64 n = *n_prev;
    const u64 warps = (u64) gridDim.x * WC_WARPS;
    const u32 take = (u32) min((u64) 32, max((u64) WC_TAKE, (n + warps - 1) / warps));
    WccOut o{buf[warp], 0};
    u64 walked = 0;
    for (u64 g = ((u64) blockIdx.x * WC_WARPS + warp) * take; g < n; g += warps * take) {
        u32 beg = 0, deg = 0, l = 0;
        if (lane < take && g + lane < n) {
            const u32 v = st.list[(level + 1) & 1][g + lane];
            if (st.n_inst == 1 || st.istop[wcc_instance(st, v)] == 0) {
                l = st.lab[(level + 1) & 1][v - st.lo];
                beg = __ldg(off + v);
                deg = __ldg(off + v + 1) - beg;
                walked += deg;
            }
        }
        const bool cut = deg > WC_LONG;
        if (__any_sync(0xffffffffu, cut)) {
            if (cut) {
                const u32 k = (deg + WC_LONG - 1) / WC_LONG;
                const unsigned long long p = atomicAdd(st.pieces + at, (unsigned long long) k);
                for (u32 i = 0; i < k; ++i)
                    st.piece[p + i] = make_uint4(beg + i * WC_LONG, min(WC_LONG, deg - i * WC_LONG), l, 0u);
                deg = 0;
            }
        }
        const u32 nz = __ballot_sync(0xffffffffu, deg != 0);
        if (!nz) continue;
        const u32 incl = warp_inclusive_sum(deg);
        const u32 total = __shfl_sync(0xffffffffu, incl, 31);
        const u32 rk = __popc(nz & lt);
        if (deg) {
            wbeg[warp][rk] = beg;
            wpre[warp][rk] = incl - deg;
            wlab[warp][rk] = l;
        }
        __syncwarp();
        const u32 rows = __popc(nz);
        const u32 cb = lane < rows ? wbeg[warp][lane] : 0u;
        const u32 pre = lane < rows ? wpre[warp][lane] : EMPTY;
        const u32 cl = lane < rows ? wlab[warp][lane] : 0u;
        __syncwarp();
        int base = -1;  // last list started before the window
        u32 nl = 0;     // label of the loaded window's words
        auto load = [&](u32 i0) -> u32 {
            const u32 start = (pre - i0) < 32u ? 1u << (pre - i0) : 0u;
            const u32 starts = __reduce_or_sync(0xffffffffu, start);
            const int row = base + __popc(starts & le);
            base += __popc(starts);
            const u32 ob = __shfl_sync(0xffffffffu, cb, row), op = __shfl_sync(0xffffffffu, pre, row);
            nl = __shfl_sync(0xffffffffu, cl, row);
            return i0 + lane < total ? __ldg(val + ob + (i0 + lane - op)) : 0u;
        };
        u32 w = load(0), wl = nl;
        for (u32 i0 = 0; i0 < total; i0 += 32) {
            const u32 wn = i0 + 32 < total ? load(i0 + 32) : 0u;
            wcc_lower(st, level, at, o, w, wl, i0 + lane < total, lane, lt);
            w = wn;
            wl = nl;
        }
    }
    wcc_finish(st, level, at, o, lane);
    walked = warp_sum(walked);
    if (lane == 0 && walked) atomicAdd(st.join + at, (unsigned long long) walked);
}

// The pieces of the iteration's long lists, a warp each; then the last block
// applies the stop rule to every running instance: the reference's
// (wcc.cu:366-383), which compares an iteration's |delta| with the one before, or
// the fixpoint.
__global__ void __launch_bounds__(WC_THREADS)
wcc_close_kernel(WccState st, const u32 *__restrict__ val, u32 level, u32 at, int fixpoint, u32 max_iterations) {
    if (*st.stop) return;
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u64 n = st.pieces[at];
    const u64 warps = (u64) gridDim.x * WC_WARPS;
    __shared__ u32 buf[WC_WARPS][64];
    WccOut o{buf[threadIdx.x >> 5], 0};
    for (u64 i = ((u64) blockIdx.x * WC_THREADS + threadIdx.x) / 32; i < n; i += warps) {
        const uint4 p = st.piece[i];
        u32 w[WC_LONG / 32];
#pragma unroll
        for (u32 q = 0; q < WC_LONG / 32; ++q) w[q] = q * 32 + lane < p.y ? __ldg(val + p.x + q * 32 + lane) : 0u;
#pragma unroll
        for (u32 q = 0; q < WC_LONG / 32; ++q) wcc_lower(st, level, at, o, w[q], p.z, q * 32 + lane < p.y, lane, lt);
    }
    wcc_finish(st, level, at, o, lane);
    __shared__ u32 last, running;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(st.done, 1u) == gridDim.x - 1;
        running = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (u32 k = threadIdx.x; k < st.n_inst; k += WC_THREADS) {
        if (st.istop[k]) continue;
        const u32 c = st.n_inst == 1 ? (u32) *reinterpret_cast<volatile unsigned long long *>(st.cnt + at)
                                     : *reinterpret_cast<volatile u32 *>(st.icnt + (u64) at * st.n_inst + k);
        bool end = fixpoint ? c == 0 : c == st.iprev[k];
        if (max_iterations && level >= max_iterations) end = true;
        st.iprev[k] = c;
        if (end) st.istop[k] = level;
        else running = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *st.done = 0;
        if (!running) *st.stop = 1;
    }
}

__global__ void wcc_final_kernel(const u32 *__restrict__ a, const u32 *__restrict__ b, u64 n, u32 *__restrict__ label) {
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x)
        label[i] = min(a[i], b[i]);
}

__global__ void wcc_label_counts_kernel(const u32 *__restrict__ label, u64 n, u32 base, u32 *__restrict__ counts) {
    const u32 lane = threadIdx.x & 31;
    const u64 step = (u64) gridDim.x * blockDim.x;
    for (u64 i0 = (u64) blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < n; i0 += step) {
        const bool have = i0 + lane < n;
        const u32 l = have ? label[i0 + lane] : EMPTY;
        const u32 same = __match_any_sync(0xffffffffu, l);
        if (have && lane == (u32) __ffs(same) - 1) atomicAdd(counts + (l - base), (u32) __popc(same));
    }
}

}  // namespace

void wcc_label_counts(Context &ctx, const u32 *label, u64 n, u32 base, u32 *counts) {
    DL_LAUNCH(ctx, K_PREP, 4.0 * n,
              wcc_label_counts_kernel<<<grid_for(n, T256, ctx, 8), T256, 0, ctx.stream>>>(label, n, base, counts));
}

WccRun wcc_propagate(Context &ctx, const Csr &csr, u64 lo, u64 hi, const std::vector<u64> &inst_lo,
                     const std::vector<u64> &n_ids, int stop_rule, int max_iterations, u32 *label) {
    Workspace &ws = ctx.ws;
    WccRun run;
    const u64 n = hi - lo, ni = inst_lo.size();
    run.deltas.resize(ni);
    // labels, tags and lists of the ranks; the pieces of the long lists
    ctx.reserve(ws.wcc_flag, 5 * n * 4);
    ctx.reserve(ws.wcc_next, (csr.n_vals / WC_LONG * 2 + 1) * 16);  // a long list's pieces are at most twice its edges / WC_LONG
    // counters: per batch [pieces, changed, walked][WC_LEVELS + 1], then per-instance ones
    const u64 head = 3 * (WC_LEVELS + 1) + 4, per = (WC_LEVELS * ni + 1) / 2, inst_words = ni + ni;
    const u64 bytes = (head + per + inst_words + ni) * 8;
    ctx.reserve(ws.offsets, bytes);
    u64 *c = ws.offsets.as<u64>();
    WccState st;
    u32 *p = ws.wcc_flag.as<u32>();
    st.lo = lo;
    st.lab[0] = p;
    st.lab[1] = p + n;
    st.tag = p + 2 * n;
    st.list[0] = p + 3 * n;
    st.list[1] = p + 4 * n;
    st.piece = ws.wcc_next.as<uint4>();
    st.pieces = reinterpret_cast<unsigned long long *>(c);
    st.cnt = st.pieces + WC_LEVELS + 1;
    st.join = st.cnt + WC_LEVELS + 1;
    st.stop = reinterpret_cast<u32 *>(c + 3 * (WC_LEVELS + 1));
    st.done = st.stop + 2;
    st.icnt = reinterpret_cast<u32 *>(c + head);
    st.n_inst = (u32) ni;
    u64 *dlo = c + head + per;
    st.inst_lo = dlo;
    st.iprev = reinterpret_cast<u32 *>(dlo + ni);
    st.istop = st.iprev + ni;
    DL_CUDA(cudaMemsetAsync(c, 0, bytes, ctx.stream));
    std::vector<u32> prev(ni);
    for (u64 k = 0; k < ni; ++k) prev[k] = (u32) n_ids[k];
    DL_CUDA(cudaMemcpyAsync(dlo, inst_lo.data(), ni * 8, cudaMemcpyHostToDevice, ctx.stream));
    DL_CUDA(cudaMemcpyAsync(st.iprev, prev.data(), ni * 4, cudaMemcpyHostToDevice, ctx.stream));
    const int fix = stop_rule == DL_WCC_STOP_FIXPOINT;
    const u32 cap = max_iterations > 0 ? (u32) max_iterations : 0u;
    std::vector<bool> over(ni, false);
    u64 live = ni;
    // the previous batch's last |delta| (the list it left) sits in slot WC_LEVELS
    std::vector<u32> got(WC_LEVELS * ni);
    for (u32 first = 1; live; first += WC_LEVELS) {
        for (u32 k = 0; k < WC_LEVELS; ++k) {
            const u32 level = first + k;
            if (level == 1) {
                DL_LAUNCH(ctx, K_WCC_PROPAGATE, 20.0 * n,
                          wcc_first_kernel<<<grid_for(n, WC_THREADS, ctx, 8), WC_THREADS, 0, ctx.stream>>>(
                              st, csr.off, csr.val, hi));
            } else {
                DL_LAUNCH(ctx, K_WCC_PROPAGATE, 0,
                          wcc_level_kernel<<<grid_for(n * 32 / WC_TAKE, WC_THREADS, ctx, 8), WC_THREADS, 0, ctx.stream>>>(
                              st, csr.off, csr.val, level, k, k ? st.cnt + k - 1 : st.cnt + WC_LEVELS));
            }
            DL_LAUNCH(ctx, K_WCC_PROPAGATE, 0,
                      wcc_close_kernel<<<grid_for(std::max<u64>(csr.n_vals / WC_LONG, 1) * 32, WC_THREADS, ctx, 8),
                                         WC_THREADS, 0, ctx.stream>>>(st, csr.val, level, k, fix, cap));
        }
        u64 *hs = ctx.host_scalars;
        DL_CUDA(cudaMemcpyAsync(hs, st.cnt, 2 * (WC_LEVELS + 1) * 8, cudaMemcpyDeviceToHost, ctx.stream));
        if (ni > 1)
            DL_CUDA(cudaMemcpyAsync(got.data(), st.icnt, WC_LEVELS * ni * 4, cudaMemcpyDeviceToHost, ctx.stream));
        // the next batch: counters cleared, the last list's length kept
        DL_CUDA(cudaMemcpyAsync(st.cnt + WC_LEVELS, st.cnt + WC_LEVELS - 1, 8, cudaMemcpyDeviceToDevice, ctx.stream));
        DL_CUDA(cudaMemsetAsync(st.pieces, 0, (WC_LEVELS + 1) * 8, ctx.stream));
        DL_CUDA(cudaMemsetAsync(st.cnt, 0, WC_LEVELS * 8, ctx.stream));
        DL_CUDA(cudaMemsetAsync(st.join, 0, (WC_LEVELS + 1) * 8, ctx.stream));
        DL_CUDA(cudaMemsetAsync(st.icnt, 0, WC_LEVELS * ni * 4, ctx.stream));
        ctx.sync();
        for (u32 k = 0; k < WC_LEVELS && live; ++k) {
            run.joins.push_back(first + k == 1 ? (i64) csr.n_vals : (i64) hs[WC_LEVELS + 1 + k]);
            ctx.prof_add_bytes(K_WCC_PROPAGATE, 36.0 * run.joins.back());
            for (u64 i = 0; i < ni; ++i) {
                if (over[i]) continue;
                const u32 d = ni == 1 ? (u32) hs[k] : got[k * ni + i];
                const bool end = (fix ? d == 0 : d == prev[i]) || (cap && first + k >= cap);
                run.deltas[i].push_back((i64) d);
                prev[i] = d;
                if (end) {
                    over[i] = true;
                    --live;
                }
            }
        }
    }
    DL_LAUNCH(ctx, K_PREP, 12.0 * n,
              wcc_final_kernel<<<grid_for(n, T256, ctx), T256, 0, ctx.stream>>>(st.lab[0], st.lab[1], n, label));
    return run;
}

}  // namespace detail
}  // namespace dl
