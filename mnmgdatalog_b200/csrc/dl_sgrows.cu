// SG on bit rows, one owner per row.
//
// sg(x, y) :- e(a, x), sg(a, b), e(b, y) (sg.cu:244-390). sg is symmetric from
// the base rule on, so with E(b) = the children of b's newest partners as a bit row,
// the new pairs of row y are
//     N(y) = OR of E(b) over y's in-neighbours b
// minus the row's known pairs, and E(y) = the children of the nodes in N(y): all
// that row y needs is its in-neighbours' rows, read as whole lines, and its
// children's scatter goes to a row in shared memory. A row has one owner (a warp,
// or a CTA for long rows), so nothing is merged between CTAs, and every new
// pair is expanded once, whatever the out-degree of its row. (The step on the matrix
// before this one, dl_bitmap.cu, expanded the pairs of a source once and folded the
// result into every child's row with an atomic per touched word of the matrix.)
// The base rule is the same step on the identity: E(x) = x's children, and N(y)
// without y itself.
//
// Measured on B200, a mesh of 22K nodes and 38K edges (2.4e8 pairs, 133
// iterations), edges and result rows on the device: 67 ms on the matrix; 17.1 ms with
// the newest pairs themselves as rows, which expands the union of the in-neighbours'
// pairs for every row (also those of nodes without children) and reads the known pairs
// only after that; 14.7 ms here.
#include "dl_closure.h"
#include "dl_pull.cuh"

namespace dl {
namespace detail {
namespace {

// has[k] bit b = node 32 k + b has out-edges (words padded to the rows' length).
__global__ void has_children_kernel(const u32 *__restrict__ off, u64 n, u64 words, u32 *__restrict__ has) {
    for (u64 k = (u64) blockIdx.x * blockDim.x + threadIdx.x; k < words; k += (u64) gridDim.x * blockDim.x) {
        u32 v = 0;
        for (u32 b = 0; b < 32; ++b) {
            const u64 x = k * 32 + b;
            if (x < n && off[x + 1] > off[x]) v |= 1u << b;
        }
        has[k] = v;
    }
}

// Level 0: the newest pair of a node x is (x, x), so its row holds x's children;
// tagged, so that the children of x get on the first list. cols[i] = i (all
// ones past n).
__global__ void sg_identity_kernel(PullShape sh, PullLevel st, const u32 *__restrict__ off,
                                   const u32 *__restrict__ val, u32 *__restrict__ cols) {
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    for (u64 x = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32; x < (u64) sh.words * 32; x += warps) {
        if (lane == 0) cols[x] = x < sh.n ? (u32) x : EMPTY;
        if (x >= sh.n || off[x + 1] == off[x]) continue;
        const u32 b = off[x], e = off[x + 1];
        u32 act = 0;
        for (u32 k = b + lane; k < e; k += 32) act |= 1u << ((val[k] >> 10) >> sh.shift);
        act = __reduce_or_sync(0xffffffffu, act);
        u32 *row = st.nxt + x * sh.words;
        for (u32 mm = act; mm; mm &= mm - 1) {
            const u32 w0 = ((u32) (__ffs(mm) - 1) << sh.shift) * 32, w1 = min(sh.words, w0 + (32u << sh.shift));
            for (u32 k = w0 + lane; k < w1; k += 32) row[k] = 0;
        }
        __syncwarp();
        for (u32 k = b + lane; k < e; k += 32) atomicOr(&row[val[k] >> 5], 1u << (val[k] & 31));
        if (lane == 0) st.tag_next[x] = make_uint2(act, st.level);
    }
}

struct SgTeam {
    u32 item;            // the team's place in the list
    u32 touched;         // activity bits of the chunks its children fell into
};

constexpr u32 SG_QUEUE = 512;  // new pairs a warp holds before it expands them

// Per-warp part of a team's shared memory.
struct SgWarp {
    u32 queue[SG_QUEUE];
    u32 wbeg[32], wpre[32];
};

// The children of the queued nodes into the row; returns the activity bits of the
// chunks this lane's fell into. Not inlined: the kernel calls it in three places,
// and with three copies of the walk it stalled on instruction fetches two issue
// slots out of three.
__device__ __noinline__ u32 sg_expand(SgWarp &mw, u32 qn, u32 *row, const u32 *__restrict__ off,
                                      const u32 *__restrict__ val, u32 shift) {
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt(), le = lane == 31 ? ~0u : (2u << lane) - 1;
    u32 mine = 0;
    __syncwarp();
    u32 nbeg = 0, nend = 0;
    auto fetch = [&](u32 q0) {  // one batch ahead
        nbeg = nend = 0;
        if (q0 + lane < qn) {
            const u32 a = mw.queue[q0 + lane];
            nbeg = __ldg(off + a);
            nend = __ldg(off + a + 1);
        }
    };
    fetch(0);
    for (u32 q0 = 0; q0 < qn; q0 += 32) {
        const u32 beg = nbeg, deg = nend - nbeg;
        fetch(q0 + 32);
        auto put = [&](u32 x) {
            atomicOr(&row[x >> 5], 1u << (x & 31));
            mine |= 1u << ((x >> 10) >> shift);
        };
        // a few children each: every lane walks its own node's (a mesh's six at most
        // cost less than sharing them out); else 32 of the batch's children at a time
        const u32 most = __reduce_max_sync(0xffffffffu, deg);
        if (most <= 8) {
            for (u32 k = 0; k < most; k += 4) {
                u32 x[4];
#pragma unroll
                for (u32 j = 0; j < 4; ++j)
                    if (k + j < deg) x[j] = __ldg(val + beg + k + j);
#pragma unroll
                for (u32 j = 0; j < 4; ++j)
                    if (k + j < deg) put(x[j]);
            }
        } else {
            walk_rows(mw.wbeg, mw.wpre, beg, deg, val, lane, lt, le, 0xFFFFFFFFu, [&](u32 x, bool have) -> bool {
                if (have) put(x);
                return true;
            });
        }
    }
    __syncwarp();
    return mine;
}

// One level: the new pairs of every row in the list, a team of NW warps per row
// (TEAMS teams to a CTA, each with its row in shared memory). The warps take
// the active chunks four at a time: OR of the in-neighbours' words and the row's known
// pairs, whose difference goes to a queue across chunks, so that the expansion
// runs on full batches of 32 pairs; their children are ORed into the shared row,
// which leaves chunk by chunk. Bound by latency and instructions (at the mesh's
// fullest level 60 % of the issue slots, 8200 instructions for a row of 960 new
// pairs in 22 chunks), not by the lines. Measured on the mesh above in the form before
// this one: chunk by chunk with batches a quarter full 26 ms, the walk in three
// copies 24 ms, 40 warps an SM at 48 registers 17.8 ms against 17.1 for 32 at 64, six
// or eight chunks in flight 17.5 and 20 ms (spills), two in-neighbours at a time
// 16.4; in this one, one prefix sum over four chunks 15.2 against 14.7 ms.
// HUBS: rows with more than PU_SEG in-neighbours have the OR of their words in hub_acc
// already (closure_pull_hub_kernel), which is cleared here. (A warp alone with thousands
// of in-neighbours held up every level: 20K nodes, 40K edges, a third of them into four
// nodes: 56 ms, on the matrix 28; now 5.2.)
template <int NW, int TEAMS, bool HUBS>
__global__ void __launch_bounds__(NW * TEAMS * 32, 1024 / (NW * TEAMS * 32))
sg_rows_kernel(PullShape sh, PullLevel st, const u32 *__restrict__ off, const u32 *__restrict__ val,
               const u32 *__restrict__ roff, const u32 *__restrict__ rval, const u32 *__restrict__ has,
               const u32 *__restrict__ hub_at, u32 *__restrict__ hub_acc, u32 *__restrict__ m, int base_rule,
               unsigned long long *__restrict__ fetch) {
    extern __shared__ __align__(16) u32 smem[];
    static_assert(NW == 1 || TEAMS == 1, "a team is a warp or the CTA");
    const u64 n_list = st.count[st.level];
    if (n_list == 0) return;  // the fixpoint was reached earlier
    __shared__ SgTeam teams[TEAMS];
    __shared__ SgWarp warps[NW * TEAMS];
    const u32 lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const u32 part = NW == 1 ? 0 : wid;  // the warp's number in its team
    u32 *row = smem + (NW == 1 ? wid : 0) * sh.words;
    SgTeam &team = teams[NW == 1 ? wid : 0];
    SgWarp &mw = warps[wid];
    const u32 tl = NW == 1 ? lane : threadIdx.x;  // thread of the team
    auto team_sync = [] {
        if constexpr (NW == 1) __syncwarp();
        else __syncthreads();
    };
    for (u32 k = tl; k < sh.words; k += NW * 32) row[k] = 0;
    if (tl == 0) team.touched = 0;
    u64 fresh = 0, rows = 0;
    // the next four chunks of the activity mask (EMPTY: none); gc: chunks of the lowest
    // granule already given out
    auto four = [&](u32 &mm, u32 &gc, u32 (&c)[4]) {
#pragma unroll
        for (u32 q = 0; q < 4; ++q) {
            c[q] = EMPTY;
            if (mm) {
                const u32 at = ((__ffs(mm) - 1) << sh.shift) + gc;
                if (++gc >> sh.shift) {
                    gc = 0;
                    mm &= mm - 1;
                }
                if (at < sh.words / 32) c[q] = at;
            }
        }
    };
    for (;;) {
        if (tl == 0) team.item = (u32) min(atomicAdd(fetch + st.level, 1ull), (unsigned long long) EMPTY);
        team_sync();  // the row is clear, nothing marked
        const u32 i = team.item;
        if (i >= n_list) break;
        const u32 y = st.list[i];
        const u32 act = st.todo[y];
        const u32 b = __ldg(roff + y), n = __ldg(roff + y + 1) - b;
        auto parents = [&](u32 e0, u32 &p, u32 &a) {  // 32 in-neighbours from the e0-th on and their activity
            p = a = 0;
            if (e0 + lane < n) {
                p = __ldg(rval + b + e0 + lane);
                const uint2 tg = st.tag[p];
                a = tg.y == st.level - 1 ? tg.x : 0u;
            }
        };
        const bool hub = HUBS && n > PU_SEG;
        u32 *hrow = nullptr;
        u32 y0 = 0, a0 = 0;
        if (hub) hrow = hub_acc + (u64) hub_at[y] * sh.words + lane;
        else parents(0, y0, a0);
        u32 mine = 0;  // chunks this lane's children fell into
        u32 qn = 0;    // queued new pairs
        auto drain = [&]() {
            mine |= sg_expand(mw, qn, row, off, val, sh.shift);
            qn = 0;
        };
        const bool can = __ldg(off + y + 1) > __ldg(off + y);
        u32 *mp = m + (u64) y * sh.words + lane;
        {
            u32 mm = act, gc = 0, turn = 0;
            while (mm) {
                u32 c[4];
                four(mm, gc, c);
                if (NW > 1 && turn++ % NW != part) continue;
                u32 w[4], old[4];
#pragma unroll
                for (u32 q = 0; q < 4; ++q) {
                    w[q] = old[q] = 0;
                    if (c[q] != EMPTY) old[q] = mp[c[q] * 32];
                }
                if (hub) {
#pragma unroll
                    for (u32 q = 0; q < 4; ++q) {
                        if (c[q] == EMPTY) continue;
                        w[q] = hrow[c[q] * 32];
                        hrow[c[q] * 32] = 0;
                    }
                }
                for (u32 e0 = 0; e0 < n && !hub; e0 += 32) {
                    u32 p = y0, a = a0;
                    if (e0) parents(e0, p, a);
                    // two in-neighbours at a time: eight lines in flight
                    for (u32 all = __ballot_sync(0xffffffffu, a != 0); all; all &= all - 1) {
                        const u32 j = __ffs(all) - 1;
                        all &= all - 1;
                        const u32 j2 = all ? __ffs(all) - 1 : j;
                        const u32 *src = st.cur + (u64) __shfl_sync(0xffffffffu, p, j) * sh.words + lane;
                        const u32 *src2 = st.cur + (u64) __shfl_sync(0xffffffffu, p, j2) * sh.words + lane;
                        const u32 aj = __shfl_sync(0xffffffffu, a, j);
                        const u32 aj2 = __shfl_sync(0xffffffffu, j2 == j ? 0u : a, j2);
                        u32 x[4], x2[4];
#pragma unroll
                        for (u32 q = 0; q < 4; ++q) {
                            x[q] = x2[q] = 0;
                            if (c[q] == EMPTY) continue;
                            if ((aj >> (c[q] >> sh.shift)) & 1u) x[q] = __ldg(src + c[q] * 32);
                            if ((aj2 >> (c[q] >> sh.shift)) & 1u) x2[q] = __ldg(src2 + c[q] * 32);
                        }
#pragma unroll
                        for (u32 q = 0; q < 4; ++q) w[q] |= x[q] | x2[q];
                    }
                }
#pragma unroll
                for (u32 q = 0; q < 4; ++q) {
                    if (c[q] == EMPTY) continue;
                    u32 v = w[q] & ~old[q];
                    if (base_rule && (y >> 5) == c[q] * 32 + lane) v &= ~(1u << (y & 31));  // x != y
                    if (v) mp[c[q] * 32] = old[q] | v;
                    fresh += __popc(v);
                    if (!can) continue;
                    v &= __ldg(has + c[q] * 32 + lane);  // the others have no children
                    const u32 cnt = __popc(v);
                    const u32 incl = warp_inclusive_sum(cnt);
                    const u32 total = __shfl_sync(0xffffffffu, incl, 31);
                    if (!total) continue;
                    rows += cnt;
                    if (qn + total > SG_QUEUE) drain();
                    if (total <= SG_QUEUE) {
                        for (u32 at = qn + incl - cnt; v; v &= v - 1) mw.queue[at++] = (c[q] * 32 + lane) * 32 + __ffs(v) - 1;
                        qn += total;
                    } else {  // eight lanes' words at a time
                        for (u32 g = 0; g < 4; ++g) {
                            const u32 before = g ? __shfl_sync(0xffffffffu, incl, 8 * g - 1) : 0u;
                            if ((lane >> 3) == g)
                                for (u32 at = incl - cnt - before; v; v &= v - 1)
                                    mw.queue[at++] = (c[q] * 32 + lane) * 32 + __ffs(v) - 1;
                            qn = __shfl_sync(0xffffffffu, incl, 8 * g + 7) - before;
                            drain();
                        }
                    }
                }
            }
            if (qn) drain();
        }
        u32 touched = __reduce_or_sync(0xffffffffu, mine);
        if constexpr (NW > 1) {
            if (lane == 0 && touched) atomicOr(&team.touched, touched);
            __syncthreads();  // the row is complete
            touched = team.touched;
            __syncthreads();  // every warp has read it
            if (tl == 0) team.touched = 0;
        } else {
            __syncwarp();
        }
        // the new pairs' children leave for the next level
        for (u32 mm = touched, turn = 0; mm; mm &= mm - 1) {
            const u32 c0 = (u32) (__ffs(mm) - 1) << sh.shift, c1 = min(sh.words / 32, c0 + (1u << sh.shift));
            for (u32 cc = c0; cc < c1; ++cc) {
                if (NW > 1 && turn++ % NW != part) continue;
                const u32 k = cc * 32 + lane;
                st.nxt[(u64) y * sh.words + k] = row[k];
                row[k] = 0;
            }
        }
        if (tl == 0) {
            st.todo[y] = 0;
            if (touched) st.tag_next[y] = make_uint2(touched, st.level);
        }
    }
    fresh = warp_sum(fresh);
    rows = warp_sum(rows);
    if (lane == 0) {
        if (fresh) atomicAdd(st.cnt + st.level, (unsigned long long) fresh);
        if (rows) atomicAdd(st.deg + st.level, (unsigned long long) rows);
    }
}

// Results of fewer bits than one in this many leave by the matrix's kernels (dl_bitmap.cu), which read
// whole rows; closure_rows_kernel takes a line at a time, whose first row it knows, and gains
// where the lines are full. Whole runs, by lines and by rows: 220K layered nodes, three iterations, one
// bit in 980, 18.5 / 13.0 ms; meshes of 22K nodes, one in 55 / 5.8 / 1.8, 1.37 / 1.34, 3.18 / 3.50 and
// 13.2 / 14.2; random 40K nodes, one in 119 / 31 / 9, 2.41 / 2.16, 3.17 / 3.05 and 4.52 / 4.99.
constexpr u64 SG_SPARSE = 32;
constexpr u64 SG_LEVELS = 8;  // levels launched between two host waits

// Targets with many in-neighbours (pull_hubs_kernel).
struct SgHubs {
    u64 n = 0, n_seg = 0;
    const uint2 *seg = nullptr;
    const u32 *at = nullptr;
    u32 *acc = nullptr;
};

template <int K>
void launch_hubs(Context &ctx, const PullShape &sh, const PullLevel &st, const u32 *roff, const u32 *rval,
                 const SgHubs &hubs) {
    const u64 passes = (sh.words + K * 128 - 1) / (K * 128);
    DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
              closure_pull_hub_kernel<K><<<grid_for(hubs.n_seg * passes * 32, PU_THREADS, ctx, 8), PU_THREADS, 0,
                                           ctx.stream>>>(sh, st, roff, rval, hubs.seg, hubs.n_seg, hubs.at, hubs.acc));
}

template <int NW, int TEAMS>
void launch_level(Context &ctx, const PullShape &sh, const PullLevel &st, const Csr &csr, const u32 *roff,
                  const u32 *rval, const u32 *has, const SgHubs &hubs, u32 *m, bool base) {
    const size_t smem = (size_t) TEAMS * sh.words * 4;
    if (hubs.n) {
        if (sh.words <= 128) launch_hubs<1>(ctx, sh, st, roff, rval, hubs);
        else if (sh.words <= 256) launch_hubs<2>(ctx, sh, st, roff, rval, hubs);
        else launch_hubs<3>(ctx, sh, st, roff, rval, hubs);
    }
    auto kern = hubs.n ? sg_rows_kernel<NW, TEAMS, true> : sg_rows_kernel<NW, TEAMS, false>;
    DL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int per_sm = 0;
    DL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NW * TEAMS * 32, smem));
    const u64 grid = std::min<u64>((sh.n + TEAMS - 1) / TEAMS, (u64) ctx.sm_count * std::max(per_sm, 1));
    DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
              kern<<<(unsigned) grid, NW * TEAMS * 32, smem, ctx.stream>>>(
                  sh, st, csr.off, csr.val, roff, rval, has, hubs.at, hubs.acc, m, base ? 1 : 0, st.deg + SG_LEVELS + 1));
}

bool sg_rows_run(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt,
                 PhaseTimer &pt, u64 &nfull) {
    Workspace &ws = ctx.ws;
    const u64 n = g.n_ids, words = (n + 1023) / 1024 * 32;
    const u64 bytes = n * words * 4;
    if (words * 4 + 24 * 1024 > 227 * 1024) return false;  // a row in shared memory beside the queues
    if (3 * bytes > ((u64) ctx.tune.bitmap_max_gib << 30)) return false;
    if (!ctx.room_for({{&r.bm_t, bytes}, {&ws.cl_rows[0], bytes}, {&ws.cl_rows[1], bytes}},
                      {&ws.bitmat[0], &ws.bitmat[1]}))
        return false;
    // (now, before smaller requests take the cached buffers that were counted on)
    ctx.reserve(r.bm_t, bytes);
    ctx.reserve(ws.cl_rows[0], bytes);
    ctx.reserve(ws.cl_rows[1], bytes);
    pt.mark(PH_INIT);
    PullShape sh{n, (u32) words, 0};
    while ((32u << sh.shift) < words / 32) ++sh.shift;
    const u64 *rev = edges_by_other(ctx, edges, ne, g.bits, ws.full[0], ws.full[1]);  // in-neighbours
    ctx.reserve(ws.cl_roff, (n + 1) * 4);
    ctx.reserve(ws.cl_rval, ne * 4);
    u32 *roff = ws.cl_roff.as<u32>(), *rval = ws.cl_rval.as<u32>();
    DL_LAUNCH(ctx, K_PREP, 0,
              key_offsets_kernel<u32><<<grid_for(n + 1, T256, ctx), T256, 0, ctx.stream>>>(rev, ne, g.bits, n, roff));
    DL_LAUNCH(ctx, K_PREP, 12.0 * ne,
              low_field_kernel<<<grid_for(ne, T256, ctx), T256, 0, ctx.stream>>>(rev, ne, (1ull << g.bits) - 1, rval));
    auto *found = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[44]);
    ctx.reserve(ws.cl_segs, (ne / PU_SEG * 2 + 1) * 8);  // a hub's segments are at most twice its in-edges / 32
    ctx.reserve(ws.cl_hub_at, n * 4);
    DL_CUDA(cudaMemsetAsync(found, 0, 16, ctx.stream));
    DL_LAUNCH(ctx, K_PREP, 4.0 * n,
              pull_hubs_kernel<<<grid_for(n, T256, ctx), T256, 0, ctx.stream>>>(roff, n, ws.cl_hub_at.as<u32>(),
                                                                               ws.cl_segs.as<uint2>(), found));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, found, 16, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.reserve(ws.bit_hasout, words * 4);
    u32 *has = ws.bit_hasout.as<u32>();
    DL_LAUNCH(ctx, K_PREP, 4.0 * n,
              has_children_kernel<<<grid_for(words, T256, ctx), T256, 0, ctx.stream>>>(g.csr.off, n, words, has));
    ctx.reserve(ws.cl_act, 8 * n * 4);
    ctx.reserve(r.cl_cols, words * 32 * 4);
    DL_CUDA(cudaMemsetAsync(r.bm_t.p, 0, bytes, ctx.stream));
    u32 *p = ws.cl_act.as<u32>();
    DL_CUDA(cudaMemsetAsync(p, 0xFF, 4 * n * 4, ctx.stream));       // tags: no level
    DL_CUDA(cudaMemsetAsync(p + 4 * n, 0, 2 * n * 4, ctx.stream));  // todo
    // counters of a batch of levels: list lengths (one more than levels), new
    // pairs, joinable ones, next places of the lists; two sets, the next batch's first list length is copied over
    constexpr u64 SET = 4 * (SG_LEVELS + 1);
    ctx.reserve(ws.cl_levels, 2 * SET * 8);
    u64 *sets[2] = {ws.cl_levels.as<u64>(), ws.cl_levels.as<u64>() + SET};
    DL_CUDA(cudaMemsetAsync(sets[0], 0, SET * 8, ctx.stream));
    u64 first = 1;  // first level of the batch
    int set = 0;
    auto view = [&](u64 level) {
        const u64 in = (level + 1) & 1, out = level & 1;
        PullLevel v;
        v.level = (u32) level;
        v.cur = ws.cl_rows[in].as<u32>();
        v.nxt = ws.cl_rows[out].as<u32>();
        v.tag = reinterpret_cast<uint2 *>(p + 2 * in * n);
        v.tag_next = reinterpret_cast<uint2 *>(p + 2 * out * n);
        v.todo = p + (4 + out) * n;
        v.todo_next = p + (4 + in) * n;
        v.list = p + (6 + out) * n;
        v.list_next = p + (6 + in) * n;
        v.count = reinterpret_cast<unsigned long long *>(sets[set]) - first;
        v.cnt = v.count + SG_LEVELS + 1;
        v.deg = v.cnt + SG_LEVELS + 1;
        return v;
    };
    auto push = [&](u64 level) {
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                  closure_push_kernel<<<grid_for(ne, PU_THREADS, ctx, 8), PU_THREADS, 0, ctx.stream>>>(
                      view(level), edges, ne, g.bits));
    };
    DL_LAUNCH(ctx, K_PREP, 128.0 * n,
              sg_identity_kernel<<<grid_for(words * 32 * 32, T256, ctx), T256, 0, ctx.stream>>>(
                  sh, view(0), g.csr.off, g.csr.val, r.cl_cols.as<u32>()));
    push(0);
    ctx.sync();
    SgHubs hubs{ctx.host_scalars[0], ctx.host_scalars[1], ws.cl_segs.as<uint2>(), ws.cl_hub_at.as<u32>(), nullptr};
    if (hubs.n) {
        ctx.reserve(ws.cl_hub_acc, hubs.n * words * 4);
        hubs.acc = ws.cl_hub_acc.as<u32>();
        DL_CUDA(cudaMemsetAsync(hubs.acc, 0, hubs.n * words * 4, ctx.stream));
    }
    pt.mark(PH_JOIN);
    // level 1 is the base rule, level k + 1 iteration k; level k + 1's joins are
    // level k's joinable pairs
    std::vector<u64> cnt(2, 0), joinable(2, 0);
    nfull = 0;
    for (bool done = false; !done;) {
        // (no level past the last iteration that was asked for)
        const u64 batch = opt.max_iterations > 0 ? std::min<u64>(SG_LEVELS, (u64) opt.max_iterations + 2 - first)
                                                 : SG_LEVELS;
        for (u64 level = first; level < first + batch; ++level) {
            const bool base = level == 1;
            u32 *m = r.bm_t.as<u32>();
            if (words <= 1024) launch_level<1, 4>(ctx, sh, view(level), g.csr, roff, rval, has, hubs, m, base);
            else if (words <= 4096) launch_level<4, 1>(ctx, sh, view(level), g.csr, roff, rval, has, hubs, m, base);
            else launch_level<8, 1>(ctx, sh, view(level), g.csr, roff, rval, has, hubs, m, base);
            push(level);
        }
        DL_CUDA(cudaMemsetAsync(sets[set ^ 1], 0, SET * 8, ctx.stream));
        DL_CUDA(cudaMemcpyAsync(sets[set ^ 1], sets[set] + SG_LEVELS, 8, cudaMemcpyDeviceToDevice, ctx.stream));
        u64 *hs = ctx.host_scalars;
        DL_CUDA(cudaMemcpyAsync(hs, sets[set], SET * 8, cudaMemcpyDeviceToHost, ctx.stream));
        ctx.sync();
        for (u64 k = 0; k < batch && !done; ++k) {
            const u64 level = first + k, c = hs[SG_LEVELS + 1 + k], j = hs[2 * (SG_LEVELS + 1) + k];
            nfull += c;
            ctx.prof_add_bytes(K_BITMAP_EXPAND, 8.0 * c);  // a new pair's word
            if (level == 1) {
                cnt[1] = c;
                joinable[1] = j;
                continue;
            }
            r.deltas.push_back((i64) c);
            r.joins.push_back((i64) joinable[1]);
            r.fulls.push_back((i64) nfull);
            joinable[1] = j;
            done = c == 0 || (opt.max_iterations > 0 && level - 1 >= (u64) opt.max_iterations);
        }
        first += SG_LEVELS;
        set ^= 1;
    }
    pt.mark(PH_FINAL);
    if (nfull) {
        ctx.reserve(ws.offsets, (n + 1) * 8);
        const bool sparse = nfull < n * words * 32 / SG_SPARSE;
        if (sparse) bitmat_row_counts(ctx, r.bm_t.as<u32>(), n, words, words, ws.offsets.as<u64>());
        else bit_rows_count(ctx, r, n, words, 0, g.bits, nullptr, ws.offsets.as<u64>());
        const u64 total = bit_rows_finish(ctx, r, n, words, ws.offsets.as<u64>());
        if (total != nfull)
            throw Error(DL_ERR_INTERNAL, "bit rows hold " + std::to_string(total) + " tuples, expected " +
                                             std::to_string(nfull));
        r.cl_rows = !sparse;
        r.bm_row_first = true;
    }
    r.from_bitmat = true;
    return true;
}

}  // namespace

bool sg_rows(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt, PhaseTimer &pt,
             u64 &nfull) {
    bool done = false;
    try {
        done = sg_rows_run(ctx, r, g, edges, ne, opt, pt, nfull);
    } catch (const Error &err) {
        if (err.status != DL_ERR_OUT_OF_MEMORY) throw;
    }
    if (!done) {
        r.deltas.clear();
        r.joins.clear();
        r.fulls.clear();
        r.from_bitmat = r.cl_rows = r.bm_row_first = false;
        Workspace &ws = ctx.ws;
        for (DevBuf *b : {&r.bm_t, &r.bm_first, &r.cl_cols, &r.cl_loff, &r.cl_start, &ws.cl_rows[0], &ws.cl_rows[1]})
            ctx.give_back(*b);
        nfull = 0;
    }
    return done;
}

}  // namespace detail
}  // namespace dl
