// SG as a breadth-first search over pairs.
//
// sg(x, y) :- e(a, x), sg(a, b), e(b, y) (sg.cu:244-390): an iteration's new
// pairs are the children pairs of the last one's that were not seen before. The
// pairs of sparse graphs are few, so the search keeps them as a list in the order
// found (an iteration's delta is a range of it) and an open-addressing set of
// their words, which stays in L2: one launch per iteration, levels launched
// eight at a time without a host wait, and one sort of the list at the end.
// The base rule sg(x, y) :- e(p, x), e(p, y), x != y is the same expansion of the
// pairs (p, p).
//
// Measured on B200 against the bit matrix stepped by one launch per iteration:
// lattice of 494K edges (1.5M pairs, 32 iterations, a 28 GB matrix) 41 -> 1.5 ms;
// 5K edges from and to host memory 1.15 -> 0.6 ms. Against the union of 32
// instances on the sorted runs (1K-100K edges, host rows) 22 -> 6.6 ms, a
// third of it the host's waits and copies.
#include "dl_pairs.h"
#include "dl_scan.cuh"

namespace dl {
namespace detail {
namespace {

constexpr int PS_THREADS = 256;
constexpr u64 FREE = ~0ull;         // never a word: ranks are below 2^32 - 1
constexpr u32 PS_DEGREE = 64;       // largest out-degree: a pair has at most 4096 children
constexpr u64 PS_LEVELS = 8;        // levels launched between two host waits
constexpr u64 PS_SLOTS = 1 << 20;   // smallest set; 148 SMs x 64 warps x 32 words in flight fit half of it

struct PairState {
    u64 *list;                       // words in the order found
    u64 cap;                         // words it holds
    u64 *set;                        // open-addressing set, mask + 1 slots
    u64 mask;
    unsigned long long *count;       // words found (may pass cap: the surplus was not stored)
    unsigned long long *bound;       // bound[k]: first word of level k
    unsigned long long *rows;        // rows[k]: pairs of level k with children
    u32 *done;                       // blocks of the current launch that are through
    // The joins in two steps (PairOptions::joins)
    u64 *mid;                        // set of a level's (x, b), at most as many slots as `set`
    u64 most;                        // largest out-degree
    unsigned long long *mids;        // words in it
    unsigned long long *over;        // they passed half of the slots in some level
    unsigned long long *first, *middle, *second;  // as in PairSearch
};

__device__ __forceinline__ u64 pair_slot(u64 w, u64 mask) {
    // splitmix64's finalizer (Steele, Lea, Flood): structured words spread evenly
    w ^= w >> 30;
    w *= 0xbf58476d1ce4e5b9ull;
    w ^= w >> 27;
    w *= 0x94d049bb133111ebull;
    w ^= w >> 31;
    return w & mask;
}

// Adds w to the set; true when it was not there. The set is never full: the
// list's capacity is half of its slots, a launch stops adding once the list is
// full, and the other half (PS_SLOTS / 2 at least) is more than the resident
// warps' windows in flight.
__device__ __forceinline__ bool pair_insert(u64 *set, u64 mask, u64 w) {
    u64 s = pair_slot(w, mask);
    for (u64 probe = 0; probe <= mask; ++probe, s = (s + 1) & mask) {
        const u64 seen = *reinterpret_cast<volatile u64 *>(set + s);
        if (seen == w) return false;
        if (seen == FREE) {
            const u64 o = atomicCAS(reinterpret_cast<unsigned long long *>(set + s), FREE, w);
            if (o == FREE) return true;
            if (o == w) return false;
        }
    }
    return false;
}

// Level `level` (0: the base rule over the nodes [lo, hi)): the children of level
// - 1's pairs. A warp takes 32 pairs, prefix-sums their child counts and walks
// the children 32 at a time, so a pair's count does not hold up its lane;
// what is new is appended with one counter atomic per warp and window.
__global__ void __launch_bounds__(PS_THREADS)
pair_level_kernel(PairState st, const u32 *__restrict__ off, const u32 *__restrict__ val, u64 lo, u64 hi, int bits,
                  u32 level) {
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u64 mask = (1ull << bits) - 1;
    u64 i0, i1;
    if (level == 0) {
        i0 = lo;
        i1 = hi;
    } else {
        i0 = st.bound[level - 1];
        i1 = st.bound[level];
    }
    const u64 warps = (u64) gridDim.x * (PS_THREADS / 32);
    u32 rows = 0;
    for (u64 g = i0 + ((u64) blockIdx.x * PS_THREADS + threadIdx.x) / 32 * 32; g < i1; g += warps * 32) {
        u32 ab = 0, bb = 0, da = 0, db = 0;
        if (g + lane < i1) {
            u64 a, b;
            if (level == 0) {
                a = b = g + lane;
            } else {
                const u64 w = st.list[g + lane];
                a = w >> bits;
                b = w & mask;
            }
            ab = __ldg(off + a);
            da = __ldg(off + a + 1) - ab;
            bb = __ldg(off + b);
            db = __ldg(off + b + 1) - bb;
            if (da && db) ++rows;
        }
        const u32 n = da * db;
        const u32 incl = warp_inclusive_sum(n);
        const u32 total = __shfl_sync(0xffffffffu, incl, 31);
        const u32 pre = incl - n;
        for (u32 c0 = 0; c0 < total; c0 += 32) {
            const u32 c = c0 + lane;
            // owner of child c: the first lane whose inclusive sum is above c
            u32 o = 0;
#pragma unroll
            for (u32 step = 16; step >= 1; step >>= 1)
                if (__shfl_sync(0xffffffffu, incl, o + step - 1) <= c) o += step;
            o = min(o, 31u);
            const u32 r = c - __shfl_sync(0xffffffffu, pre, o);
            const u32 od = __shfl_sync(0xffffffffu, db, o);
            const u32 oa = __shfl_sync(0xffffffffu, ab, o), ob = __shfl_sync(0xffffffffu, bb, o);
            bool fresh = false;
            u64 w = 0;
            if (c < total && *reinterpret_cast<volatile unsigned long long *>(st.count) < st.cap) {
                const u32 i = r / od;
                const u64 x = __ldg(val + oa + i), y = __ldg(val + ob + (r - i * od));
                w = (x << bits) | y;
                if (level != 0 || x != y) fresh = pair_insert(st.set, st.mask, w);
            }
            const u32 fm = __ballot_sync(0xffffffffu, fresh);
            if (!fm) continue;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(st.count, (unsigned long long) __popc(fm));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(fm & lt);
            if (fresh && at < st.cap) st.list[at] = w;
        }
    }
    rows = warp_sum(rows);
    if (level && lane == 0 && rows) atomicAdd(st.rows + level - 1, (unsigned long long) rows);
    // the last block through closes the level
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(st.done, 1u) == gridDim.x - 1) {
            __threadfence();
            const unsigned long long n = *reinterpret_cast<volatile unsigned long long *>(st.count);
            st.bound[level + 1] = n < st.cap ? n : st.cap;
            *st.done = 0;
        }
    }
}

// Slots of `mid` for a level of so many pairs: twice the words that it can have, where `set` has
// as many (then it is never full: `bounded`). Cleared and probed whole it was 64 to 268 MB a level
// whatever the level held: SG of a binary tree of 1M nodes, two iterations, 2.89 -> 2.33 ms (2.31 on
// the sorted runs); a lattice of 1M edges 3.4 -> 2.6 (12.6).
__device__ __forceinline__ u64 mid_slots(const PairState &st, u64 pairs, bool &bounded) {
    const u64 want = 2 * pairs * st.most;
    bounded = want <= st.mask;
    return !bounded ? st.mask + 1 : want <= 1024 ? 1024 : 1ull << (64 - __clzll((long long) (want - 1)));
}

__global__ void pair_clear_kernel(PairState st, u32 level) {
    const u64 pairs = st.bound[level] - st.bound[level - 1];
    if (pairs == 0) return;
    bool bounded;
    const u64 n = mid_slots(st, pairs, bounded) / 2;
    ulonglong2 *p = reinterpret_cast<ulonglong2 *>(st.mid);
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x)
        p[i] = make_ulonglong2(FREE, FREE);
    if (blockIdx.x == 0 && threadIdx.x == 0) *st.mids = 0;
}

// The first join of level - 1's pairs (a, b): the distinct (x, b), x a child of a, and the second
// one's rows, b's children for each. For graphs past the bit matrix, whose join sizes are
// those of the sorted runs; `mid` is empty before the launch.
__global__ void __launch_bounds__(PS_THREADS)
pair_joins_kernel(PairState st, const u32 *__restrict__ off, const u32 *__restrict__ val, int bits, u32 level) {
    const u32 lane = threadIdx.x & 31;
    const u64 mask = (1ull << bits) - 1;
    const u64 i0 = st.bound[level - 1], i1 = st.bound[level];
    const u64 warps = (u64) gridDim.x * (PS_THREADS / 32);
    bool bounded;
    const u64 slots = mid_slots(st, i1 - i0, bounded);
    u64 first = 0, middle = 0, second = 0;
    for (u64 g = i0 + ((u64) blockIdx.x * PS_THREADS + threadIdx.x) / 32 * 32; g < i1; g += warps * 32) {
        u32 ab = 0, da = 0, b = 0, db = 0;
        if (g + lane < i1) {
            const u64 w = st.list[g + lane], a = w >> bits;
            b = (u32) (w & mask);
            ab = __ldg(off + a);
            da = __ldg(off + a + 1) - ab;
            db = __ldg(off + b + 1) - __ldg(off + b);
        }
        first += da;
        const u32 most = __reduce_max_sync(0xffffffffu, da);  // (64 at most)
        for (u32 k = 0; k < most; ++k) {
            const bool room = bounded || *reinterpret_cast<volatile unsigned long long *>(st.mids) < st.cap;
            const bool fresh = k < da && room && pair_insert(st.mid, slots - 1, ((u64) __ldg(val + ab + k) << bits) | b);
            const u32 fm = __ballot_sync(0xffffffffu, fresh);
            if (!room) *st.over = 1;
            if (!fm) continue;
            if (lane == 0 && !bounded) atomicAdd(st.mids, (unsigned long long) __popc(fm));
            middle += fresh;
            second += fresh ? db : 0u;
        }
    }
    first = warp_sum(first);
    middle = warp_sum(middle);
    second = warp_sum(second);
    if (lane == 0) {
        if (first) atomicAdd(st.first + level - 1, (unsigned long long) first);
        if (middle) atomicAdd(st.middle + level - 1, (unsigned long long) middle);
        if (second) atomicAdd(st.second + level - 1, (unsigned long long) second);
    }
}

__global__ void pair_refill_kernel(const u64 *__restrict__ list, u64 n, u64 *set, u64 mask) {
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x)
        pair_insert(set, mask, list[i]);
}

// found[0] = largest degree, found[1] = edges, found[2] = sum of the degrees' squares.
__global__ void degrees_kernel(const u32 *__restrict__ off, u64 lo, u64 hi, unsigned long long *__restrict__ found) {
    u32 m = 0;
    u64 c = 0, s = 0;
    for (u64 r = lo + (u64) blockIdx.x * blockDim.x + threadIdx.x; r < hi; r += (u64) gridDim.x * blockDim.x) {
        const u32 d = off[r + 1] - off[r];
        m = max(m, d);
        c += d;
        s += (u64) d * d;
    }
    m = __reduce_max_sync(0xffffffffu, m);
    c = warp_sum(c);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0 && m) {
        atomicMax(found, (unsigned long long) m);
        atomicAdd(found + 1, (unsigned long long) c);
        atomicAdd(found + 2, (unsigned long long) s);
    }
}

// counts[instance * levels + level] += words. A warp's words are of one level mostly and
// of few instances: one atomic for equal ones (a session of 32 lattices: 0.22 -> 0.14 ms
// per admission).
__global__ void pair_counts_kernel(const u64 *__restrict__ list, u64 n, int bits, const u64 *__restrict__ bound,
                                   u32 levels, const u64 *__restrict__ inst_lo, u32 n_inst,
                                   unsigned long long *__restrict__ counts) {
    const u32 lane = threadIdx.x & 31;
    for (u64 i0 = (u64) blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < n; i0 += (u64) gridDim.x * blockDim.x) {
        const u64 i = i0 + lane;
        unsigned long long at = ~0ull;
        if (i < n) {
            const u64 x = list[i] >> bits;
            u32 a = 0, b = n_inst;
            while (a < b) {
                const u32 m = (a + b) >> 1;
                if (inst_lo[m] <= x) a = m + 1;
                else b = m;
            }
            const u32 inst = a - 1;
            a = 0;
            b = levels;
            while (a < b) {  // the last level whose first word is at most i
                const u32 m = (a + b) >> 1;
                if (bound[m] <= i) a = m + 1;
                else b = m;
            }
            at = (u64) inst * levels + (a - 1);
        }
        const u32 same = __match_any_sync(0xffffffffu, at);
        if (i < n && lane == (u32) __ffs(same) - 1) atomicAdd(counts + at, (unsigned long long) __popc(same));
    }
}

}  // namespace

bool PairDegrees::fits() const { return most <= PS_DEGREE; }

PairDegrees pair_degrees(Context &ctx, const Csr &csr, u64 lo, u64 hi) {
    auto *found = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[24]);
    DL_CUDA(cudaMemsetAsync(found, 0, 24, ctx.stream));
    DL_LAUNCH(ctx, K_PREP, 4.0 * (hi - lo),
              degrees_kernel<<<grid_for(hi - lo, T256, ctx, 8), T256, 0, ctx.stream>>>(csr.off, lo, hi, found));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, found, 24, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    PairDegrees d;
    d.most = ctx.host_scalars[0];
    d.edges = ctx.host_scalars[1];
    d.squares = ctx.host_scalars[2];
    return d;
}

// The search inserts every child of every pair, the product of two sources' out-edges, at
// random places: 0.06 ns each while the set is in L2, 0.25 ns for a new one past it. The
// sorted runs join twice, drop duplicates in between and sort, 0.07 ns a word, but an
// iteration costs half a millisecond however little it finds. So the search loses where
// an edge's source has three out-edges or more and the pairs, or the children to look up, are
// many. Measured, batches on both forms, sorted runs against the search:
//   random graphs (1 + d out-edges of an edge's source) of d = 2.5 / 3 / 4 / 6 edges a node, 8 of
//   3000 nodes: 32 / 42 / 46 / 63 ms against 46 / 61 / 91 / 147; of 2, one of 10,000 nodes: 31
//   against 37; 8 of 1000 nodes, 4 edges: 10.0 against 9.1, 6 edges: 9.7 against 13.0;
//   trees of three children a node (3.0), 8 of 1000 inner nodes: 6.8 against 10.9, 3 of 20K nodes
//   with both directions: 169 against 323;
//   below the line: 1.5 edges a node (2.5), 8 of 3000: 22 against 10; 2 edges, 8 of 1000: 72
//   against 4.3; meshes of 1.8 edges a node (2.5), 4 of 4096 nodes: 143 against 20, one of 22K:
//   163 against 133.
bool pair_search_outrun(const PairDegrees &d, const std::vector<u64> &n_ids) {
    if (d.of_sources() <= 2.9) return false;
    double nodes = 0, squares = 0;
    for (u64 n : n_ids) {
        nodes += (double) n;
        squares += (double) n * (double) n;
    }
    const double mean = (double) d.edges / std::max(nodes, 1.0);
    const double children = mean * mean * squares;  // pairs of edges
    return std::min(squares, children) > 1.6e7 || children > 2e8;
}

PairSearch pair_search(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const PairOptions &opt) {
    Workspace &ws = ctx.ws;
    PairSearch ps;
    DevBuf &list = ws.jbuf[0], &set = ws.jbuf[1], &mid = ws.full[0];
    // room for four pairs a node at first, slots for twice as many words (a set of
    // up to 16M slots stays in L2, where an insert costs a fifth); a level
    // that needs more is repeated on a set four times the size
    u64 slots = PS_SLOTS;
    while (slots < 8 * (hi - lo)) slots <<= 1;
    // A matrix costs its size whatever it holds and 50 to 200 us an iteration, the list 0.3 ns a
    // pair: past 16 pairs a node (and the first set), levels of more than one a node are the
    // matrix's, and so are results past 512. Measured: a binary tree of 100K nodes, two
    // iterations, 7 pairs a node, 1.9 ms on the matrix, 0.65 on the list; a mesh of 264K nodes, 17 a
    // node in 67 levels, 20 against 3.1; random graphs past the line lose 1 to 5 % to it.
    const u64 n = hi - lo, many = std::max<u64>(16 * n, PS_SLOTS / 2);
    // Whether the levels left under max_levels end with at most 128 pairs a node, if each is as many
    // times the one before as the last whole one is (the first: as random nodes' or siblings' children):
    // then the list is the faster form to the end. Measured, handed over or not (on the matrix
    // alone): 220K layered nodes, two iterations, 64 a node, 16.9 / 3.5 (12.1) ms; random graph of 260K
    // nodes and 300K edges, ten, 83 a node, 48 / 6.2 (21.7); tree of 250K nodes with five children each,
    // two, 124 a node, 18.4 / 7.9 (7.1); mesh of 60K nodes, ten, 121 a node, 4.2 / 4.4 (3.9).
    auto ends_soon = [&](u64 next) {
        if (!opt.max_levels || next == 0 || opt.max_levels - next > 16) return false;
        const double mean = (double) opt.deg.edges / (double) n;
        double all = (double) ps.bound[next], last = all - (double) ps.bound[next - 1];
        const double by = next < 2 ? std::max(mean * mean, opt.deg.of_sources())
                                   : last / (double) std::max<u64>(ps.bound[next - 1] - ps.bound[next - 2], 1);
        for (u64 k = next; k <= opt.max_levels; ++k) all += last *= by;
        return all <= 128.0 * (double) n;
    };
    const std::initializer_list<DevBuf *> idle = {&ws.bitmat[0], &ws.bitmat[1], &ws.cl_rows[0], &ws.cl_rows[1]};
    const u64 unit = opt.joins ? 20 : 12;  // bytes a slot: the set, half as many words, the joins' set
    if (slots * unit > opt.limit || !ctx.room_for({{&list, slots / 2 * 8}, {&set, slots * 8}}, idle)) return ps;
    // After the counters of the list, the blocks and the joins' set, five arrays by level
    // (PairState): bound, rows, first, middle, second, each levels + 4 words
    u64 levels = 64;
    constexpr u64 HEAD = 8, ARRAYS = 5;
    auto words = [](u64 lv) { return HEAD + ARRAYS * (lv + 4); };
    ctx.reserve(ws.cl_levels, words(levels) * 8);
    DL_CUDA(cudaMemsetAsync(ws.cl_levels.p, 0, words(levels) * 8, ctx.stream));
    PairState st;
    auto bind = [&]() {
        st.list = list.as<u64>();
        st.cap = slots / 2;
        st.set = set.as<u64>();
        st.mask = slots - 1;
        st.mid = mid.as<u64>();
        st.most = opt.deg.most;
        auto *b = ws.cl_levels.as<unsigned long long>();
        st.count = b;
        st.done = reinterpret_cast<u32 *>(b + 1);
        st.mids = b + 2;
        st.over = b + 3;
        st.bound = b + HEAD;
        st.rows = st.bound + levels + 4;
        st.first = st.rows + levels + 4;
        st.middle = st.first + levels + 4;
        st.second = st.middle + levels + 4;
    };
    ctx.reserve(list, slots / 2 * 8);
    ctx.reserve(set, slots * 8);
    DL_CUDA(cudaMemsetAsync(set.p, 0xFF, slots * 8, ctx.stream));
    if (opt.joins) ctx.reserve(mid, slots * 8);
    bind();
    ps.bound.assign(1, 0);
    auto launch = [&](u64 level, u64 pairs) {
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                  pair_level_kernel<<<grid_for(pairs, PS_THREADS, ctx, 8), PS_THREADS, 0, ctx.stream>>>(
                      st, csr.off, csr.val, lo, hi, bits, (u32) level));
        if (opt.joins && level) {
            DL_LAUNCH(ctx, K_PREP, 0,
                      pair_clear_kernel<<<grid_for(slots / 2, T256, ctx, 8), T256, 0, ctx.stream>>>(st, (u32) level));
            DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                      pair_joins_kernel<<<grid_for(pairs, PS_THREADS, ctx, 8), PS_THREADS, 0, ctx.stream>>>(
                          st, csr.off, csr.val, bits, (u32) level));
        }
    };
    for (u64 level = 0;;) {
        // room for the levels of this batch
        if (level + PS_LEVELS + 2 > levels) {
            const u64 old = levels;
            levels *= 4;
            DevBuf nb;
            ctx.reserve(nb, words(levels) * 8);
            DL_CUDA(cudaMemsetAsync(nb.p, 0, words(levels) * 8, ctx.stream));
            u64 *f = ws.cl_levels.as<u64>(), *t = nb.as<u64>();
            DL_CUDA(cudaMemcpyAsync(t, f, HEAD * 8, cudaMemcpyDeviceToDevice, ctx.stream));
            for (u64 a = 0; a < ARRAYS; ++a)
                DL_CUDA(cudaMemcpyAsync(t + HEAD + a * (levels + 4), f + HEAD + a * (old + 4), (old + 4) * 8,
                                        cudaMemcpyDeviceToDevice, ctx.stream));
            ctx.give_back(ws.cl_levels);
            ws.cl_levels = nb;
            bind();
        }
        // an unknown number of pairs: the grid for all nodes, or for the last known level
        const u64 batch = opt.max_levels ? std::min<u64>(PS_LEVELS, opt.max_levels - level + 1) : PS_LEVELS;
        const u64 known = level ? ps.bound[level] - ps.bound[level - 1] : n;
        for (u64 k = 0; k < batch; ++k) launch(level + k, level || k ? std::max<u64>(4 * known, 1 << 15) : known);
        // host copies: the head's words [0, 4), then `batch` of each array (all but bound from the
        // rows that this batch's first level counts on)
        u64 *hs = ctx.host_scalars;
        const u64 row0 = level ? level - 1 : 0;
        DL_CUDA(cudaMemcpyAsync(hs, st.count, 32, cudaMemcpyDeviceToHost, ctx.stream));
        DL_CUDA(cudaMemcpyAsync(hs + 4, st.bound + level + 1, batch * 8, cudaMemcpyDeviceToHost, ctx.stream));
        DL_CUDA(cudaMemcpyAsync(hs + 4 + PS_LEVELS, st.rows + row0, batch * 8, cudaMemcpyDeviceToHost, ctx.stream));
        if (opt.joins)
            for (u64 a = 0; a < 3; ++a)
                DL_CUDA(cudaMemcpyAsync(hs + 4 + (2 + a) * PS_LEVELS, st.first + a * (levels + 4) + row0, batch * 8,
                                        cudaMemcpyDeviceToHost, ctx.stream));
        static_assert(4 + ARRAYS * PS_LEVELS < 2 * 31, "fits the host scalars");
        ctx.sync();
        const u64 found = hs[0], *bounds = hs + 4;
        if (opt.joins && hs[3]) break;  // (x, b) words were not counted
        bool full = found >= st.cap, end = false;
        u64 good = batch;  // levels of the batch that are whole
        if (full) {
            good = 0;
            while (good < batch && bounds[good] < st.cap) ++good;
        }
        const u64 listed = ps.n_words(), begun = level;
        for (u64 k = 0; k < good; ++k) {
            const u64 lv = level + k;
            if (lv) {
                const u64 at = level ? k : k - 1;
                ps.rows.push_back(hs[4 + PS_LEVELS + at]);
                if (opt.joins) {
                    ps.first.push_back(hs[4 + 2 * PS_LEVELS + at]);
                    ps.middle.push_back(hs[4 + 3 * PS_LEVELS + at]);
                    ps.second.push_back(hs[4 + 4 * PS_LEVELS + at]);
                }
            }
            ps.bound.push_back(bounds[k]);
            if (ps.bound[lv + 1] == ps.bound[lv]) {  // nothing new
                ps.complete = end = true;
                break;
            }
        }
        ctx.prof_add_bytes(K_BITMAP_EXPAND, 8.0 * (ps.n_words() - listed));  // a new pair's word
        if (end) break;
        level += good;
        if (!full && opt.max_levels && level > opt.max_levels) {
            ps.complete = true;
            break;
        }
        if (opt.handover) {
            const u64 all = full ? found : ps.n_words(), last = all - (level ? ps.bound[full ? level : level - 1] : 0);
            if (all > 512 * n + many || (all >= many && last > n && !ends_soon(level))) break;
        }
        if (full) {  // repeat level `level` with more room: the set again from the words listed before it
            const u64 keep = ps.bound[level];
            slots *= 4;
            DevBuf nl;
            if (slots * unit > opt.limit || !ctx.room_for({{&nl, slots / 2 * 8}, {&set, slots * 8}}, idle)) break;
            ctx.reserve(nl, slots / 2 * 8);
            DL_CUDA(cudaMemcpyAsync(nl.p, list.p, keep * 8, cudaMemcpyDeviceToDevice, ctx.stream));
            ctx.give_back(list);
            list = nl;
            ctx.reserve(set, slots * 8);
            DL_CUDA(cudaMemsetAsync(set.p, 0xFF, slots * 8, ctx.stream));
            if (opt.joins) ctx.reserve(mid, slots * 8);
            bind();
            if (keep)
                DL_LAUNCH(ctx, K_BITMAP_EXPAND, 16.0 * keep,
                          pair_refill_kernel<<<grid_for(keep, T256, ctx), T256, 0, ctx.stream>>>(st.list, keep, st.set,
                                                                                                st.mask));
            DL_CUDA(cudaMemcpyAsync(st.count, ps.bound.data() + level, 8, cudaMemcpyHostToDevice, ctx.stream));
            // rows counted by the levels that are repeated: the batch's last one counted rows[begun + batch - 2]
            const u64 row = level ? level - 1 : 0;
            for (u64 a = 0; a < 4; ++a)
                DL_CUDA(cudaMemsetAsync(st.rows + a * (levels + 4) + row, 0, (begun + batch - 1 - row) * 8, ctx.stream));
            ctx.sync();  // ps.bound is host memory
        }
    }
    return ps;
}

void pair_level_counts(Context &ctx, const PairSearch &ps, int bits, const u64 *inst_lo, u64 n_inst, u64 *counts) {
    const u64 levels = ps.bound.size() - 1;
    DL_CUDA(cudaMemsetAsync(counts, 0, n_inst * levels * 8, ctx.stream));
    if (ps.n_words() == 0) return;
    DL_LAUNCH(ctx, K_PREP, 8.0 * ps.n_words(),
              pair_counts_kernel<<<grid_for(ps.n_words(), T256, ctx), T256, 0, ctx.stream>>>(
                  ctx.ws.jbuf[0].as<u64>(), ps.n_words(), bits, ctx.ws.cl_levels.as<u64>() + 8, (u32) levels, inst_lo,
                  (u32) n_inst, reinterpret_cast<unsigned long long *>(counts)));
}

}  // namespace detail
}  // namespace dl
