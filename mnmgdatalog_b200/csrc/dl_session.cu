// Multi-instance fixpoint session: the batched and served forms.
//
// Many independent queries of one program run as ONE union fixpoint. Every
// admitted instance gets its own contiguous range of node ranks, so its
// tuples never meet another instance's: joins, sorts, the set difference and
// the merge of one iteration process every active instance at once, and the
// per-iteration launch and synchronisation cost is paid once for all of them.
// Instances are admitted at any iteration boundary (continuous batching):
// their edges are appended to the union's offset table (their ranks are above
// every rank in use, so the table stays sorted). No instance needs the common
// steps: a source's (TC, dl_closure.cu) or a pair's (SG, dl_pairs.cu) search and a
// component's labels (WCC, dl_wcc.cu) never meet another instance's, so the
// instances admitted together are computed to their own stops in one go -- for
// WCC with the reference's rule the iteration where that rule fires for the
// instance -- and the steps report their iterations one by one. SG instances that the
// search does not suit (degrees, many pairs, memory) keep the common steps: their initial
// delta joins the next iteration, and each leaves the union at its own fixpoint.
// Results are bit-exact with running each query alone.
#include <algorithm>
#include <cstring>
#include <memory>

#include "dl_closure.h"
#include "dl_engine_detail.h"
#include "dl_join.cuh"
#include "dl_pairs.h"
#include "dl_scan.cuh"
#include "dl_session.h"
#include "dl_wcc.h"

namespace dl {
namespace {

using namespace detail;

#define GRID_STRIDE(i, n) \
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (u64) gridDim.x * blockDim.x)

// Instance of row r of a concatenation: last k with off[k] <= r.
__device__ __forceinline__ u32 segment_of(const u64 *__restrict__ off, u32 count, u64 r) {
    u32 a = 0, b = count;
    while (a < b) {
        const u32 m = (a + b) >> 1;
        if (off[m] <= r) a = m + 1;
        else b = m;
    }
    return a - 1;
}

// (instance << 32 | biased node id) for both columns of every row.
__global__ void session_tag_kernel(const int32_t *__restrict__ rows, u64 n, const u64 *__restrict__ off, u32 count,
                                   u64 *__restrict__ out) {
    GRID_STRIDE(r, n) {
        const u64 k = (u64) segment_of(off, count, r) << 32;
        out[2 * r] = k | ((u32) rows[2 * r] ^ 0x80000000u);
        out[2 * r + 1] = k | ((u32) rows[2 * r + 1] ^ 0x80000000u);
    }
}

// first[k] = index of the first tagged word of instance k (k in [0, count]).
__global__ void session_first_kernel(const u64 *__restrict__ u, u64 nu, u32 count, u64 *__restrict__ first) {
    GRID_STRIDE(k, (u64) count + 1) {
        const u64 target = k << 32;
        u64 l = 0, h = nu;
        while (l < h) {
            const u64 m = (l + h) >> 1;
            if (u[m] < target) l = m + 1;
            else h = m;
        }
        first[k] = l;
    }
}

__global__ void session_ids_kernel(const u64 *__restrict__ u, u64 nu, int32_t *__restrict__ ids) {
    GRID_STRIDE(i, nu) ids[i] = (int32_t) ((u32) u[i] ^ 0x80000000u);
}

__device__ __forceinline__ u64 lower_bound_u64(const u64 *__restrict__ a, u64 n, u64 x) {
    u64 l = 0, h = n;
    while (l < h) {
        const u64 m = (l + h) >> 1;
        if (a[m] < x) l = m + 1;
        else h = m;
    }
    return l;
}

// Rows of many instances -> words over union ranks (rank = base + position
// of (instance, id) among the sorted distinct tagged ids).
__global__ void session_pack_many_kernel(const int32_t *__restrict__ rows, u64 n, const u64 *__restrict__ off,
                                         u32 count, const u64 *__restrict__ u, u64 nu, u64 base, int bits,
                                         u64 *__restrict__ fwd, u64 *__restrict__ rev) {
    GRID_STRIDE(r, n) {
        const u64 k = (u64) segment_of(off, count, r) << 32;
        const u64 ra = base + lower_bound_u64(u, nu, k | ((u32) rows[2 * r] ^ 0x80000000u));
        const u64 rb = base + lower_bound_u64(u, nu, k | ((u32) rows[2 * r + 1] ^ 0x80000000u));
        if (fwd) fwd[r] = (ra << bits) | rb;
        if (rev) rev[r] = (rb << bits) | ra;
    }
}

// Appends the sorted words of ranks [lo, hi) to the union offset table:
// off[r] = base + (first word with key >= r) for r in [lo, hi].
__global__ void session_csr_kernel(const u64 *__restrict__ w, u64 n, int bits, u64 lo, u64 hi, u64 base,
                                   u32 *__restrict__ off, u32 *__restrict__ val) {
    GRID_STRIDE(k, hi - lo + 1) {
        const u64 target = (lo + k) << bits;
        u64 l = 0, h = n;
        while (l < h) {
            const u64 m = (l + h) >> 1;
            if (w[m] < target) l = m + 1;
            else h = m;
        }
        off[lo + k] = (u32) (base + l);
    }
    const u64 mask = (1ull << bits) - 1;
    GRID_STRIDE(i, n) val[base + i] = (u32) (w[i] & mask);
}

// Instance index of a rank: last active instance whose first rank <= r.
__device__ __forceinline__ u32 instance_of(const u64 *__restrict__ lo, u32 n, u64 r) {
    u32 a = 0, b = n;
    while (a < b) {
        const u32 m = (a + b) >> 1;
        if (lo[m] <= r) a = m + 1;
        else b = m;
    }
    return a - 1;
}

// Per-instance count of delta words; the rank is word >> shift.
__global__ void session_hist_kernel(const u64 *__restrict__ d, u64 n, int shift, const u64 *__restrict__ lo, u32 ninst,
                                    unsigned long long *__restrict__ cnt) {
    extern __shared__ u32 sh[];
    const bool smem = ninst <= 8192;
    if (smem)
        for (u32 i = threadIdx.x; i < ninst; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    GRID_STRIDE(i, n) {
        const u32 k = instance_of(lo, ninst, d[i] >> shift);
        if (k >= ninst) continue;  // below every active range: not counted
        if (smem) atomicAdd(&sh[k], 1u);
        else atomicAdd(&cnt[k], 1ull);
    }
    __syncthreads();
    if (smem)
        for (u32 i = threadIdx.x; i < ninst; i += blockDim.x)
            if (sh[i]) atomicAdd(&cnt[i], (unsigned long long) sh[i]);
}

// Word ranges of instances in the three sorted runs: for instance k (ranks
// lohi[k] .. lohi[n + k]) out[6k..6k+5] = [first, end) in run 0, 1 and 2.
struct Runs3 {
    const u64 *w[3];
    u64 n[3];
};
__global__ void session_bounds_kernel(Runs3 runs, const u64 *__restrict__ lohi, u32 n, int bits,
                                      u64 *__restrict__ out) {
    GRID_STRIDE(t, 6 * (u64) n) {
        const u64 k = t / 6, which = t % 6, r = which >> 1;
        const u64 target = (which & 1 ? lohi[n + k] : lohi[k]) << bits;
        out[t] = lower_bound_u64(runs.w[r], runs.n[r], target);
    }
}

struct NonZero {
    const u32 *c;
    __device__ __forceinline__ u64 degree(u64 i) const { return c[i] != 0u; }
};

// Components of every instance (local ranks, ascending), the largest size
// per instance, and where each instance's components start.
__global__ void session_wcc_comp_kernel(const u32 *__restrict__ cnt, const u64 *__restrict__ pos,
                                        const u64 *__restrict__ off, u32 n, u64 total, u32 *__restrict__ comp,
                                        unsigned long long *__restrict__ largest, u64 *__restrict__ start) {
    GRID_STRIDE(t, total) {
        const u32 k = segment_of(off, n, t);
        if (t == off[k]) start[k] = pos[t];
        const u32 c = cnt[t];
        if (c) {
            comp[pos[t]] = (u32) (t - off[k]);
            atomicMax(&largest[k], (unsigned long long) c);
        }
    }
}

// Keep delta words whose instance is still active (freezing finished ones).
struct KeepActive {
    const u64 *lo;
    const uint8_t *live;
    u32 n;
    int shift;
    __device__ bool operator()(u64 cur, u64, bool) const {
        const u32 k = instance_of(lo, n, cur >> shift);
        return k < n && live[k] != 0;
    }
};

template <bool KeyFirst>
__global__ void session_unpack_kernel(const u64 *__restrict__ w, u64 n, int bits, u64 base,
                                      const int32_t *__restrict__ ids, int32_t *__restrict__ out) {
    const u64 mask = (1ull << bits) - 1;
    GRID_STRIDE(i, n) {
        const u64 x = w[i];
        const int32_t hi = ids[(x >> bits) - base], lo = ids[(x & mask) - base];
        int2 r;
        r.x = KeyFirst ? hi : lo;
        r.y = KeyFirst ? lo : hi;
        reinterpret_cast<int2 *>(out)[i] = r;
    }
}

__global__ void session_unpack_comp_kernel(const u32 *__restrict__ comp, u64 n, const int32_t *__restrict__ ids,
                                           int32_t *__restrict__ out) {
    GRID_STRIDE(i, n) {
        int2 r;
        r.x = ids[comp[i]];
        r.y = 0;
        reinterpret_cast<int2 *>(out)[i] = r;
    }
}

// labels: union label rank of each local node; ids indexed by local rank.
__global__ void session_unpack_labels_kernel(const u32 *__restrict__ label, u64 lo, u64 n,
                                             const int32_t *__restrict__ ids, int32_t *__restrict__ out) {
    GRID_STRIDE(i, n) out[i] = ids[label[i] - lo];
}

// Keeps the words whose instance (rank = word >> shift) is live.
template <class Keep>
u64 session_select(Context &ctx, u64 *buf, u64 n, Keep keep, int slot) {
    if (n == 0) return 0;
    const u64 tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    u64 *lb = ctx.lookback_words(tiles);
    u32 *ctr = ctx.tile_counter(slot);
    u64 *cnt = &ctx.ctrl->scalar[28];
    DL_CUDA(cudaMemsetAsync(ctr, 0, sizeof(u32), ctx.stream));
    DL_LAUNCH(ctx, K_SELECT, 16.0 * n,
              select_kernel<Keep><<<(unsigned) tiles, SCAN_THREADS, 0, ctx.stream>>>(
                  buf, n, buf, keep, lb, ctr, ctx.next_epoch(), &ctx.ctrl->err, cnt));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars + 4, cnt, sizeof(u64), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    return ctx.host_scalars[4];
}

// Grows a buffer keeping its first `keep` bytes.
void grow_keep(Context &ctx, DevBuf &b, size_t bytes, size_t keep) {
    if (b.p && b.cap >= bytes) return;
    DevBuf nb;
    ctx.reserve(nb, std::max(bytes, b.cap * 3 / 2));
    if (keep && b.p) DL_CUDA(cudaMemcpyAsync(nb.p, b.p, keep, cudaMemcpyDeviceToDevice, ctx.stream));
    ctx.give_back(b);  // reused on the same stream, after the copy
    b = nb;
}

}  // namespace

struct SessionImpl {
    Context ctx;  // private workspace; shares the caller's stream
    Context *parent = nullptr;
    int program = DL_PROGRAM_TC;
    dl_options opt{};
    int bits = 30;
    u64 rank_cap = 0;
    u64 next_rank = 0;
    DevBuf off, val;  // union offset table over ranks, values
    u64 n_vals = 0;
    FullSet F = [] {
        FullSet f;
        f.three = true;
        return f;
    }();
    u64 dead = 0;  // words of finished instances still in the full runs
    DevBuf delta;  // union delta (probe of the next iteration)
    u64 n_delta = 0;
    DevBuf inst_lo, inst_hi;    // device copies of the active instances' rank ranges
    DevBuf counts;              // per instance delta counts
    DevBuf range_lo;            // first ranks of the instances of a range count
    DevBuf admit_off, admit_first;  // row offsets / first tagged ids of an admission
    DevBuf live;                // per active instance flag (frozen by max_iterations)
    std::vector<SessionInstance> inst;
    std::vector<i64> active;    // instance ids in rank order
    std::vector<i64> finished;  // finished since the last poll
    std::vector<i64> pending;   // TC: admitted since the last step, not searched yet
    u64 pending_vals = 0;       // their first edge
    bool inst_dirty = true;
};

namespace {

Graph union_graph(SessionImpl &s) {
    Graph g;
    g.n_ids = (u32) s.next_rank;
    g.bits = s.bits;
    g.csr.off = s.off.as<u32>();
    g.csr.val = s.val.as<u32>();
    g.csr.n_keys = (u32) s.next_rank;
    g.csr.n_vals = s.n_vals;
    // both rank fields are below next_rank: sort only the bits that can vary
    g.nwin = plan_windows(s.bits, bits_for(std::max<u64>(s.next_rank, 2)), g.win);
    return g;
}

// Sorts the n words of buf (alt: ping-pong) whose rank fields are below
// 2^used_bits and drops duplicates.
u64 *sort_unique_fields(Context &ctx, DevBuf &buf, DevBuf &alt, u64 n, int field_bits, int used_bits, u64 &n_out) {
    ctx.reserve(alt, std::max<u64>(n, 1) * 8);
    int w[8];
    const int nw = plan_windows(field_bits, used_bits, w);
    u64 *r = radix_sort_windows(ctx, buf.as<u64>(), alt.as<u64>(), n, w, nw);
    n_out = unique_words(ctx, r, n, r);
    return r;
}

// Inserts the words of a brand-new key range into the full relation.
void full_insert_new(SessionImpl &s, const u64 *w, u64 n) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    FullSet &F = s.F;
    if (n == 0) return;
    // new ranks are above every word in the runs: the merge appends
    ctx.reserve(ws.tiny[1 - F.tcur], (F.ntiny + n) * 8);
    merge_words(ctx, ws.tiny[F.tcur].as<u64>(), F.ntiny, w, n, ws.tiny[1 - F.tcur].as<u64>(), Codec::Raw);
    F.tcur = 1 - F.tcur;
    F.ntiny += n;
    if (F.ntiny * ctx.tune.small_ratio >= F.nsmall) fold_tiny(ctx, F);  // also when the small run is empty
    if (F.nsmall && F.nsmall * ctx.tune.small_ratio >= F.nbig) {
        fold_tiny(ctx, F);
        ctx.reserve(ws.full[1 - F.cur], (F.nbig + F.nsmall) * 8);
        merge_words(ctx, ws.full[F.cur].as<u64>(), F.nbig, ws.small[F.scur].as<u64>(), F.nsmall,
                    ws.full[1 - F.cur].as<u64>(), Codec::Raw);
        F.cur = 1 - F.cur;
        F.nbig += F.nsmall;
        F.nsmall = 0;
        F.sample_ok = false;
        F.ssample_ok = false;
    }
}

void delta_append(SessionImpl &s, const u64 *w, u64 n) {
    if (n == 0) return;
    grow_keep(s.ctx, s.delta, (s.n_delta + n) * 8, s.n_delta * 8);
    DL_CUDA(cudaMemcpyAsync(s.delta.as<u64>() + s.n_delta, w, n * 8, cudaMemcpyDeviceToDevice, s.ctx.stream));
    s.n_delta += n;
}

void upload_active(SessionImpl &s) {
    if (!s.inst_dirty) return;
    const u64 na = s.active.size();
    std::vector<u64> lo(std::max<u64>(na, 1)), hi(std::max<u64>(na, 1));
    for (u64 i = 0; i < na; ++i) {
        lo[i] = s.inst[s.active[i]].rank_lo;
        hi[i] = s.inst[s.active[i]].rank_hi;
    }
    s.ctx.reserve(s.inst_lo, lo.size() * 8);
    s.ctx.reserve(s.inst_hi, hi.size() * 8);
    DL_CUDA(cudaMemcpyAsync(s.inst_lo.p, lo.data(), na * 8, cudaMemcpyHostToDevice, s.ctx.stream));
    DL_CUDA(cudaMemcpyAsync(s.inst_hi.p, hi.data(), na * 8, cudaMemcpyHostToDevice, s.ctx.stream));
    s.ctx.sync();  // lo/hi are host temporaries
    s.inst_dirty = false;
}

// Counts of the words of d (rank = word >> shift) per instance, given the
// instances' first ranks in increasing order on the device.
std::vector<u64> counts_by_lo(SessionImpl &s, const u64 *d, u64 n, int shift, const u64 *d_lo, u64 na) {
    Context &ctx = s.ctx;
    std::vector<u64> c(na, 0);
    if (na == 0 || n == 0) return c;
    ctx.reserve(s.counts, na * 8);
    DL_CUDA(cudaMemsetAsync(s.counts.p, 0, na * 8, ctx.stream));
    const unsigned smem = na <= 8192 ? (unsigned) (na * 4) : 0u;
    DL_LAUNCH(ctx, K_PREP, 8.0 * n,
              session_hist_kernel<<<grid_for(n, 256, ctx, 8), 256, smem, ctx.stream>>>(
                  d, n, shift, d_lo, (u32) na, (unsigned long long *) s.counts.p));
    DL_CUDA(cudaMemcpyAsync(c.data(), s.counts.p, na * 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    return c;
}

// Per-active-instance counts.
std::vector<u64> delta_counts(SessionImpl &s, const u64 *d, u64 n, int shift) {
    if (s.active.empty() || n == 0) return std::vector<u64>(s.active.size(), 0);
    upload_active(s);
    return counts_by_lo(s, d, n, shift, s.inst_lo.as<u64>(), s.active.size());
}

// Counts for the instances whose first ranks are `lo` (increasing).
std::vector<u64> range_counts(SessionImpl &s, const u64 *d, u64 n, int shift, const std::vector<u64> &lo) {
    if (lo.empty() || n == 0) return std::vector<u64>(lo.size(), 0);
    s.ctx.reserve(s.range_lo, lo.size() * 8);
    DL_CUDA(cudaMemcpyAsync(s.range_lo.p, lo.data(), lo.size() * 8, cudaMemcpyHostToDevice, s.ctx.stream));
    return counts_by_lo(s, d, n, shift, s.range_lo.as<u64>(), lo.size());  // syncs before `lo` goes
}

// A device block shared by the instances extracted or admitted together; its
// memory returns to the session's buffer cache with the last instance.
std::shared_ptr<DevBuf> make_block(Context &ctx, size_t bytes) {
    DevBuf *b = new DevBuf;
    try {
        ctx.reserve(*b, std::max<size_t>(bytes, 8));
    } catch (...) {
        delete b;
        throw;
    }
    Context *c = &ctx;
    return std::shared_ptr<DevBuf>(b, [c](DevBuf *x) {
        c->give_back(*x);
        delete x;
    });
}

// Uploads the rank ranges of `ids` ([lo..., hi...]) to s.range_lo.
void upload_ranges(SessionImpl &s, const std::vector<i64> &ids) {
    const u64 n = ids.size();
    std::vector<u64> h(2 * n);
    for (u64 k = 0; k < n; ++k) {
        h[k] = s.inst[ids[k]].rank_lo;
        h[n + k] = s.inst[ids[k]].rank_hi;
    }
    s.ctx.reserve(s.range_lo, 2 * n * 8);
    DL_CUDA(cudaMemcpyAsync(s.range_lo.p, h.data(), 2 * n * 8, cudaMemcpyHostToDevice, s.ctx.stream));
    s.ctx.sync();  // h is a host temporary
}

// Sorted words of finished TC/SG instances out of the full runs, into one
// block (each instance's words are a key range of each run).
void extract_words(SessionImpl &s, const std::vector<i64> &ids) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    const u64 n = ids.size();
    upload_ranges(s, ids);
    ctx.reserve(s.counts, 6 * n * 8);
    Runs3 runs;
    runs.w[0] = ws.full[s.F.cur].as<u64>();
    runs.n[0] = s.F.nbig;
    runs.w[1] = ws.small[s.F.scur].as<u64>();
    runs.n[1] = s.F.nsmall;
    runs.w[2] = ws.tiny[s.F.tcur].as<u64>();
    runs.n[2] = s.F.ntiny;
    DL_LAUNCH(ctx, K_PREP, 0,
              session_bounds_kernel<<<grid_for(6 * n, 256, ctx, 4), 256, 0, ctx.stream>>>(
                  runs, s.range_lo.as<u64>(), (u32) n, s.bits, s.counts.as<u64>()));
    std::vector<u64> hb(6 * n);
    DL_CUDA(cudaMemcpyAsync(hb.data(), s.counts.p, 6 * n * 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    u64 total = 0, pair_max = 0;
    for (u64 k = 0; k < n; ++k) {
        const u64 na = hb[6 * k + 1] - hb[6 * k], nb = hb[6 * k + 3] - hb[6 * k + 2], nc = hb[6 * k + 5] - hb[6 * k + 4];
        total += na + nb + nc;
        if (na && nb && nc) pair_max = std::max(pair_max, na + nb);
    }
    auto block = make_block(ctx, total * 8);
    DevBuf tmp;  // run 0 + run 1 slices of an instance that has words in all three runs
    if (pair_max) ctx.reserve(tmp, pair_max * 8);
    u64 at = 0;
    for (u64 k = 0; k < n; ++k) {
        SessionInstance &in = s.inst[ids[k]];
        const u64 *src[3];
        u64 len[3];
        int m = 0;
        for (int r = 0; r < 3; ++r) {
            const u64 b = hb[6 * k + 2 * r], e = hb[6 * k + 2 * r + 1];
            if (e > b) {
                src[m] = runs.w[r] + b;
                len[m] = e - b;
                ++m;
            }
        }
        u64 *dst = block->as<u64>() + at;
        u64 cnt = 0;
        if (m == 1) {
            DL_CUDA(cudaMemcpyAsync(dst, src[0], len[0] * 8, cudaMemcpyDeviceToDevice, ctx.stream));
            cnt = len[0];
        } else if (m == 2) {
            merge_words(ctx, src[0], len[0], src[1], len[1], dst, Codec::Raw);
            cnt = len[0] + len[1];
        } else if (m == 3) {
            merge_words(ctx, src[0], len[0], src[1], len[1], tmp.as<u64>(), Codec::Raw);
            merge_words(ctx, tmp.as<u64>(), len[0] + len[1], src[2], len[2], dst, Codec::Raw);
            cnt = len[0] + len[1] + len[2];
        }
        in.result_block = block;
        in.result_off = at;
        in.n_result = cnt;
        at += cnt;
        s.dead += cnt;
    }
    if (pair_max) {
        ctx.sync();  // the merges that read tmp are done
        ctx.give_back(tmp);
    }
}

void mark_done(SessionImpl &s, SessionInstance &in) {
    in.active = false;
    in.done = true;
    s.finished.push_back(in.id);
}

// Drops the union state once no instance is active: ranks, offsets and the
// full relation start again from zero (results live with their instances).
void reset_if_idle(SessionImpl &s) {
    if (!s.active.empty()) return;
    s.next_rank = 0;
    s.n_vals = 0;
    s.F = FullSet();
    s.F.three = true;
    s.dead = 0;
    s.n_delta = 0;
    s.inst_dirty = true;
}

// Words whose key rank lies in an active instance's range.
struct KeepLive {
    const u64 *lo, *hi;
    u32 n;
    int shift;
    __device__ bool operator()(u64 cur, u64, bool) const {
        const u64 r = cur >> shift;
        const u32 k = instance_of(lo, n, r);
        return k < n && r < hi[k];
    }
};

// Removes the words of finished instances from the full runs once they are
// at least half of the full relation.
void maybe_compact(SessionImpl &s) {
    if (s.active.empty()) return;
    const u64 total = s.F.size();
    if (s.dead == 0 || s.dead * 2 < total) return;
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    upload_active(s);
    KeepLive keep{s.inst_lo.as<u64>(), s.inst_hi.as<u64>(), (u32) s.active.size(), s.bits};
    s.F.nbig = session_select(ctx, ws.full[s.F.cur].as<u64>(), s.F.nbig, keep, 60);
    s.F.nsmall = session_select(ctx, ws.small[s.F.scur].as<u64>(), s.F.nsmall, keep, 60);
    s.F.ntiny = session_select(ctx, ws.tiny[s.F.tcur].as<u64>(), s.F.ntiny, keep, 60);
    s.F.sample_ok = false;
    s.F.ssample_ok = false;
    if (s.F.nsmall == 0) fold_tiny(ctx, s.F);  // a tiny run needs a small run
    s.dead = 0;
}

// The words of a search (ws.jbuf[0], unsorted) in result order, into one block;
// every instance's are one range of it. `sources`: ranks searched when the words are
// those of a TC search alone, else 0.
void place_results(SessionImpl &s, const std::vector<i64> &ids, u64 words, u64 sources) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    const u64 n = ids.size();
    std::vector<u64> hb(6 * n, 0);
    auto block = std::shared_ptr<DevBuf>();
    if (words) {
        const int used = bits_for(std::max<u64>(s.next_rank, 2));
        u64 *r;
        if (sources) {
            r = closure_order(ctx, sources, words, s.bits, used);
        } else {
            ctx.reserve(ws.jbuf[1], words * 8);
            int w[8];
            const int nw = plan_windows(s.bits, used, w);
            r = radix_sort_windows(ctx, ws.jbuf[0].as<u64>(), ws.jbuf[1].as<u64>(), words, w, nw);
        }
        upload_ranges(s, ids);
        ctx.reserve(s.counts, 6 * n * 8);
        Runs3 runs{{r, r, r}, {words, 0, 0}};
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_bounds_kernel<<<grid_for(6 * n, 256, ctx, 4), 256, 0, ctx.stream>>>(
                      runs, s.range_lo.as<u64>(), (u32) n, s.bits, s.counts.as<u64>()));
        DL_CUDA(cudaMemcpyAsync(hb.data(), s.counts.p, 6 * n * 8, cudaMemcpyDeviceToHost, ctx.stream));
        DevBuf &held = holder(ws, r);
        if (held.cap <= 2 * words * 8 + (1 << 20)) {  // the sorted buffer becomes the result block
            block = make_block(ctx, 0);
            std::swap(*block, held);
        } else {
            block = make_block(ctx, words * 8);
            DL_CUDA(cudaMemcpyAsync(block->p, r, words * 8, cudaMemcpyDeviceToDevice, ctx.stream));
        }
        ctx.sync();
    }
    for (u64 k = 0; k < n; ++k) {
        SessionInstance &in = s.inst[ids[k]];
        in.result_block = block;
        in.result_off = hb[6 * k];
        in.n_result = hb[6 * k + 1] - hb[6 * k];
    }
}

// SG: the whole fixpoint of the newly admitted instances `ids` (ranks [lo, hi)) as one
// search over pairs (dl_pairs.cu). False (nothing done) when the sorted runs take them:
// their degrees do not suit the search, the runs are faster, or its list and set would pass
// bitmap_max_gib or half of the free memory.
bool search_pairs(SessionImpl &s, const std::vector<i64> &ids, u64 lo, u64 hi) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    const u64 limit = (u64) ctx.tune.bitmap_max_gib << 30;
    if (limit == 0) return false;
    Csr csr;
    csr.off = s.off.as<u32>();
    csr.val = s.val.as<u32>();
    csr.n_keys = (u32) s.next_rank;
    csr.n_vals = s.n_vals;
    const u64 n = ids.size();
    const int stop = s.opt.max_iterations;
    const PairDegrees deg = pair_degrees(ctx, csr, lo, hi);
    if (!deg.fits()) return false;
    std::vector<u64> n_ids(n);
    for (u64 k = 0; k < n; ++k) n_ids[k] = s.inst[ids[k]].n_ids;
    if (pair_search_outrun(deg, n_ids)) return false;
    PairOptions po;
    po.max_levels = stop > 0 ? (u64) stop : 0;
    po.limit = limit;
    PairSearch ps;
    try {
        ps = pair_search(ctx, csr, lo, hi, s.bits, po);
    } catch (const Error &err) {
        if (err.status != DL_ERR_OUT_OF_MEMORY) throw;
        ps.complete = false;
    }
    if (!ps.complete) {
        ctx.give_back(ws.jbuf[0]);  // the list and the set, for whatever the runs need
        ctx.give_back(ws.jbuf[1]);
        return false;
    }
    const u64 levels = ps.bound.size() - 1;
    std::vector<u64> first(n), cnt(n * levels);
    for (u64 k = 0; k < n; ++k) first[k] = s.inst[ids[k]].rank_lo;
    ctx.reserve(s.range_lo, n * 8);
    DL_CUDA(cudaMemcpyAsync(s.range_lo.p, first.data(), n * 8, cudaMemcpyHostToDevice, ctx.stream));
    ctx.reserve(s.counts, n * levels * 8);
    pair_level_counts(ctx, ps, s.bits, s.range_lo.as<u64>(), n, s.counts.as<u64>());
    DL_CUDA(cudaMemcpyAsync(cnt.data(), s.counts.p, n * levels * 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    for (u64 k = 0; k < n; ++k) {
        SessionInstance &in = s.inst[ids[k]];
        in.ahead.clear();
        for (u64 d = 1;; ++d) {  // iteration d finds level d (sg.cu:244-390)
            const i64 c = d < levels ? (i64) cnt[k * levels + d] : 0;
            in.ahead.push_back(c);
            if (c == 0 || (stop > 0 && (int) in.ahead.size() >= stop)) break;
        }
    }
    place_results(s, ids, ps.n_words(), 0);
    return true;
}

// WCC: the fixpoints of the newly admitted instances `ids` (ranks [lo, hi), in
// instance order) and their results: components (ascending local ranks), largest
// component and per-node labels.
void propagate_labels(SessionImpl &s, const std::vector<i64> &ids, u64 lo, u64 hi, u64 edges) {
    if (ids.empty()) return;
    Context &ctx = s.ctx;
    const u64 n = ids.size(), total = hi - lo;
    Csr csr;
    csr.off = s.off.as<u32>();
    csr.val = s.val.as<u32>();
    csr.n_keys = (u32) hi;
    csr.n_vals = edges;
    std::vector<u64> first(n), n_ids(n), off(n + 1);
    for (u64 k = 0; k < n; ++k) {
        first[k] = s.inst[ids[k]].rank_lo;
        n_ids[k] = s.inst[ids[k]].n_ids;
        off[k] = first[k] - lo;
    }
    off[n] = total;
    auto labels = make_block(ctx, total * 4);
    u32 *label = labels->as<u32>();
    WccRun run = wcc_propagate(ctx, csr, lo, hi, first, n_ids, s.opt.wcc_stop, s.opt.max_iterations, label);
    // s.counts: slot offsets [n + 1] then largest [n] then component starts [n]
    ctx.reserve(s.counts, (3 * n + 1) * 8);
    u64 *d_off = s.counts.as<u64>(), *d_big = d_off + n + 1, *d_start = d_big + n;
    DL_CUDA(cudaMemcpyAsync(d_off, off.data(), (n + 1) * 8, cudaMemcpyHostToDevice, ctx.stream));
    DL_CUDA(cudaMemsetAsync(d_big, 0, n * 8, ctx.stream));
    DevBuf cnt, pos;
    ctx.reserve(cnt, total * 4);
    ctx.reserve(pos, total * 8);
    DL_CUDA(cudaMemsetAsync(cnt.p, 0, total * 4, ctx.stream));
    wcc_label_counts(ctx, label, total, (u32) lo, cnt.as<u32>());
    const u64 nc = count_matches(ctx, NonZero{cnt.as<u32>()}, total, pos.as<u64>());
    auto comps = make_block(ctx, nc * 4);
    DL_LAUNCH(ctx, K_PREP, 0,
              session_wcc_comp_kernel<<<grid_for(total, 256, ctx, 8), 256, 0, ctx.stream>>>(
                  cnt.as<u32>(), pos.as<u64>(), d_off, (u32) n, total, comps->as<u32>(),
                  (unsigned long long *) d_big, d_start));
    std::vector<u64> h(2 * n);
    DL_CUDA(cudaMemcpyAsync(h.data(), d_big, 2 * n * 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    for (u64 k = 0; k < n; ++k) {
        SessionInstance &in = s.inst[ids[k]];
        const u64 start = h[n + k], end = k + 1 < n ? h[n + k + 1] : nc;
        in.ahead = std::move(run.deltas[k]);
        in.result_block = comps;
        in.result_off = start;
        in.n_result = end - start;
        in.largest = (i64) h[k];
        in.labels_block = labels;
        in.labels_off = off[k];
    }
    ctx.give_back(cnt);
    ctx.give_back(pos);
}

// TC: the whole fixpoint of the instances admitted since the last step
// (dl_closure.cu: a search per source, whatever the instance, so all of them
// run in one launch), their rows sorted into one block and every iteration's
// |delta|. The steps then only report iteration after iteration.
void search_pending(SessionImpl &s) {
    if (s.pending.empty()) return;
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    const std::vector<i64> ids = s.pending;
    const u64 n = ids.size();
    // first ranks; ranks between two of them that no instance holds (a failed
    // admission's) become an entry of their own
    std::vector<u64> lo, at(n);
    u64 end = s.inst[ids[0]].rank_lo, widest = 1;
    for (u64 k = 0; k < n; ++k) {
        const SessionInstance &in = s.inst[ids[k]];
        if (in.rank_lo != end) lo.push_back(end);
        at[k] = lo.size();
        lo.push_back(in.rank_lo);
        end = in.rank_hi;
        widest = std::max<u64>(widest, in.n_ids);
    }
    const u64 first = lo[0], ni = lo.size(), stride = std::min<u64>(CL_LEVELS, widest) + 1;
    ctx.reserve(s.range_lo, ni * 8);
    DL_CUDA(cudaMemcpyAsync(s.range_lo.p, lo.data(), ni * 8, cudaMemcpyHostToDevice, ctx.stream));
    ctx.reserve(s.counts, ni * stride * 8);
    const u64 max_level = s.opt.max_iterations > 0 ? (u64) s.opt.max_iterations + 1 : 0;
    Csr csr;
    csr.off = s.off.as<u32>();
    csr.val = s.val.as<u32>();
    csr.n_keys = (u32) s.next_rank;
    csr.n_vals = s.n_vals;
    const ClosureLight light = closure_search(ctx, csr, first, end, s.bits, s.range_lo.as<u64>(), ni, s.pending_vals,
                                              s.n_vals, stride, max_level, s.counts.as<u64>(), nullptr);
    const u64 width = light.levels + 1;
    std::vector<u64> hc(ni * width, 0);
    if (light.levels)
        DL_CUDA(cudaMemcpy2DAsync(hc.data(), width * 8, s.counts.p, stride * 8, width * 8, ni, cudaMemcpyDeviceToHost,
                                  ctx.stream));
    std::vector<u64> heavy(light.n_heavy);
    if (light.n_heavy)
        DL_CUDA(cudaMemcpyAsync(heavy.data(), ws.cl_heavy.p, light.n_heavy * 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    std::sort(heavy.begin(), heavy.end());
    u64 words = light.n_words;
    auto hp = heavy.begin();
    for (u64 k = 0; k < n; ++k) {
        SessionInstance &in = s.inst[ids[k]];
        std::vector<u64> cnt(hc.begin() + at[k] * width, hc.begin() + (at[k] + 1) * width);
        hp = std::lower_bound(hp, heavy.end(), in.rank_lo);
        const auto he = std::lower_bound(hp, heavy.end(), in.rank_hi);
        if (he != hp)
            closure_heavy_words(ctx, csr, in.rank_lo, in.rank_hi, s.bits, std::vector<u64>(hp, he), max_level, cnt,
                                words);
        hp = he;
        in.ahead.clear();
        for (u64 d = 2;; ++d) {  // iteration d - 2 finds the targets at distance d (tc.cu:216-314)
            const i64 c = d < cnt.size() ? (i64) cnt[d] : 0;
            in.ahead.push_back(c);
            if (c == 0 || (s.opt.max_iterations > 0 && (int) in.ahead.size() >= s.opt.max_iterations)) break;
        }
    }
    place_results(s, ids, words, words == light.n_words ? end - first : 0);
    s.pending.clear();
}

// Reports one iteration of an instance whose fixpoint was searched ahead;
// true when it was the last.
bool report_ahead(SessionInstance &in) {
    in.deltas.push_back(in.ahead[in.deltas.size()]);
    return in.deltas.size() == in.ahead.size();
}

// One iteration of instances that were computed ahead.
u64 ahead_step(SessionImpl &s) {
    if (s.program == DL_PROGRAM_TC) search_pending(s);
    std::vector<i64> still;
    for (i64 id : s.active) {
        SessionInstance &in = s.inst[id];
        if (report_ahead(in)) mark_done(s, in);
        else still.push_back(id);
    }
    if (still.size() != s.active.size()) {
        s.active = still;
        s.inst_dirty = true;
    }
    reset_if_idle(s);
    return s.active.size();
}

// One SG iteration (sg.cu:244-390): the instances searched ahead report theirs,
// the others (a node of more out-edges than the search takes) advance together
// on the sorted runs.
u64 sg_step(SessionImpl &s) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    u64 nnew = 0;
    std::vector<u64> c(s.active.size(), 0);
    bool runs = false;
    for (i64 id : s.active) runs |= s.inst[id].ahead.empty();
    if (runs) {
        Graph g = union_graph(s);
        PhaseTimer pt(ctx, false);
        u64 *dnew = nullptr;
        u64 n1 = 0, n2 = 0;
        u64 *j1 = join_and_sort(ctx, g, s.delta.as<u64>(), s.n_delta, EmitKind::VZ, n1, nullptr, pt);
        if (n1) n1 = unique_words(ctx, j1, n1, j1);
        if (n1) {
            u64 *j2 = join_and_sort(ctx, g, j1, n1, EmitKind::VZ, n2, nullptr, pt);
            dnew = absorb(ctx, s.F, j2, n2, nnew);
        }
        // the new delta sits in one of the join buffers: trade it for the old delta's buffer
        if (nnew) std::swap(s.delta, holder(ws, dnew));
        s.n_delta = nnew;
        c = delta_counts(s, s.delta.as<u64>(), nnew, s.bits);
    }
    std::vector<i64> still, done, extract;
    std::vector<uint8_t> live(s.active.size(), 1);
    bool rows_left = false;  // an instance stopped by max_iterations keeps rows in the delta
    for (u64 k = 0; k < s.active.size(); ++k) {
        SessionInstance &in = s.inst[s.active[k]];
        bool stop;
        if (!in.ahead.empty()) {
            stop = report_ahead(in);
        } else {
            in.deltas.push_back((i64) c[k]);
            stop = c[k] == 0;  // |full| unchanged
            if (!stop && s.opt.max_iterations > 0 && (int) in.deltas.size() >= s.opt.max_iterations) stop = true;
            if (stop) {
                extract.push_back(s.active[k]);
                live[k] = 0;
                rows_left |= c[k] != 0;
            }
        }
        (stop ? done : still).push_back(s.active[k]);
    }
    if (rows_left && still.size()) {
        upload_active(s);
        ctx.reserve(s.live, live.size());
        DL_CUDA(cudaMemcpyAsync(s.live.p, live.data(), live.size(), cudaMemcpyHostToDevice, ctx.stream));
        KeepActive keep{s.inst_lo.as<u64>(), s.live.as<uint8_t>(), (u32) s.active.size(), s.bits};
        s.n_delta = session_select(ctx, s.delta.as<u64>(), s.n_delta, keep, 61);  // syncs: `live` may go
    }
    if (!extract.empty()) extract_words(s, extract);
    for (i64 id : done) mark_done(s, s.inst[id]);
    if (still.size() != s.active.size()) {
        s.active = still;
        s.inst_dirty = true;
    }
    reset_if_idle(s);
    maybe_compact(s);
    return s.active.size();
}

}  // namespace

SessionImpl *session_create(Context &parent, int program, const dl_options &opt, u64 max_nodes) {
    if (program != DL_PROGRAM_TC && program != DL_PROGRAM_SG && program != DL_PROGRAM_WCC)
        throw Error(DL_ERR_INVALID_ARGUMENT, "sessions run TC, SG or WCC");
    auto s = std::make_unique<SessionImpl>();
    s->program = program;
    s->opt = opt;
    if (program == DL_PROGRAM_WCC) {
        s->bits = 32;
        s->rank_cap = 0xFFFFFFFFull;
    } else {
        // TC/SG words hold two rank fields of `bits` bits; the sorts only
        // visit the bits the ranks in use can set
        s->bits = max_nodes ? std::max(1, bits_for(max_nodes)) : 32;
        if (max_nodes >= 0xFFFFFFFFull) throw Error(DL_ERR_INVALID_ARGUMENT, "max_nodes above 2^32 - 2");
        s->rank_cap = s->bits == 32 ? 0xFFFFFFFFull : (1ull << s->bits);
    }
    Context &c = s->ctx;
    s->parent = &parent;
    c.device = parent.device;
    c.stream = parent.stream;
    c.sm_count = parent.sm_count;
    c.prof_on = parent.prof_on;
    c.tune = parent.tune;
    SessionKit kit;
    if (!parent.kits.empty()) {
        kit = parent.kits.back();
        parent.kits.pop_back();
    } else {
        void *p = nullptr;
        DL_CUDA(cudaMalloc(&p, sizeof(Ctrl)));
        kit.ctrl = (Ctrl *) p;
        const cudaError_t e = cudaMallocHost((void **) &kit.host_scalars, 64 * sizeof(u64));
        if (e != cudaSuccess) {
            kit.release();
            DL_CUDA(e);
        }
    }
    c.ctrl = kit.ctrl;
    c.host_scalars = kit.host_scalars;
    c.epoch = kit.epoch;
    c.lookback = kit.lookback;
    c.sort_hist = kit.sort_hist;
    c.lbs_splits = kit.lbs_splits;
    c.radix_part = kit.radix_part;
    c.merge_splits = kit.merge_splits;
    c.bucket_cursor = kit.bucket_cursor;
    c.host_stage = kit.host_stage;
    c.host_stage_bytes = kit.host_stage_bytes;
    std::memset(c.host_scalars, 0, 64 * sizeof(u64));
    DL_CUDA(cudaMemsetAsync(c.ctrl, 0, sizeof(Ctrl), c.stream));
    c.spares = std::move(parent.spares);  // the parent's cached buffers serve the session
    parent.spares.clear();
    return s.release();
}

void session_destroy(SessionImpl *s) {
    if (!s) return;
    Context &c = s->ctx;
    cudaStreamSynchronize(c.stream);
    c.prof_resolve();
    // Every buffer goes back to the parent context's cache: the next run or
    // session on it reuses the memory instead of allocating it again.
    Context &p = *s->parent;
    for (auto &in : s->inst) {  // blocks return to the session's cache
        in.ids_block.reset();
        in.result_block.reset();
        in.labels_block.reset();
    }
    DevBuf *bufs[] = {&s->off,     &s->val,    &s->delta,    &s->inst_lo,   &s->inst_hi,
                      &s->counts,    &s->live,
                      &s->range_lo, &s->admit_off, &s->admit_first};
    for (DevBuf *b : bufs) p.give_back(*b);
    Workspace &w = c.ws;
    DevBuf *wbufs[] = {&w.input,    &w.ids,      &w.w0,       &w.w1,      &w.csr_off,  &w.csr_val,
                       &w.full[0],  &w.full[1],  &w.small[0], &w.small[1], &w.tiny[0], &w.tiny[1],
                       &w.sample,   &w.sample_small, &w.jbuf[0],
                       &w.jbuf[1],  &w.offsets,  &w.wcc_label, &w.wcc_flag, &w.wcc_next,
                       &w.cl_left,  &w.cl_heavy, &w.cl_seg, &w.cl_seg_at, &w.cl_levels, &w.cl_roff,  &w.cl_rval, &w.cl_segs,
                       &w.cl_hub_at, &w.cl_hub_acc, &w.cl_rows[0], &w.cl_rows[1], &w.cl_act, &w.cl_rec};
    for (DevBuf *b : wbufs) p.give_back(*b);
    for (auto &b : c.spares) p.give_back(b);
    c.spares.clear();
    // the control block, page-locked scalars and scan scratch serve the next session
    SessionKit kit{c.ctrl, c.host_scalars, c.epoch, c.lookback, c.sort_hist, c.lbs_splits, c.radix_part, c.merge_splits,
                   c.bucket_cursor, c.host_stage, c.host_stage_bytes};
    c.host_stage = nullptr;
    c.host_stage_bytes = 0;
    c.lookback = c.sort_hist = c.lbs_splits = c.radix_part = c.merge_splits = c.bucket_cursor = DevBuf();
    if (p.kits.size() < Context::kKits) p.kits.push_back(kit);
    else kit.release();
    c.release_all();  // events
    delete s;
}

std::vector<i64> session_admit_many(SessionImpl &s, const int32_t *const *rows, const u64 *nrows, u64 count,
                                    bool on_device) {
    Context &ctx = s.ctx;
    Workspace &ws = ctx.ws;
    if (count >= (1ull << 31)) throw Error(DL_ERR_INVALID_ARGUMENT, "too many instances in one admission");
    std::vector<u64> off(count + 1, 0);
    for (u64 k = 0; k < count; ++k) off[k + 1] = off[k] + nrows[k];
    const u64 N = off[count];
    const bool tc = s.program == DL_PROGRAM_TC;
    const u64 first_id = s.inst.size();
    std::vector<i64> ids(count);
    for (u64 k = 0; k < count; ++k) {
        s.inst.emplace_back();
        SessionInstance &in = s.inst.back();
        in.id = (i64) (first_id + k);
        in.input_rows = (i64) nrows[k];
        in.rank_lo = in.rank_hi = s.next_rank;
        ids[k] = in.id;
    }
    auto inst = [&](u64 k) -> SessionInstance & { return s.inst[first_id + k]; };
    if (N == 0) {  // no instance enters its loop: zero iterations, empty results
        for (u64 k = 0; k < count; ++k) mark_done(s, inst(k));
        return ids;
    }
    try {
        // every instance's rows, back to back, and their row offsets
        ctx.reserve(ws.input, N * 8);
        for (u64 k = 0; k < count; ++k)
            if (nrows[k])
                DL_CUDA(cudaMemcpyAsync(ws.input.as<int32_t>() + 2 * off[k], rows[k], nrows[k] * 8,
                                        on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, ctx.stream));
        ctx.reserve(s.admit_off, (count + 1) * 8);
        DL_CUDA(cudaMemcpyAsync(s.admit_off.p, off.data(), (count + 1) * 8, cudaMemcpyHostToDevice, ctx.stream));
        const int32_t *in_rows = ws.input.as<int32_t>();
        const u64 *d_off = s.admit_off.as<u64>();
        // distinct (instance, node id) pairs, sorted: position = union rank
        // offset (tc.cu:171-176 ranks nothing; node ids are only renamed)
        const u64 m = 2 * N;
        ctx.reserve(ws.w0, m * 8);
        ctx.reserve(ws.w1, m * 8);
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_tag_kernel<<<grid_for(N, 256, ctx, 16), 256, 0, ctx.stream>>>(in_rows, N, d_off, (u32) count,
                                                                                         ws.w0.as<u64>()));
        u64 nu = 0;
        u64 *u = sort_unique_into(ctx, ws.w0, ws.w1, m, 32 + bits_for(count), nu);
        const u64 B = s.next_rank;
        if (B + nu > s.rank_cap)
            throw Error(DL_ERR_OVERFLOW, "session node capacity exhausted (" + std::to_string(s.rank_cap) + " ranks)");
        DevBuf &wu = ws.w0.p == u ? ws.w0 : ws.w1;
        DevBuf &wo = ws.w0.p == u ? ws.w1 : ws.w0;
        ctx.reserve(s.admit_first, (count + 1) * 8);
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_first_kernel<<<grid_for(count + 1, 256, ctx, 16), 256, 0, ctx.stream>>>(
                      u, nu, (u32) count, s.admit_first.as<u64>()));
        std::vector<u64> first(count + 1);
        DL_CUDA(cudaMemcpyAsync(first.data(), s.admit_first.p, (count + 1) * 8, cudaMemcpyDeviceToHost, ctx.stream));
        // node ids of the admitted ranks, shared by the instances of this admission
        auto block = make_block(ctx, nu * 4);
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_ids_kernel<<<grid_for(nu, 256, ctx, 16), 256, 0, ctx.stream>>>(u, nu, block->as<int32_t>()));
        // rows -> rank words; the edge relation keyed by source (tc.cu:171-176,
        // sg.cu:150-153, wcc.cu:140-167: WCC stores both directions)
        if (tc && s.pending.empty()) s.pending_vals = s.n_vals;
        const int bits = s.bits;
        const bool wcc = s.program == DL_PROGRAM_WCC;
        u64 *fw = wo.as<u64>();
        u64 *rv = wcc ? fw + N : nullptr;
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_pack_many_kernel<<<grid_for(N, 256, ctx, 16), 256, 0, ctx.stream>>>(
                      in_rows, N, d_off, (u32) count, u, nu, B, bits, fw, rv));
        u64 ne = 0;
        const int used = bits_for(std::max<u64>(B + nu, 2));
        u64 *e = sort_unique_fields(ctx, wo, wu, wcc ? m : N, bits, used, ne);
        if (s.n_vals + ne >= (1ull << 32)) throw Error(DL_ERR_OVERFLOW, "session edge capacity exhausted");
        grow_keep(ctx, s.off, (B + nu + 1) * 4, (B + 1) * 4);
        grow_keep(ctx, s.val, (s.n_vals + ne + 1) * 4, s.n_vals * 4);
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_csr_kernel<<<grid_for(std::max<u64>(ne, nu + 1), 256, ctx, 16), 256, 0, ctx.stream>>>(
                      e, ne, bits, B, B + nu, s.n_vals, s.off.as<u32>(), s.val.as<u32>()));
        s.n_vals += ne;
        s.next_rank = B + nu;
        ctx.sync();  // `first` is ready
        for (u64 k = 0; k < count; ++k) {
            SessionInstance &in = inst(k);
            in.rank_lo = B + first[k];
            in.rank_hi = B + first[k + 1];
            in.n_ids = (u32) (first[k + 1] - first[k]);
            in.ids_block = block;
            in.ids_off = first[k];
        }
        std::vector<bool> empty_base(count, false);
        std::vector<i64> with_rows;
        for (u64 k = 0; k < count; ++k)
            if (nrows[k]) with_rows.push_back(inst(k).id);
        if (tc) {
            // searched as a whole in the next step
        } else if (s.program == DL_PROGRAM_SG && search_pairs(s, with_rows, B, B + nu)) {
            for (u64 k = 0; k < count; ++k) empty_base[k] = nrows[k] && inst(k).ahead[0] == 0 && inst(k).n_result == 0;
        } else if (s.program == DL_PROGRAM_SG) {
            // sg.cu:170-217: the base rule of the admitted instances, probing the union table
            Graph g = union_graph(s);
            u64 *selfs = &ctx.ctrl->scalar[30];
            DL_CUDA(cudaMemsetAsync(selfs, 0, 8, ctx.stream));
            u64 nb = 0;
            PhaseTimer pt(ctx, false);
            u64 *b = join_and_sort(ctx, g, e, ne, EmitKind::ZV_NOSELF, nb, selfs, pt);
            DL_CUDA(cudaMemcpyAsync(ctx.host_scalars + 5, selfs, 8, cudaMemcpyDeviceToHost, ctx.stream));
            ctx.sync();
            const u64 nv = nb - ctx.host_scalars[5];  // self pairs sorted to the end
            const u64 nd = nv ? unique_words(ctx, b, nv, b) : 0;
            std::vector<u64> lo(count);
            for (u64 k = 0; k < count; ++k) lo[k] = inst(k).rank_lo;
            const std::vector<u64> c = range_counts(s, b, nd, bits, lo);
            for (u64 k = 0; k < count; ++k) empty_base[k] = c[k] == 0;
            full_insert_new(s, b, nd);
            delta_append(s, b, nd);
        } else {  // wcc.cu:211-231: cc(n, n) for every node, all nodes in the first delta
            propagate_labels(s, with_rows, B, B + nu, ne);
        }
        ctx.sync();
        for (u64 k = 0; k < count; ++k) {
            SessionInstance &in = inst(k);
            if (nrows[k] == 0) {
                mark_done(s, in);
            } else if (empty_base[k]) {  // the loop runs once on an empty delta (sg.cu:244-390)
                in.deltas.push_back(0);
                mark_done(s, in);
            } else {
                in.active = true;
                s.active.push_back(in.id);
                if (tc) s.pending.push_back(in.id);
            }
        }
        s.inst_dirty = true;
    } catch (...) {
        // the union tables may hold part of these instances; their ranks are never reused
        for (u64 k = 0; k < count; ++k) {
            inst(k).done = true;
            inst(k).released = true;
        }
        throw;
    }
    return ids;
}

i64 session_admit(SessionImpl &s, const int32_t *rows, u64 n, bool on_device) {
    return session_admit_many(s, &rows, &n, 1, on_device)[0];
}

u64 session_step(SessionImpl &s) {
    if (s.active.empty()) return 0;
    return s.program == DL_PROGRAM_SG ? sg_step(s) : ahead_step(s);
}

u64 session_poll(SessionImpl &s, int64_t *ids, u64 capacity) {
    const u64 n = std::min<u64>(capacity, s.finished.size());
    for (u64 i = 0; i < n; ++i) ids[i] = s.finished[i];
    s.finished.erase(s.finished.begin(), s.finished.begin() + (std::ptrdiff_t) n);
    return n;
}

void session_fold_profile(SessionImpl &s, Context &parent) {
    s.ctx.sync();  // resolves the timed launches
    for (int k = 0; k < K_COUNT; ++k) {
        KernelStat &a = parent.kstat[k];
        KernelStat &b = s.ctx.kstat[k];
        a.launches += b.launches;
        a.timed += b.timed;
        a.seconds += b.seconds;
        a.bytes += b.bytes;
        b = KernelStat();
    }
    s.ctx.prof_on = parent.prof_on;
}

const SessionInstance &session_instance(const SessionImpl &s, i64 id) {
    if (id < 0 || id >= (i64) s.inst.size()) throw Error(DL_ERR_INVALID_ARGUMENT, "unknown instance " + std::to_string(id));
    return s.inst[id];
}

void session_info(const SessionImpl &s, i64 id, dl_run_info &info) {
    const SessionInstance &in = session_instance(s, id);
    std::memset(&info, 0, sizeof(info));
    info.program = s.program;
    info.iterations = (int32_t) in.deltas.size();
    info.input_rows = in.input_rows;
    info.output_rows = info.output_tuples = in.done ? (i64) in.n_result : 0;
    info.largest_component = in.done ? in.largest : 0;
    info.nodes = in.n_ids;
}

static SessionInstance &finished_instance(SessionImpl &s, i64 id) {
    session_instance(s, id);
    SessionInstance &in = s.inst[id];
    if (!in.done) throw Error(DL_ERR_INVALID_ARGUMENT, "instance " + std::to_string(id) + " has not finished");
    if (in.released) throw Error(DL_ERR_INVALID_ARGUMENT, "instance " + std::to_string(id) + " was released");
    return in;
}

// Rows of a finished instance into device memory (no wait).
static void unpack_result(SessionImpl &s, const SessionInstance &in, int32_t *out) {
    Context &ctx = s.ctx;
    const u64 n = in.n_result;
    const int32_t *ids = in.ids();
    const unsigned g = grid_for(n, 256, ctx, 16);
    if (s.program == DL_PROGRAM_WCC)
        DL_LAUNCH(ctx, K_PREP, 0, session_unpack_comp_kernel<<<g, 256, 0, ctx.stream>>>(in.result_u32(), n, ids, out));
    else if (s.program == DL_PROGRAM_SG)
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_unpack_kernel<true><<<g, 256, 0, ctx.stream>>>(in.result_words(), n, s.bits, in.rank_lo,
                                                                          ids, out));
    else
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_unpack_kernel<false><<<g, 256, 0, ctx.stream>>>(in.result_words(), n, s.bits, in.rank_lo,
                                                                           ids, out));
}

void session_copy_outputs(SessionImpl &s, const i64 *ids, u64 count, int32_t *const *dst, const i64 *capacity,
                          bool on_device) {
    Context &ctx = s.ctx;
    u64 largest = 0, total = 0;
    for (u64 k = 0; k < count; ++k) {
        const u64 n = finished_instance(s, ids[k]).n_result;
        if ((u64) capacity[k] < n) throw Error(DL_ERR_INVALID_ARGUMENT, "output capacity too small");
        largest = std::max(largest, n);
        total += n;
    }
    if (total == 0) return;
    if (on_device) {
        for (u64 k = 0; k < count; ++k)
            if (s.inst[ids[k]].n_result) unpack_result(s, s.inst[ids[k]], dst[k]);
        ctx.sync();
        return;
    }
    DevBuf stage;
    ctx.reserve(stage, largest * 8);
    for (u64 k = 0; k < count; ++k) {
        const u64 n = s.inst[ids[k]].n_result;
        if (!n) continue;
        unpack_result(s, s.inst[ids[k]], stage.as<int32_t>());
        DL_CUDA(cudaMemcpyAsync(dst[k], stage.p, n * 8, cudaMemcpyDeviceToHost, ctx.stream));
    }
    ctx.sync();
    ctx.give_back(stage);
}

void session_copy_output(SessionImpl &s, i64 id, int32_t *dst, u64 capacity, bool on_device) {
    const i64 cap = (i64) capacity;
    session_copy_outputs(s, &id, 1, &dst, &cap, on_device);
}

void session_copy_labels_many(SessionImpl &s, const i64 *ids, u64 count, int32_t *const *node_ids,
                              int32_t *const *labels, const i64 *capacity) {
    u64 total = 0;
    for (u64 k = 0; k < count; ++k) {
        const SessionInstance &in = finished_instance(s, ids[k]);
        if ((u64) capacity[k] < in.n_ids) throw Error(DL_ERR_INVALID_ARGUMENT, "label capacity too small");
        total += in.n_ids;
    }
    if (s.program != DL_PROGRAM_WCC) throw Error(DL_ERR_INVALID_ARGUMENT, "labels exist only for WCC sessions");
    if (total == 0) return;
    // [node ids, labels] of every instance on the device, then to the host: in one
    // page-locked copy while that is small, else straight to the destinations
    Context &ctx = s.ctx;
    DevBuf stage;
    ctx.reserve(stage, total * 8);
    int32_t *at = stage.as<int32_t>();
    for (u64 k = 0; k < count; ++k) {
        const SessionInstance &in = s.inst[ids[k]];
        const u64 n = in.n_ids;
        if (!n) continue;
        DL_CUDA(cudaMemcpyAsync(at, in.ids(), n * 4, cudaMemcpyDeviceToDevice, ctx.stream));
        DL_LAUNCH(ctx, K_PREP, 0,
                  session_unpack_labels_kernel<<<grid_for(n, 256, ctx, 16), 256, 0, ctx.stream>>>(
                      in.labels(), in.rank_lo, n, in.ids(), at + n));
        at += 2 * n;
    }
    int32_t *host = (int32_t *) ctx.host_staging(total * 8);
    if (host) {
        DL_CUDA(cudaMemcpyAsync(host, stage.p, total * 8, cudaMemcpyDeviceToHost, ctx.stream));
        ctx.sync();
    }
    at = host ? host : stage.as<int32_t>();
    for (u64 k = 0; k < count; ++k) {
        const u64 n = s.inst[ids[k]].n_ids;
        if (!n) continue;
        if (host) {
            std::memcpy(node_ids[k], at, n * 4);
            std::memcpy(labels[k], at + n, n * 4);
        } else {
            DL_CUDA(cudaMemcpyAsync(node_ids[k], at, n * 4, cudaMemcpyDeviceToHost, ctx.stream));
            DL_CUDA(cudaMemcpyAsync(labels[k], at + n, n * 4, cudaMemcpyDeviceToHost, ctx.stream));
        }
        at += 2 * n;
    }
    if (!host) ctx.sync();
    ctx.give_back(stage);
}

void session_copy_labels(SessionImpl &s, i64 id, int32_t *node_ids, int32_t *labels, u64 capacity) {
    const i64 cap = (i64) capacity;
    session_copy_labels_many(s, &id, 1, &node_ids, &labels, &cap);
}

void session_release(SessionImpl &s, i64 id) {
    SessionInstance &in = finished_instance(s, id);
    in.result_block.reset();  // each block goes with its last instance
    in.labels_block.reset();
    in.ids_block.reset();
    in.released = true;
}

u64 session_device_bytes(const SessionImpl &s) {
    const Context &c = s.ctx;
    const Workspace &w = c.ws;
    u64 b = 0;
    const DevBuf *bufs[] = {&s.off,     &s.val,       &s.delta,
                            &w.input,   &w.ids,       &w.w0,       &w.w1,         &w.csr_off,    &w.csr_val,
                            &w.full[0], &w.full[1],   &w.small[0], &w.small[1],   &w.tiny[0],    &w.tiny[1],
                            &w.sample,  &w.sample_small, &w.jbuf[0],
                            &w.jbuf[1], &w.offsets,   &c.lookback, &c.radix_part, &c.lbs_splits, &c.sort_hist,
                            &c.merge_splits, &w.cl_left, &w.cl_heavy, &w.cl_seg, &w.cl_seg_at, &w.cl_levels, &w.cl_roff, &w.cl_rval, &w.cl_segs,
                            &w.cl_hub_at, &w.cl_hub_acc, &w.cl_rows[0], &w.cl_rows[1], &w.cl_act, &w.cl_rec,
                            &w.wcc_label, &w.wcc_flag, &w.wcc_next};
    for (const DevBuf *x : bufs) b += x->cap;  // cached spare buffers are not counted: they are free memory
    std::vector<const DevBuf *> blocks;
    for (const auto &in : s.inst)
        for (const DevBuf *x : {in.ids_block.get(), in.result_block.get(), in.labels_block.get()})
            if (x && std::find(blocks.begin(), blocks.end(), x) == blocks.end()) blocks.push_back(x);
    for (const DevBuf *x : blocks) b += x->cap;
    return b;
}

u64 session_active(const SessionImpl &s) { return s.active.size(); }
u64 session_instance_count(const SessionImpl &s) { return s.inst.size(); }

}  // namespace dl
