// TC as one breadth-first search per source.
//
// The reference's TC is left-linear: an iteration joins the newest paths
// (x, y) with the edges (y, w) and keeps the pairs not seen before
// (tc.cu:216-314), so Delta_k holds exactly the pairs (x, w) at distance k + 1
// and the join output of an iteration is the out-edges of the newest pairs'
// targets. Both depend on one source x at a time: every source's fixpoint is
// its own breadth-first search, with no other source's state in it. A whole
// run is then one launch of independent searches instead of a launch, a full
// relation in HBM and a host wait per iteration, and the per-iteration sizes
// are sums of the searches' level sizes.
//
// Two kinds of work, by what a source reaches:
//  * closure_group_kernel / closure_warp_kernel / closure_cta_kernel: a search
//    whose visited set fits in shared memory (a hash set and the visit queue: up
//    to 255 targets for eight lanes, 1024 for a warp, 4096 for a CTA; a source
//    that outgrows one goes to the next). Result pairs leave as words, sorted
//    afterwards.
//  * closure_pull_kernel: the sources that reach more ("heavy"), 32 of them
//    to a word: bit c of row z of T says whether heavy source c reaches z.
//    One iteration ORs, for every target z, the newest bits of its
//    in-neighbours and keeps the bits T does not have: whole 128-byte lines
//    (1024 sources) for one edge instead of one operation per source. Heavy
//    sources reach much of the graph, so their rows share most edges.
//
// Measured on B200 against the n x n bit matrix stepped by one launch per
// iteration (dl_bitmap.cu), edges and result rows on the device: Chung-Lu graph
// of 317K nodes (1.88e9 pairs; 9.3K heavy sources hold 99 % of them)
// 45.5 -> 11.5 ms; DAG of 500K edges (2.5e7 pairs, 175 iterations) 89 -> 3.6 ms
// (with a warp for every source a millisecond more); DAG of 5.5K edges from and to
// host memory 3.5 -> 0.53 ms.
#include <cstring>
#include <type_traits>

#include "dl_closure.h"
#include "dl_pull.cuh"
#include "dl_scan.cuh"

namespace dl {
namespace detail {
namespace {

// Counters of a search launch (device).
struct SearchCounters {
    unsigned long long fetch;   // next source (group)
    unsigned long long words;   // result words reserved
    unsigned long long left;    // sources left over
    unsigned long long levels;  // largest level of a finished source
    unsigned long long kept;    // eight-lane searches: first word that did not fit (all ones: all did)
};

// Where a launch's words go. Finished sources leave theirs in any order;
// seg[source - lo] = (first word << 16) | words says where (a search holds at most
// 4096), so that closure_order can line them up.
struct SearchOut {
    u64 *out;
    u64 cap;   // room, in words
    u64 base;  // words before `out`
    u64 *seg;
    __device__ __forceinline__ void note(u64 s, u64 p, u32 n) const { seg[s] = (base + p) << 16 | n; }
};

__device__ __forceinline__ u32 hash_slot(u32 w, int shift) { return (w * 2654435769u) >> shift; }

// Adds w to an open-addressing set of MASK + 1 slots that always has empty
// ones; true when it was not there.
template <u32 MASK>
__device__ __forceinline__ bool set_insert(u32 *hash, u32 w, int shift) {
    u32 s = hash_slot(w, shift);
    for (;;) {
        const u32 o = atomicCAS(&hash[s], EMPTY, w);
        if (o == EMPTY) return true;
        if (o == w) return false;
        s = (s + 1) & MASK;
    }
}

// Instance of rank x: the last one whose first rank is at most x.
__device__ __forceinline__ u32 instance_at(const u64 *__restrict__ inst_lo, u32 n_inst, u64 x) {
    u32 a = 0, b = n_inst;
    while (a < b) {
        const u32 m = (a + b) >> 1;
        if (inst_lo[m] <= x) a = m + 1;
        else b = m;
    }
    return a - 1;
}

// Level counts of finished searches, summed in a warp's registers (lane l holds
// levels 32 j + l + 1) and added to the instance's counters when it changes.
constexpr int LV_REGS = 4;
struct LevelSums {
    u32 rc[LV_REGS], rd[LV_REGS];
    u32 held, inst;
    u64 lo, end;  // ranks of the instance
    __device__ void init(bool one, u64 hi) {
#pragma unroll
        for (int j = 0; j < LV_REGS; ++j) rc[j] = rd[j] = 0;
        held = inst = 0;
        lo = 0;
        end = one ? ~0ull : 0;
    }
    __device__ void flush(unsigned long long *cnt, unsigned long long *deg, u32 stride, u32 lane) {
        const u64 at = (u64) inst * stride + 1 + lane;
#pragma unroll
        for (int j = 0; j < LV_REGS; ++j) {
            if (rc[j]) atomicAdd(cnt + at + 32 * j, (unsigned long long) rc[j]);
            if (deg && rd[j]) atomicAdd(deg + at + 32 * j, (unsigned long long) rd[j]);
            rc[j] = rd[j] = 0;
        }
        held = 0;
    }
    // What is added next is of source x's instance. All lanes.
    __device__ void enter(u64 x, const u64 *__restrict__ inst_lo, u32 n_inst, unsigned long long *cnt,
                          unsigned long long *deg, u32 stride, u32 lane) {
        if (x >= lo && x < end) return;
        flush(cnt, deg, stride, lane);
        inst = instance_at(inst_lo, n_inst, x);
        lo = inst_lo[inst];
        end = inst + 1 < n_inst ? inst_lo[inst + 1] : ~0ull;
    }
    // `searches` of at most three levels at once (n[d]: targets of level d + 1), whose targets
    // of all levels but the last have one out-edge each and those of the last one none.
    __device__ void add_tiny(u32 searches, const u32 (&n)[3], unsigned long long *cnt, unsigned long long *deg,
                             u32 stride, u32 lane) {
        if (lane < 3) {
            rc[0] += lane == 0 ? n[0] : lane == 1 ? n[1] : n[2];
            rd[0] += lane == 0 ? n[1] : lane == 1 ? n[2] : 0u;
        }
        if ((held += searches) >= (1u << 16)) flush(cnt, deg, stride, lane);
    }
    // The levels of a search from x: sizes lc[0 .. levels), join words ld[...]. All lanes.
    template <class C>
    __device__ void add(u64 x, u32 levels, const C *lc, const unsigned short *ld,
                        const u64 *__restrict__ inst_lo, u32 n_inst, unsigned long long *cnt, unsigned long long *deg,
                        u32 stride, u32 lane) {
        enter(x, inst_lo, n_inst, cnt, deg, stride, lane);
#pragma unroll
        for (int j = 0; j < LV_REGS; ++j) {
            const u32 k = 32 * j + lane;
            if (k < levels) {
                rc[j] += lc[k];
                rd[j] += ld[k];
            }
        }
        for (u32 k = 32 * LV_REGS + lane; k < levels; k += 32) {
            const u64 at = (u64) inst * stride + 1 + k;
            atomicAdd(cnt + at, (unsigned long long) lc[k]);
            if (deg) atomicAdd(deg + at, (unsigned long long) ld[k]);
        }
        if (++held >= (1u << 16)) flush(cnt, deg, stride, lane);  // 2^16 searches x 2^16 words fit 32 bits
    }
};

// ---- searches by eight lanes --------------------------------------------
//
// Most searches are thin -- a DAG's levels hold two or three targets -- so a
// warp runs four at a time, eight lanes each, in lockstep: every pass of the
// loop takes up to eight frontier rows or eight of their edges per search. An
// edge record brings its target's row along, so a level costs one dependent
// global load. Bound by the latency of a pass times the searches the shared
// memory holds, so a search is packed into 2.8 KB: the visited set is a table of
// one-byte places in the queue, and a target with one in-edge is not looked up
// at all (only the node it comes from could have brought it).
constexpr int CG_THREADS = 64;
constexpr u32 CG_REACH = 255;      // places 0 .. 254; 255 marks an empty slot
constexpr u32 CG_HASH = 512;
constexpr int CG_HASH_SHIFT = 23;  // 32 - log2(CG_HASH)
constexpr u32 CG_LEVELS = 96;
constexpr u32 CG_EDGES = 4096;     // join words of one search
constexpr u32 CG_WIDE = 48;        // a source's or eight rows' edges above which a warp is the better form
constexpr u64 CG_MAX_EDGES = 1ull << 25;
constexpr u64 CL_FEW = 8192;       // sources that go to the warps at once

struct CgSmem {
    unsigned char hash[CG_HASH];
    u32 qw[CG_REACH + 1];             // targets in visiting order
    u32 qr[CG_REACH + 1];             // their rows (record format)
    unsigned short ld[CG_LEVELS];     // join words out of level d at [d - 1]
    unsigned char lc[CG_LEVELS];      // targets of level d at [d - 1]
};
static_assert(sizeof(CgSmem) % 16 == 0, "the table is cleared 16 bytes a lane");

// Edge records, 8 bytes: the target, and its row: first edge (25 bits, from
// k0), whether it has several in-edges (bit 6), degree (6 bits; 63: wide).
constexpr u32 ROW_WIDE = 63;

// flags[w - lo]: 1 when w has an in-edge, 3 when it has several.
__global__ void in_edges_kernel(const u32 *__restrict__ val, u64 k0, u64 k1, u64 lo, u32 *flags) {
    for (u64 k = k0 + (u64) blockIdx.x * blockDim.x + threadIdx.x; k < k1; k += (u64) gridDim.x * blockDim.x) {
        u32 *f = flags + (val[k] - lo);
        if (*reinterpret_cast<volatile u32 *>(f) == 3u) continue;
        if (atomicOr(f, 1u)) atomicOr(f, 3u);
    }
}

__global__ void edge_records_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val, u64 k0, u64 k1, u64 lo,
                                    const u32 *__restrict__ flags, uint2 *__restrict__ rec) {
    for (u64 k = k0 + (u64) blockIdx.x * blockDim.x + threadIdx.x; k < k1; k += (u64) gridDim.x * blockDim.x) {
        const u32 w = val[k];
        const u32 b = off[w], d = off[w + 1] - b;
        const u32 first = d ? b - (u32) k0 : 0u;  // (a sink's row may lie past the last edge)
        rec[k - k0] = make_uint2(w, (first << 7) | (flags[w - lo] == 3u ? 64u : 0u) | min(d, ROW_WIDE));
    }
}

constexpr u32 TINY_PATH = 3;  // targets of a path a lane follows
constexpr u32 TINY_ROW = 4;   // edges of a row whose targets are all sinks

// The sources of a batch (this lane's: x, edges [bb, bb + bd)) whose result a lane sees by itself:
// a path of up to TINY_PATH targets that ends in a sink, or up to TINY_ROW targets that
// are all sinks. Returns them as lane bits, with their words and levels out. A search by
// eight lanes has 0.7 ns of turns and synchronisation whatever it finds, and the sorted
// runs did shallow graphs in a few passes: 8M edges into 8M sinks 2.8 ms by runs, 8.2 by
// searches alone, 2.6 with these; a DAG of 500K edges, few of whose sources are such, is not slower.
__device__ u32 tiny_searches(const uint2 *__restrict__ rec, u32 bb, u32 bd, u64 x, int bits, LevelSums &sums,
                             unsigned long long *__restrict__ cnt, unsigned long long *__restrict__ deg, u32 stride,
                             u32 lane, const SearchOut &to, u64 xb, SearchCounters *__restrict__ ctr, u32 &top) {
    static_assert(TINY_PATH < TINY_ROW, "w[] holds a path");
    u32 w[TINY_ROW], n = 0, levels = 0;
    bool ok = bd >= 1 && bd <= TINY_ROW && x >= sums.lo && x < sums.end;
    if (ok && bd == 1) {
        u32 at = bb;
#pragma unroll
        for (u32 k = 0; k < TINY_PATH; ++k) {
            if (levels) continue;
            const uint2 r = __ldg(rec + at);
            bool seen = r.x == (u32) x;
#pragma unroll
            for (u32 j = 0; j < k; ++j) seen |= w[j] == r.x;
            w[k] = r.x;
            n = k + 1;
            const u32 d = r.y & 63u;
            if (seen || d > 1) ok = false;
            if (d != 1 || !ok) levels = k + 1;  // the path ends
            at = r.y >> 7;
        }
        if (!levels) ok = false;  // it goes on
    } else if (ok) {
        levels = 1;
        n = bd;
#pragma unroll
        for (u32 k = 0; k < TINY_ROW; ++k)
            if (k < bd) {
                const uint2 r = __ldg(rec + bb + k);
                w[k] = r.x;
                if ((r.y & 63u) || r.x == (u32) x) ok = false;
            }
    }
    const u32 all = __ballot_sync(0xffffffffu, ok);
    if (!all) return 0;
    if (!ok) n = levels = 0;
    const u32 incl = warp_inclusive_sum(n);
    const u32 total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long p = 0;
    if (lane == 0) p = atomicAdd(&ctr->words, (unsigned long long) total);
    p = __shfl_sync(0xffffffffu, p, 0);
    if (p + total > to.cap) {  // no room: to the searches, which leave them over
        if (lane == 0) atomicMin(&ctr->kept, p);
        return 0;
    }
    const u32 two = __popc(__ballot_sync(0xffffffffu, levels >= 2));
    const u32 three = __popc(__ballot_sync(0xffffffffu, levels >= 3));
    const u32 counts[3] = {total - two - three, two, three};
    sums.add_tiny(__popc(all), counts, cnt, deg, stride, lane);
    top = max(top, three ? 3u : two ? 2u : 1u);
    if (ok) {
        const u64 q = p + incl - n;
        to.note(xb + lane, q, n);
#pragma unroll
        for (u32 k = 0; k < TINY_ROW; ++k)
            if (k < n) to.out[q + k] = ((u64) w[k] << bits) | x;
    }
    return all;
}

// Searches from the sources of [lo, hi), `batch` (at most 32) consecutive ones
// per warp at a time. `rec` holds the records of edges k0 and up.
__global__ void __launch_bounds__(CG_THREADS)
closure_group_kernel(const u32 *__restrict__ off, const uint2 *__restrict__ rec, u32 k0, u64 lo, u64 hi, u32 batch,
                     int bits, const u64 *__restrict__ inst_lo, u32 n_inst, u32 stride, u32 max_level,
                     unsigned long long *__restrict__ cnt, unsigned long long *__restrict__ deg,
                     SearchOut to, SearchCounters *__restrict__ ctr, u64 *__restrict__ left) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const u32 lane = threadIdx.x & 31, l = lane & 7, g8 = lane & 24;
    CgSmem *const all = reinterpret_cast<CgSmem *>(smem_raw) + (threadIdx.x >> 5) * 4;
    CgSmem &s = all[lane >> 3];
    LevelSums sums;
    sums.init(inst_lo == nullptr, hi);
    u32 top = 0;
    // the warp's current batch of sources: first edge and degree in the lanes
    u64 xb = 0;
    u32 bb = 0, bd = 0, bm = 0;
    bool more = true;
    // the group's search
    bool act = false, done = true, over = false;
    u32 x = 0, head = 0, end = 0, tail = 0, level = 0, rp = 0, tot = 0, ip = 0, edges = 0, led = 0;
    u32 cb = 0, incl = 0, pre = 0;
    for (;;) {
        // ---- finished searches: result, next source (one group at a time, all lanes) ----
        u32 fin = __ballot_sync(0xffffffffu, l == 0 && (done || over));
        while (fin) {
            const u32 q = __ffs(fin) - 1;
            fin &= fin - 1;
            CgSmem &sq = all[q >> 3];
            const bool was = __shfl_sync(0xffffffffu, act, q), ov = __shfl_sync(0xffffffffu, over, q);
            const u32 xq = __shfl_sync(0xffffffffu, x, q), tq = __shfl_sync(0xffffffffu, tail, q);
            bool fits = was && !ov;
            unsigned long long p = 0;
            if (fits) {
                if (lane == 0) p = atomicAdd(&ctr->words, (unsigned long long) tq);
                p = __shfl_sync(0xffffffffu, p, 0);
                fits = p + tq <= to.cap;
                if (!fits && lane == 0) atomicMin(&ctr->kept, p);
            }
            if (fits) {
                const u32 lq = __shfl_sync(0xffffffffu, level, q);
                top = max(top, lq);
                sums.add(lo + xq, lq, sq.lc, sq.ld, inst_lo, n_inst, cnt, deg, stride, lane);
                if (lane == 0) to.note(xq, p, tq);
                for (u32 k = lane; k < tq; k += 32) to.out[p + k] = ((u64) sq.qw[k] << bits) | (lo + xq);
            } else if (was && lane == 0) {
                left[atomicAdd(&ctr->left, 1ull)] = lo + xq;
                to.note(xq, 0, 0);
            }
            while (bm == 0 && more) {
                unsigned long long f = ~0ull;  // (no further sources once the room is full)
                if (lane == 0 && *reinterpret_cast<volatile unsigned long long *>(&ctr->words) <= to.cap)
                    f = atomicAdd(&ctr->fetch, (unsigned long long) batch);
                xb = __shfl_sync(0xffffffffu, f, 0);
                if (xb >= hi - lo) {
                    more = false;
                    break;
                }
                bb = bd = 0;
                if (lane < batch && lo + xb + lane < hi) {
                    bb = __ldg(off + lo + xb + lane);
                    bd = __ldg(off + lo + xb + lane + 1) - bb;
                    bb -= k0;
                }
                bm = __ballot_sync(0xffffffffu, bd != 0);
                if (max_level == 0 || max_level > TINY_PATH) {
                    const u32 first = __ffs(bm) - 1;
                    if (bm) sums.enter(lo + xb + first, inst_lo, n_inst, cnt, deg, stride, lane);
                    bm &= ~tiny_searches(rec, bb, bd, lo + xb + lane, bits, sums, cnt, deg, stride, lane, to, xb, ctr, top);
                }
            }
            const bool mine = g8 == q;
            if (bm) {
                const u32 j = __ffs(bm) - 1;
                bm &= bm - 1;
                const u32 b = __shfl_sync(0xffffffffu, bb, j), d = __shfl_sync(0xffffffffu, bd, j);
                reinterpret_cast<uint4 *>(sq.hash)[lane] = make_uint4(EMPTY, EMPTY, EMPTY, EMPTY);
                if (mine) {  // level 0: one row, the source's
                    x = (u32) (xb + j);
                    act = true;
                    done = false;
                    over = d > CG_WIDE;
                    head = end = tail = level = rp = ip = edges = led = 0;
                    tot = over ? 0 : d;
                    cb = b;
                    pre = l == 0 ? 0u : tot;
                    incl = tot;
                }
                if (d > CG_WIDE) fin |= 1u << q;  // handed over at once
            } else if (mine) {
                act = false;
                done = over = false;
                tot = ip = 0;
            }
            __syncwarp();
        }
        if (!__any_sync(0xffffffffu, act)) break;
        // ---- rows: the next eight of the frontier, or the next level ----
        const bool need = act && ip >= tot;
        if (__any_sync(0xffffffffu, need)) {
            u32 d = 0;
            if (need) {
                rp += 8;
                if (rp >= end) {  // the level is expanded
                    if (level && l == 0) {
                        s.lc[level - 1] = (unsigned char) (end - head);
                        s.ld[level - 1] = (unsigned short) led;
                    }
                    if (tail == end) {
                        done = true;
                    } else {
                        head = rp = end;
                        end = tail;
                        led = 0;
                        if (++level > CG_LEVELS) {
                            over = true;
                        } else if (level == max_level) {
                            if (l == 0) {
                                s.lc[level - 1] = (unsigned char) (end - head);
                                s.ld[level - 1] = 0;
                            }
                            done = true;
                        }
                    }
                }
                ip = tot = 0;
                if (!done && !over && rp + l < end) {
                    const u32 r = s.qr[rp + l];
                    cb = r >> 7;
                    d = r & 63u;
                }
            }
            u32 v = d;
#pragma unroll
            for (u32 o = 1; o < 8; o <<= 1) {
                const u32 y = __shfl_up_sync(0xffffffffu, v, o, 8);
                if (l >= o) v += y;
            }
            const u32 t = __shfl_sync(0xffffffffu, v, 7, 8);
            if (need && !done && !over) {
                incl = v;
                pre = v - d;
                tot = t;
                if (t > CG_WIDE || edges + t > CG_EDGES) over = true;
            }
        }
        // ---- edges: eight of the rows' ----
        const u32 p = ip + l;
        const bool have = act && !done && !over && p < tot;
        u32 o = 0;
        if (__shfl_sync(0xffffffffu, incl, 3, 8) <= p) o = 4;
        if (__shfl_sync(0xffffffffu, incl, o + 1, 8) <= p) o += 2;
        if (__shfl_sync(0xffffffffu, incl, o, 8) <= p) o += 1;
        const u32 at = __shfl_sync(0xffffffffu, cb, o, 8) + (p - __shfl_sync(0xffffffffu, pre, o, 8));
        uint2 r = make_uint2(0, 0);
        if (have) r = __ldg(rec + at);
        // New targets take places in the queue: those with one in-edge at
        // once, the others when the table does not hold them.
        bool fresh = have && !(r.y & 64u), look = have && (r.y & 64u);
        // a source that reaches itself would bring its targets a second time
        const bool bad = have && (r.x == (u32) lo + x || (r.y & 63u) == ROW_WIDE);
        if (((__ballot_sync(0xffffffffu, bad) >> g8) & 0xFFu) != 0) {
            over = true;
            fresh = look = false;
        }
        u32 slot = 0;
        bool put = false;  // this round's new one goes into the table
        for (u32 h = hash_slot(r.x, CG_HASH_SHIFT);;) {
            const u32 gm = (__ballot_sync(0xffffffffu, fresh) >> g8) & 0xFFu;
            const u32 n = __popc(gm);
            if (tail + n > CG_REACH) {
                over = true;
                fresh = look = put = false;
            }
            if (fresh) {
                const u32 k = tail + __popc(gm & ((1u << l) - 1));
                s.qw[k] = r.x;
                s.qr[k] = r.y;
                if (put) s.hash[slot] = (unsigned char) k;
            }
            if (!over) tail += n;
            fresh = put = false;
            __syncwarp();
            if (!__any_sync(0xffffffffu, look)) break;
            // a step of the probe: found, occupied by another, or empty: then the
            // lanes that want the slot write their number and the one that stays has it
            const u32 e = look ? s.hash[h] : 0u;
            const bool empty = look && e == 255u;
            if (look && !empty) {
                if (s.qw[e] == r.x) look = false;
                else h = (h + 1) & (CG_HASH - 1);
            }
            __syncwarp();
            if (empty) s.hash[h] = (unsigned char) l;
            __syncwarp();
            const u32 win = empty ? s.hash[h] : l;
            const u32 ww = __shfl_sync(0xffffffffu, r.x, win, 8);
            __syncwarp();
            if (empty) {
                if (win == l) {
                    fresh = put = true;
                    slot = h;
                    look = false;
                } else if (ww == r.x) {
                    look = false;
                }
            }
        }
        if (act && !done && !over) {
            edges += min(8u, tot - ip);
            led += min(8u, tot - ip);
            ip += 8;
        }
    }
    sums.flush(cnt, deg, stride, lane);
    if (lane == 0 && top) atomicMax(&ctr->levels, (unsigned long long) top);
}

// ---- searches by a warp -------------------------------------------------

constexpr int CW_THREADS = 64;
constexpr u32 CW_REACH = 1024;
constexpr u32 CW_HASH = 2 * CW_REACH;
constexpr int CW_HASH_SHIFT = 21;     // 32 - log2(CW_HASH)
constexpr u32 CW_LEVELS = 512;
constexpr u32 CW_EDGES = 16384;       // join words of one search

struct CwSmem {
    u32 hash[CW_HASH];
    u32 queue[CW_REACH];
    unsigned short lcnt[CW_LEVELS];   // targets of level d at [d - 1]
    unsigned short ldeg[CW_LEVELS];   // join words out of level d at [d - 1]
    u32 wbeg[32], wpre[32];           // compacted rows of the group being expanded
};

// The same search by a warp, for the sources eight lanes' slice could not
// hold (src; null: every rank from lo on). A search that outgrows its slice goes to
// `left`.
__global__ void __launch_bounds__(CW_THREADS)
closure_warp_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val, const u64 *__restrict__ src, u64 lo,
                    u64 n_src, int bits, const u64 *__restrict__ inst_lo, u32 n_inst, u32 stride, u32 max_level,
                    unsigned long long *__restrict__ cnt, unsigned long long *__restrict__ deg,
                    SearchOut to, SearchCounters *__restrict__ ctr, u64 *__restrict__ left) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CwSmem &s = reinterpret_cast<CwSmem *>(smem_raw)[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u32 le = lane == 31 ? ~0u : (2u << lane) - 1;
    LevelSums sums;
    sums.init(inst_lo == nullptr, 0);
    u32 top = 0;            // largest level seen
    for (;;) {
        unsigned long long g = 0;
        if (lane == 0) g = atomicAdd(&ctr->fetch, 1ull);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= n_src) break;
        {
            const u64 x = src ? src[g] : lo + g;
            const u32 b0 = __ldg(off + x), d0 = __ldg(off + x + 1) - b0;
            if (d0 == 0) continue;
            // visited set empty
            uint4 *hv = reinterpret_cast<uint4 *>(s.hash);
#pragma unroll
            for (u32 k = 0; k < CW_HASH / 4 / 32; ++k) hv[k * 32 + lane] = make_uint4(EMPTY, EMPTY, EMPTY, EMPTY);
            __syncwarp();
            u32 tail = 0, edges = 0;
            bool over = false;
            auto visit = [&](u32 w, bool have) -> bool {
                const bool fresh = have && set_insert<CW_HASH - 1>(s.hash, w, CW_HASH_SHIFT);
                const u32 fm = __ballot_sync(0xffffffffu, fresh);
                const u32 n = __popc(fm);
                if (tail + n > CW_REACH) {
                    over = true;
                    return false;
                }
                if (fresh) s.queue[tail + __popc(fm & lt)] = w;
                tail += n;
                return true;
            };
            // level 1: x's own edges
            if (walk_rows(s.wbeg, s.wpre, b0, lane == 0 ? d0 : 0u, val, lane, lt, le, CW_REACH, visit) > CW_REACH)
                over = true;
            u32 head = 0, level = 1;
            while (!over) {
                __syncwarp();
                const u32 end = tail;
                u32 ld = 0;
                if (level != max_level) {
                    for (u32 h = head; h < end && !over; h += 32) {
                        u32 b = 0, d = 0;
                        if (h + lane < end) {
                            const u32 y = s.queue[h + lane];
                            b = __ldg(off + y);
                            d = __ldg(off + y + 1) - b;
                        }
                        const u32 t = walk_rows(s.wbeg, s.wpre, b, d, val, lane, lt, le, CW_EDGES - edges, visit);
                        if (t > CW_EDGES - edges) {
                            over = true;
                            break;
                        }
                        edges += t;
                        ld += t;
                    }
                }
                if (over) break;
                if (lane == 0) {
                    s.lcnt[level - 1] = (unsigned short) (end - head);
                    s.ldeg[level - 1] = (unsigned short) ld;
                }
                if (tail == end) break;  // no level after this one
                head = end;
                if (++level > CW_LEVELS) over = true;
            }
            __syncwarp();
            if (over) {
                if (lane == 0) {
                    left[atomicAdd(&ctr->left, 1ull)] = x;
                    to.note(x - lo, 0, 0);
                }
                continue;
            }
            // level sizes
            top = max(top, level);
            sums.add(x, level, s.lcnt, s.ldeg, inst_lo, n_inst, cnt, deg, stride, lane);
            // result words
            unsigned long long p = 0;
            if (lane == 0) p = atomicAdd(&ctr->words, (unsigned long long) tail);
            p = __shfl_sync(0xffffffffu, p, 0);
            if (lane == 0) to.note(x - lo, p, tail);
            if (p + tail <= to.cap)
                for (u32 k = lane; k < tail; k += 32) to.out[p + k] = ((u64) s.queue[k] << bits) | x;
            __syncwarp();
        }
    }
    sums.flush(cnt, deg, stride, lane);
    if (lane == 0 && top) atomicMax(&ctr->levels, (unsigned long long) top);
}

// ---- searches by a CTA --------------------------------------------------

constexpr int CC_THREADS = 256;
constexpr u32 CC_REACH = 4096;
constexpr u32 CC_HASH = 2 * CC_REACH;
constexpr int CC_HASH_SHIFT = 19;  // 32 - log2(CC_HASH)
constexpr u32 CC_EDGES = 1u << 18;
// Once more than half of the sources begun (the first ones aside) were left over, those that follow are
// too, unsearched: the bit rows take them at less than a failed search costs. A prime step
// through the sources makes the first ones a sample of all. Random graph of 20K nodes and 30K
// edges 3.76 -> 2.50 ms, of 24K 3.53 -> 2.75.
constexpr u64 CC_SPREAD = 2654435761ull;  // prime, and far more than the sources that come here
constexpr u64 CC_TRIED = 512;

struct CcSmem {
    u32 hash[CC_HASH];
    u32 queue[CC_REACH];
    u32 wbeg[CC_THREADS / 32][32], wpre[CC_THREADS / 32][32];
    u32 tail, edges;
    u64 x, pos;
};

// The same search by a CTA, for the sources a warp's slice could not hold:
// each level's rows are shared by the CTA's warps, 32 rows at a time. Level
// sizes go to the CTA's slice of `lev` (2 * CL_LEVELS words) until the search has
// finished: in shared memory they would cost a quarter of the resident CTAs.
__global__ void __launch_bounds__(CC_THREADS)
closure_cta_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val, const u64 *__restrict__ src, u64 lo,
                   u64 n_src,
                   u32 reach, int bits, const u64 *__restrict__ inst_lo, u32 n_inst, u32 stride, u32 max_level,
                   unsigned long long *__restrict__ cnt, unsigned long long *__restrict__ deg, u32 *lev,
                   SearchOut to, SearchCounters *__restrict__ ctr, u64 *__restrict__ left) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    u32 *lcnt = lev + (u64) blockIdx.x * 2 * CL_LEVELS, *ldeg = lcnt + CL_LEVELS;
    CcSmem &s = *reinterpret_cast<CcSmem *>(smem_raw);
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 lt = lanemask_lt();
    const u32 le = lane == 31 ? ~0u : (2u << lane) - 1;
    for (;;) {
        if (tid == 0) {
            u64 x = ~0ull;
            for (;;) {
                const u64 i = atomicAdd(&ctr->fetch, 1ull);
                if (i >= n_src) break;
                x = src[i * CC_SPREAD % n_src];
                if (inst_lo || i < CC_TRIED || 2 * *reinterpret_cast<volatile unsigned long long *>(&ctr->left) <= i) break;
                left[atomicAdd(&ctr->left, 1ull)] = x;
                to.note(x - lo, 0, 0);
                x = ~0ull;
            }
            s.x = x;
            s.tail = 0;
            s.edges = 0;
        }
        uint4 *hv = reinterpret_cast<uint4 *>(s.hash);
        for (u32 k = tid; k < CC_HASH / 4; k += CC_THREADS) hv[k] = make_uint4(EMPTY, EMPTY, EMPTY, EMPTY);
        __syncthreads();
        const u64 x = s.x;
        if (x == ~0ull) break;
        auto visit = [&](u32 w, bool have) -> bool {
            // the set holds at most `reach` words and the warps' windows in flight
            if (__any_sync(0xffffffffu, *reinterpret_cast<volatile u32 *>(&s.tail) > reach)) return false;
            const bool fresh = have && set_insert<CC_HASH - 1>(s.hash, w, CC_HASH_SHIFT);
            const u32 fm = __ballot_sync(0xffffffffu, fresh);
            if (fm) {
                u32 at = 0;
                if (lane == 0) at = atomicAdd(&s.tail, (u32) __popc(fm));
                at = __shfl_sync(0xffffffffu, at, 0) + __popc(fm & lt);
                if (fresh && at < CC_REACH) s.queue[at] = w;
            }
            return true;
        };
        // rows of a group of up to 32 nodes; the level's edges are added to s.edges. A group
        // past the limit was not walked at all, so the search must not end here even if
        // nothing else is new: it counts as one that outgrew its reach.
        auto expand = [&](u32 b, u32 d) {
            const u32 t = walk_rows(s.wbeg[warp], s.wpre[warp], b, d, val, lane, lt, le, CC_EDGES, visit);
            if (lane == 0 && t) {
                atomicAdd(&s.edges, min(t, CC_EDGES + 1));
                if (t > CC_EDGES) atomicMax(&s.tail, reach + 1);
            }
        };
        if (warp == 0) {
            const u32 b0 = __ldg(off + x), d0 = __ldg(off + x + 1) - b0;
            if (d0 <= reach) expand(b0, lane == 0 ? d0 : 0u);
            else if (lane == 0) s.tail = reach + 1;
        }
        u32 head = 0, level = 1;
        bool over = false;
        for (;;) {
            __syncthreads();  // the level's targets are queued
            const u32 end = s.tail;
            if (end > reach || s.edges > CC_EDGES) {
                over = true;
                break;
            }
            __syncthreads();  // every thread has read the level's bounds
            if (tid == 0) s.edges = 0;
            __syncthreads();
            if (level != max_level) {
                for (u32 h = head + warp * 32; h < end; h += CC_THREADS) {
                    u32 b = 0, d = 0;
                    if (h + lane < end) {
                        const u32 y = s.queue[h + lane];
                        b = __ldg(off + y);
                        d = __ldg(off + y + 1) - b;
                    }
                    expand(b, d);
                }
            }
            __syncthreads();
            if (tid == 0) {
                lcnt[level - 1] = end - head;
                ldeg[level - 1] = s.edges;
            }
            if (s.tail == end) break;
            head = end;
            if (++level > CL_LEVELS) {
                over = true;
                break;
            }
        }
        __syncthreads();
        if (over) {
            if (tid == 0) {
                left[atomicAdd(&ctr->left, 1ull)] = x;
                to.note(x - lo, 0, 0);
            }
            __syncthreads();
            continue;
        }
        const u32 tail = s.tail;
        const u32 inst = inst_lo ? instance_at(inst_lo, n_inst, x) : 0;
        for (u32 k = tid; k < level; k += CC_THREADS) {
            const u64 at = (u64) inst * stride + 1 + k;
            atomicAdd(cnt + at, (unsigned long long) lcnt[k]);
            if (deg) atomicAdd(deg + at, (unsigned long long) ldeg[k]);
        }
        if (tid == 0) {
            s.pos = atomicAdd(&ctr->words, (unsigned long long) tail);
            to.note(x - lo, s.pos, tail);
            atomicMax(&ctr->levels, (unsigned long long) level);
        }
        __syncthreads();
        const u64 p = s.pos;
        if (p + tail <= to.cap)
            for (u32 k = tid; k < tail; k += CC_THREADS) to.out[p + k] = ((u64) s.queue[k] << bits) | x;
        __syncthreads();  // the queue and x are free
    }
}

// ---- heavy sources: 32 to a word ----------------------------------------

__global__ void add_counts_kernel(u64 *__restrict__ a, const unsigned long long *__restrict__ b, u64 n) {
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x) a[i] += b[i];
}

// Column i = heavy source src[i] (a warp each): its level-0 row is its own bit
// at node src[i]; pads the column ids up to `words` * 32.
__global__ void pull_init_kernel(PullShape sh, PullLevel st, const u64 *__restrict__ src, u64 h,
                                 u32 *__restrict__ cols) {
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    for (u64 i = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32; i < (u64) sh.words * 32; i += warps) {
        if (i >= h) {
            if (lane == 0) cols[i] = EMPTY;
            continue;
        }
        const u64 x = src[i];
        const u32 gr = (u32) (i >> 10) >> sh.shift;
        u32 *row = st.nxt + x * sh.words;
        const u32 w0 = (gr << sh.shift) * 32, w1 = min(sh.words, w0 + (32u << sh.shift));
        for (u32 k = w0 + lane; k < w1; k += 32) row[k] = k == (u32) (i >> 5) ? 1u << (i & 31) : 0u;
        if (lane == 0) {
            cols[i] = (u32) x;
            st.tag_next[x] = make_uint2(1u << gr, 0u);
        }
    }
}

// One level: for every target in the level's list (a warp each), the new bits
// of its row = (OR of its in-neighbours' newest bits) & ~T, K * 512 bytes of the
// row at a time (K by the row's length: the work per in-neighbour that does
// not depend on the row is paid once for all K pieces). Only words that are
// tagged as newest are ever read, so nothing is cleared between levels.
template <int K>
__global__ void __launch_bounds__(PU_THREADS, K >= 3 ? 3 : 4)
closure_pull_kernel(PullShape sh, PullLevel st, const u32 *__restrict__ off, const u32 *__restrict__ roff,
                    const u32 *__restrict__ rval, const u32 *__restrict__ hub_at, u32 *__restrict__ hub_acc,
                    u32 *__restrict__ t) {
    const u64 n_list = st.count[st.level];
    if (n_list == 0) return;  // the fixpoint was reached earlier
    __shared__ unsigned long long part[2][PU_THREADS / 32];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u64 warps = (u64) gridDim.x * (PU_THREADS / 32);
    u64 fresh = 0, dsum = 0;
    for (u64 i = ((u64) blockIdx.x * PU_THREADS + threadIdx.x) / 32; i < n_list; i += warps) {
        const u32 w = st.list[i];
        const u32 m = st.todo[w];
        const u32 b = __ldg(roff + w), n = __ldg(roff + w + 1) - b;
        const bool hub = n > PU_SEG;
        u32 y0 = 0, a0 = 0;
        u32 *hrow = nullptr;
        if (hub) {
            hrow = hub_acc + (u64) hub_at[w] * sh.words + lane * 4;
        } else if (lane < n) {
            y0 = __ldg(rval + b + lane);
            const uint2 tg = st.tag[y0];
            a0 = tg.y == st.level - 1 ? tg.x : 0u;
        }
        u32 news = 0, bits_new = 0;
        const u64 row = (u64) w * sh.words + lane * 4;
        for (u32 base = 0; base < sh.words; base += K * 128) {
            u32 in = 0, need = 0;
            uint4 old[K], acc[K];
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const bool on = base + 128 * k + lane * 4 < sh.words && (m & piece_bit<K>(sh, base, k, lane));
                if (on) in |= 1u << k;
                old[k] = on ? *reinterpret_cast<const uint4 *>(t + row + base + 128 * k)
                            : make_uint4(~0u, ~0u, ~0u, ~0u);
                acc[k] = make_uint4(0, 0, 0, 0);
            }
            if (!__any_sync(0xffffffffu, in != 0)) continue;
            if (hub) {
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if ((in >> k) & 1u) {
                        uint4 *hp = reinterpret_cast<uint4 *>(hrow + base + 128 * k);
                        acc[k] = *hp;
                        *hp = make_uint4(0, 0, 0, 0);
                    }
            } else {
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if ((old[k].x & old[k].y & old[k].z & old[k].w) != ~0u) need |= 1u << k;
                or_neighbours<K>(sh, st.cur, base, y0, a0, need, lane, acc);
            }
            u32 mark = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint4 nw = make_uint4(acc[k].x & ~old[k].x, acc[k].y & ~old[k].y, acc[k].z & ~old[k].z,
                                            acc[k].w & ~old[k].w);
                const bool any = (nw.x | nw.y | nw.z | nw.w) != 0;
                if (any) {
                    *reinterpret_cast<uint4 *>(t + row + base + 128 * k) =
                        make_uint4(old[k].x | nw.x, old[k].y | nw.y, old[k].z | nw.z, old[k].w | nw.w);
                    bits_new += __popc(nw.x) + __popc(nw.y) + __popc(nw.z) + __popc(nw.w);
                }
                const u32 lines = __ballot_sync(0xffffffffu, any);
                const bool line = ((lines >> (lane & 24)) & 0xFFu) != 0;  // this piece's chunk has new bits
                if (line) mark |= piece_bit<K>(sh, base, k, lane);
                if (((in >> k) & 1u) && (line || sh.shift))
                    *reinterpret_cast<uint4 *>(st.nxt + row + base + 128 * k) = nw;
            }
            news |= __reduce_or_sync(0xffffffffu, mark);
        }
        if (lane == 0) {
            st.todo[w] = 0;
            if (news) st.tag_next[w] = make_uint2(news, st.level);
        }
        if (bits_new) {
            fresh += bits_new;
            dsum += (u64) bits_new * (__ldg(off + w + 1) - __ldg(off + w));
        }
    }
    fresh = warp_sum(fresh);
    dsum = warp_sum(dsum);
    if (lane == 0) {
        part[0][warp] = fresh;
        part[1][warp] = dsum;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long v = 0;
        for (int i = 0; i < PU_THREADS / 32; ++i) v += part[threadIdx.x][i];
        if (v) atomicAdd((threadIdx.x == 0 ? st.cnt : st.deg) + st.level, v);
    }
}

// The same level for rows of P = 1 or 2 chunks (up to 2048 heavy sources), by eight lanes for a
// target: a warp's 32 lanes, one target at a time, left most of a short row's idle,
// and the level is a chain of dependent loads. Trees, whose heavy sources are few: 4M nodes,
// three children each, 1.0 -> 0.26 ms a level (the whole run 24.7 -> 13.0, 12.4 on the sorted
// runs); 1M nodes, ten children, 4.2 -> 3.0 (2.5).
template <int P>
__global__ void __launch_bounds__(PU_THREADS, 4)
closure_pull_thin_kernel(PullShape sh, PullLevel st, const u32 *__restrict__ off, const u32 *__restrict__ roff,
                         const u32 *__restrict__ rval, const u32 *__restrict__ hub_at, u32 *__restrict__ hub_acc,
                         u32 *__restrict__ t) {
    const u64 n_list = st.count[st.level];
    if (n_list == 0) return;  // the fixpoint was reached earlier
    __shared__ unsigned long long part[2][PU_THREADS / 32];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l = lane & 7;
    const u64 groups = (u64) gridDim.x * (PU_THREADS / 8);
    u64 fresh = 0, dsum = 0;
    for (u64 i0 = ((u64) blockIdx.x * PU_THREADS + (threadIdx.x & ~31u)) / 8; i0 < n_list; i0 += groups) {
        const u64 i = i0 + (lane >> 3);
        const bool have = i < n_list;
        u32 w = 0, m = 0, b = 0, n = 0;
        if (have) {
            w = st.list[i];
            m = st.todo[w];
            b = __ldg(roff + w);
            n = __ldg(roff + w + 1) - b;
        }
        const u64 row = (u64) w * sh.words + l * 4;
        uint4 old[P], acc[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            acc[p] = old[p] = make_uint4(0, 0, 0, 0);
            if ((m >> p) & 1u) old[p] = *reinterpret_cast<const uint4 *>(t + row + 32 * p);
        }
        if (n > PU_SEG) {
            u32 *hrow = hub_acc + (u64) hub_at[w] * sh.words + l * 4;
#pragma unroll
            for (int p = 0; p < P; ++p)
                if ((m >> p) & 1u) {
                    uint4 *hp = reinterpret_cast<uint4 *>(hrow + 32 * p);
                    acc[p] = *hp;
                    *hp = make_uint4(0, 0, 0, 0);
                }
            n = 0;
        }
        const u32 most = __reduce_max_sync(0xffffffffu, n);
        for (u32 k0 = 0; k0 < most; k0 += 8) {
            u32 y = 0, a = 0;
            if (k0 + l < n) {
                y = __ldg(rval + b + k0 + l);
                const uint2 tg = st.tag[y];
                a = tg.y == st.level - 1 ? tg.x : 0u;
            }
            constexpr u32 FLIGHT = 4 / P;  // in-neighbours whose pieces are in flight
            uint4 v[FLIGHT][P];
#pragma unroll
            for (u32 h = 0; h < 8; h += FLIGHT) {
#pragma unroll
                for (u32 j = 0; j < FLIGHT; ++j) {
                    const u32 yj = __shfl_sync(0xffffffffu, y, h + j, 8), aj = __shfl_sync(0xffffffffu, a, h + j, 8);
                    const uint4 *src = reinterpret_cast<const uint4 *>(st.cur + (u64) yj * sh.words + l * 4);
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        v[j][p] = make_uint4(0, 0, 0, 0);
                        if ((aj >> p) & 1u) v[j][p] = __ldg(src + 8 * p);
                    }
                }
#pragma unroll
                for (u32 j = 0; j < FLIGHT; ++j)
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        acc[p].x |= v[j][p].x;
                        acc[p].y |= v[j][p].y;
                        acc[p].z |= v[j][p].z;
                        acc[p].w |= v[j][p].w;
                    }
            }
        }
        u32 mark = 0, bits_new = 0;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const uint4 nw = make_uint4(acc[p].x & ~old[p].x, acc[p].y & ~old[p].y, acc[p].z & ~old[p].z,
                                        acc[p].w & ~old[p].w);
            const bool any = (nw.x | nw.y | nw.z | nw.w) != 0;
            if (any) {
                *reinterpret_cast<uint4 *>(t + row + 32 * p) =
                    make_uint4(old[p].x | nw.x, old[p].y | nw.y, old[p].z | nw.z, old[p].w | nw.w);
                bits_new += __popc(nw.x) + __popc(nw.y) + __popc(nw.z) + __popc(nw.w);
            }
            const u32 lines = __ballot_sync(0xffffffffu, any);
            if ((lines >> (lane & 24)) & 0xFFu) {  // this chunk has new bits: the whole line is written
                mark |= 1u << p;
                *reinterpret_cast<uint4 *>(st.nxt + row + 32 * p) = nw;
            }
        }
        if (have && l == 0) {
            st.todo[w] = 0;
            if (mark) st.tag_next[w] = make_uint2(mark, st.level);
        }
        if (bits_new) {
            fresh += bits_new;
            dsum += (u64) bits_new * (__ldg(off + w + 1) - __ldg(off + w));
        }
    }
    fresh = warp_sum(fresh);
    dsum = warp_sum(dsum);
    if (lane == 0) {
        part[0][warp] = fresh;
        part[1][warp] = dsum;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long v = 0;
        for (int i = 0; i < PU_THREADS / 32; ++i) v += part[threadIdx.x][i];
        if (v) atomicAdd((threadIdx.x == 0 ? st.cnt : st.deg) + st.level, v);
    }
}

// ---- results ------------------------------------------------------------

// Row z's result rows by chunk: start[z * chunks + c] = (rows of z before
// chunk c, light pairs of z before it), a light pair belonging to the chunk of
// the column it comes before (the last chunk when there is none). counts[z] =
// rows of z. A warp per target.
__global__ void closure_counts_kernel(const u32 *__restrict__ t, u64 n, u32 words, const u64 *__restrict__ light,
                                      const u64 *__restrict__ loff, u64 mask, const u32 *__restrict__ place,
                                      uint2 *__restrict__ start, u64 *__restrict__ counts) {
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    const u32 chunks = words / 32;
    for (u64 z = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32; z < n; z += warps) {
        const u32 *row = t + z * words;
        const u64 *lz = light + loff[z];
        const u32 nl = (u32) (loff[z + 1] - loff[z]);
        u32 rows = 0, li = 0, wb = 0;
        u32 lc = lane < nl ? __ldg(place + (__ldg(lz + lane) & mask)) : EMPTY;
        u32 v = row[lane];
        for (u32 c = 0; c < chunks; ++c) {
            const u32 vn = c + 1 < chunks ? row[(c + 1) * 32 + lane] : 0u;
            if (lane == 0) start[z * chunks + c] = make_uint2(rows + li, li);
            rows += __reduce_add_sync(0xffffffffu, __popc(v));
            for (;;) {  // light pairs before columns of this chunk
                const u32 m = __ballot_sync(0xffffffffu, lc < (c + 1) * 1024);
                li += __popc(m);
                if (lc < (c + 1) * 1024) lc = EMPTY;
                if (li < wb + 32 || li >= nl) break;
                wb += 32;
                lc = wb + lane < nl ? __ldg(place + (__ldg(lz + wb + lane) & mask)) : EMPTY;
            }
            v = vn;
        }
        if (lane == 0) counts[z] = (u64) rows + nl;
    }
}

struct SumValue {
    const u64 *v;
    __device__ __forceinline__ u64 operator()(u64 i) const { return v[i]; }
};

// Edges of ranks [lo, hi) as words over ranks from lo.
__global__ void local_edges_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val, u64 lo, u64 hi, int bits,
                                   u64 *__restrict__ out) {
    const u32 b = off[lo];
    for (u64 r = lo + (u64) blockIdx.x * blockDim.x + threadIdx.x; r < hi; r += (u64) gridDim.x * blockDim.x)
        for (u32 k = off[r]; k < off[r + 1]; ++k) out[k - b] = ((r - lo) << bits) | (val[k] - lo);
}

// The set bits of T as words (z << bits) | x over ranks from lo, unordered.
__global__ void heavy_words_kernel(const u32 *__restrict__ t, u64 n, u32 words, const u32 *__restrict__ cols, u64 lo,
                                   int bits, u64 *__restrict__ out, u64 cap, unsigned long long *__restrict__ count) {
    const u32 lane = threadIdx.x & 31;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    for (u64 z = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32; z < n; z += warps) {
        for (u32 k0 = 0; k0 < words; k0 += 32) {
            u32 v = t[z * words + k0 + lane];
            const u32 incl = warp_inclusive_sum((u32) __popc(v));
            const u32 total = __shfl_sync(0xffffffffu, incl, 31);
            if (!total) continue;
            unsigned long long p = 0;
            if (lane == 0) p = atomicAdd(count, (unsigned long long) total);
            p = __shfl_sync(0xffffffffu, p, 0);
            if (p + total > cap) continue;
            p += incl - __popc(v);
            for (; v; v &= v - 1)
                out[p++] = ((z + lo) << bits) | (cols[(k0 + lane) * 32 + __ffs(v) - 1] + lo);
        }
    }
}

// place[r] = heavy sources below rank r.
__global__ void heavy_below_kernel(const u32 *__restrict__ cols, u64 h, u64 n, u32 *__restrict__ place) {
    for (u64 r = (u64) blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (u64) gridDim.x * blockDim.x) {
        u64 a = 0, b = h;
        while (a < b) {
            const u64 m = (a + b) >> 1;
            if (cols[m] < r) a = m + 1;
            else b = m;
        }
        place[r] = (u32) a;
    }
}

// Result rows (x, z) of targets [z0, z1), by (z, x): the set bits of row z of
// T (ascending columns = ascending sources) merged with z's light pairs
// (ascending sources; one comes before the heavy sources at columns
// place[source] and up). A warp walks the targets of one chunk of 1024 columns;
// where a target's rows of that chunk go is known from the counts, so chunks and
// targets are independent. In a chunk, a word's first position comes from a
// prefix sum over the words plus the light pairs before it. Then
//  * DENSE (a third of the bits set or more): a lane per bit of a word, whose rows
//    leave as consecutive 8-byte stores, the columns' node ids in 32 registers
//    (ten instructions a word: with the ids loaded per word it was bound by
//    issue, 40 a word);
//  * else a lane per word walks its bits' positions into shared memory, and the
//    chunk's rows leave with consecutive stores; their columns are looked up there
//    (not at the walk, which takes as many turns as its fullest word has bits),
//    or, where the chunk's columns are consecutive ranks, added up.
// Light pairs are placed lane-parallel; a word that one falls inside is done
// last, its lanes shifted by the light pairs below them.

constexpr u32 MERGE_PAIRS = 32;  // light pairs of a chunk that closure_rows_kernel takes: a window

template <bool DENSE, bool ROW_FIRST>
__global__ void __launch_bounds__(256)
closure_rows_kernel(const u32 *__restrict__ t, u32 words, const u32 *__restrict__ cols,
                    const u32 *__restrict__ place, const uint2 *__restrict__ start, u64 z0, u64 z1,
                    const u64 *__restrict__ first, const u64 *__restrict__ light, const u64 *__restrict__ loff,
                    u64 mask, const int32_t *__restrict__ ids, bool affine, int32_t base, u64 *__restrict__ out) {
    __shared__ unsigned short staged[DENSE ? 1 : 8][DENSE ? 1 : 1024];
    unsigned short *stage = staged[DENSE ? 0 : threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u32 chunks = words / 32;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    const u64 me = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32;
    auto node = [&](u32 r) -> u32 { return (u32) (affine ? (int32_t) (base + (int64_t) r) : __ldg(ids + r)); };
    // chunk me % chunks for the targets me / chunks, + warps / chunks, ... (more
    // chunks than warps: the same warp takes further chunks)
    const u64 step = max(warps / chunks, (u64) 1);
    for (u64 c0 = me % min((u64) chunks, warps); c0 < chunks; c0 += warps) {
        if (me / chunks >= step) break;  // warps beyond a whole number of rounds
        const u32 k0 = (u32) c0 * 32;
        const u32 *cc = cols + c0 * 1024;
        u32 id[DENSE ? 32 : 1];
        if constexpr (DENSE) {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const u32 x = __ldg(cc + j * 32 + lane);
                id[j] = x == EMPTY ? 0u : node(x);
            }
        }
        const u32 c_first = __ldg(cc);
        const bool consecutive = __ldg(cc + 1023) - c_first == 1023;  // columns ascend (EMPTY past the last)
        u64 z = z0 + me / chunks;
        u32 v_next = 0;
        uint2 st_next = make_uint2(0, 0);
        u64 first_next = 0;
        auto fetch = [&](u64 y) {  // one target ahead
            if (y >= z1) return;
            v_next = t[y * words + k0 + lane];
            st_next = start[y * chunks + c0];
            first_next = first[y];
        };
        fetch(z);
        for (; z < z1; z += step) {
            u32 v = v_next;
            const uint2 st = st_next;
            u64 *dst = out + first_next + st.x;
            fetch(z + step);
            const u32 lend = c0 + 1 < chunks ? start[z * chunks + c0 + 1].y : (u32) (loff[z + 1] - loff[z]);
            const u32 any = __ballot_sync(0xffffffffu, v != 0);
            if ((!any && st.y == lend) || lend - st.y > MERGE_PAIRS) continue;  // (closure_merge_kernel's)
            const u32 zid = node((u32) z);
            // a row (x, z), or (z, x) when the targets come first, as one little-endian word
            auto pack = [&](u32 x) -> u64 { return ROW_FIRST ? ((u64) x << 32) | zid : ((u64) zid << 32) | x; };
            const u32 n = __popc(v);
            const u32 incl = warp_inclusive_sum(n);
            u32 at = incl - n;
            if constexpr (!DENSE) {
                const u32 total = __shfl_sync(0xffffffffu, incl, 31);
                if (st.y == lend) {
                    for (; v; v &= v - 1) stage[at++] = (unsigned short) (lane * 32 + __ffs(v) - 1);
                    __syncwarp();
                    if (consecutive) {
                        for (u32 i = lane; i < total; i += 32) dst[i] = pack(node(c_first + stage[i]));
                    } else {
                        for (u32 i = lane; i < total; i += 32) dst[i] = pack(node(__ldg(cc + stage[i])));
                    }
                    __syncwarp();
                    continue;
                }
            }
            u32 inside = 0;
            const u64 *lz = light + loff[z];
            // light pairs st.y .. lend - 1: one in word j before bit b
            auto pair = [&](u32 l, u32 &x, u32 &rel) {
                x = 0;
                rel = EMPTY;
                if (l < lend) {
                    x = (u32) (__ldg(lz + l) & mask);
                    rel = min(__ldg(place + x) - k0 * 32, 1024u);
                }
            };
            u32 rel = EMPTY;
            if (st.y < lend) {
                u32 x;
                pair(st.y + lane, x, rel);
                const bool in = st.y + lane < lend;
                const u32 j = rel >> 5, b = rel & 31;
                // (rel 1024: after every column)
                const u32 wj = __shfl_sync(0xffffffffu, v, j & 31), pj = __shfl_sync(0xffffffffu, incl - n, j & 31);
                const u32 total = __shfl_sync(0xffffffffu, incl, 31);
                if (in) dst[(j < 32 ? pj + __popc(wj & ((1u << b) - 1)) : total) + lane] = pack(node(x));
                const u32 key = in ? (b ? j : j - 1) : EMPTY - 1;  // words above `key` are shifted whole
                for (u32 k = 0; k < lend - st.y; ++k) at += (int) lane > (int) __shfl_sync(0xffffffffu, key, k);
                inside = __reduce_or_sync(0xffffffffu, in && b && j < 32 ? 1u << j : 0u);
            }
            u32 slow = any & inside;
            const u32 v0 = v;
            if ((inside >> lane) & 1u) v = 0;
            if constexpr (DENSE) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const u32 word = __shfl_sync(0xffffffffu, v, j);
                    const u32 p = __shfl_sync(0xffffffffu, at, j) + __popc(word & lt);
                    if ((word >> lane) & 1u) dst[p] = pack(id[j]);
                }
            } else {
                // (of a tree's 32 words three hold bits: 1M targets 0.78 -> 0.48 ms)
                for (u32 nz = any & ~inside; nz; nz &= nz - 1) {
                    const u32 j = __ffs(nz) - 1;
                    const u32 word = __shfl_sync(0xffffffffu, v, j);
                    const u32 p = __shfl_sync(0xffffffffu, at, j) + __popc(word & lt);
                    if ((word >> lane) & 1u) dst[p] = pack(node(__ldg(cc + j * 32 + lane)));
                }
            }
            while (slow) {
                const u32 j = __ffs(slow) - 1;
                slow &= slow - 1;
                const u32 word = __shfl_sync(0xffffffffu, v0, j);
                u32 p = __shfl_sync(0xffffffffu, at, j) + __popc(word & lt);
                for (u32 mm = __ballot_sync(0xffffffffu, (rel >> 5) == j && (rel & 31)); mm; mm &= mm - 1)
                    p += (__shfl_sync(0xffffffffu, rel, __ffs(mm) - 1) & 31) <= lane;
                if ((word >> lane) & 1u) dst[p] = pack(node(__ldg(cc + j * 32 + lane)));
            }
        }
    }
}

// The rows of (target, chunk)s with more light pairs than a window. Their places in the
// chunk ascend, so a window of 32 pairs shifts the words by the number of its pairs below each
// (six shuffles); the last pair of every place leaves its number there, and a
// column's shift is the largest number up to it. (Going through all of a chunk's pairs again
// for each of its words was quadratic: 21K nodes in 20 layers, 44M pairs, half of them
// light, 4.8 ms of 7.2; 3.0 for the whole run here. Within the kernel above it cost every run a
// third of its resident warps in registers.) A warp looks at `take`
// (target, chunk)s at a time, up to 32, so that all warps have some.
__global__ void __launch_bounds__(256)
closure_merge_kernel(const u32 *__restrict__ t, u32 words, const u32 *__restrict__ cols, const u32 *__restrict__ place,
                     const uint2 *__restrict__ start, u64 z0, u64 z1, const u64 *__restrict__ first,
                     const u64 *__restrict__ light, const u64 *__restrict__ loff, u64 mask,
                     const int32_t *__restrict__ ids, bool affine, int32_t base, u32 take, u64 *__restrict__ out) {
    __shared__ __align__(4) unsigned short staged[8][1024];
    unsigned short *stage = staged[threadIdx.x >> 5];
    const u32 lane = threadIdx.x & 31;
    const u32 lt = lanemask_lt();
    const u32 chunks = words / 32;
    const u64 warps = (u64) gridDim.x * (blockDim.x / 32);
    auto node = [&](u32 r) -> u32 { return (u32) (affine ? (int32_t) (base + (int64_t) r) : __ldg(ids + r)); };
    for (u64 i0 = z0 * chunks + ((u64) blockIdx.x * blockDim.x + threadIdx.x) / 32 * take; i0 < z1 * chunks;
         i0 += warps * take) {
        u64 zl = 0;
        u32 from = 0, to = 0, rows = 0;
        if (lane < take && i0 + lane < z1 * chunks) {
            zl = (i0 + lane) / chunks;
            const uint2 st = start[i0 + lane];
            rows = st.x;
            from = st.y;
            to = (i0 + lane + 1) % chunks ? start[i0 + lane + 1].y : (u32) (loff[zl + 1] - loff[zl]);
        }
        for (u32 todo = __ballot_sync(0xffffffffu, to - from > MERGE_PAIRS); todo; todo &= todo - 1) {
            const u32 q = __ffs(todo) - 1;
            const u64 z = __shfl_sync(0xffffffffu, zl, q);
            const u32 k0 = (u32) ((i0 + q) % chunks) * 32;
            const u32 lbeg = __shfl_sync(0xffffffffu, from, q), lend = __shfl_sync(0xffffffffu, to, q);
            u64 *dst = out + first[z] + __shfl_sync(0xffffffffu, rows, q);
            const u64 *lz = light + loff[z];
            const u64 zid = (u64) node((u32) z) << 32;
            const u32 v = t[z * words + k0 + lane];
            const u32 incl = warp_inclusive_sum((u32) __popc(v));
            const u32 before = incl - __popc(v), total = __shfl_sync(0xffffffffu, incl, 31);
            auto place_of = [&](u32 x) { return min(__ldg(place + x) - k0 * 32, 1024u); };  // 1024: after every column
            const bool counted = lend - lbeg <= 0xFFFFu;  // else a column's shift is searched for
            if (counted)
                for (u32 k = lane; k < 512; k += 32) reinterpret_cast<u32 *>(stage)[k] = 0;
            __syncwarp();
            u32 shift = 0;  // pairs at or before the first column of this lane's word
            for (u32 l0 = lbeg; l0 < lend; l0 += 32) {
                const u32 i = l0 + lane - lbeg;
                const bool in = l0 + lane < lend;
                u32 x = 0, rel = EMPTY;
                if (in) {
                    x = (u32) (__ldg(lz + l0 + lane) & mask);
                    rel = place_of(x);
                }
                const u32 j = rel >> 5, b = rel & 31;
                const u32 wj = __shfl_sync(0xffffffffu, v, j & 31), pj = __shfl_sync(0xffffffffu, before, j & 31);
                if (in) dst[(j < 32 ? pj + __popc(wj & ((1u << b) - 1)) : total) + i] = zid | node(x);
                u32 c = 0;
#pragma unroll
                for (u32 step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(0xffffffffu, rel, c + step - 1) <= 32 * lane) c += step;
                if (__shfl_sync(0xffffffffu, rel, c) <= 32 * lane) ++c;
                shift += c;
                const u32 next = __shfl_down_sync(0xffffffffu, rel, 1);
                if (counted && in && rel < 1024 && (lane == 31 || next != rel)) stage[rel] = (unsigned short) (i + 1);
                __syncwarp();
            }
            for (u32 j = 0; j < 32; ++j) {
                const u32 word = __shfl_sync(0xffffffffu, v, j);
                if (!word) continue;
                const u32 p = __shfl_sync(0xffffffffu, before, j) + __popc(word & lt);
                u32 s = __shfl_sync(0xffffffffu, shift, j);
                if (counted) {
                    u32 m = stage[j * 32 + lane];
                    if (__any_sync(0xffffffffu, m != 0)) {
#pragma unroll
                        for (u32 o = 1; o < 32; o <<= 1) {
                            const u32 y = __shfl_up_sync(0xffffffffu, m, o);
                            if (lane >= o) m = max(m, y);
                        }
                        s = max(s, m);
                    }
                } else {
                    u32 a = lbeg, e = lend;
                    while (a < e) {
                        const u32 mid = (a + e) >> 1;
                        if (place_of((u32) (__ldg(lz + mid) & mask)) <= j * 32 + lane) a = mid + 1;
                        else e = mid;
                    }
                    s = a - lbeg;
                }
                if ((word >> lane) & 1u) dst[p + s] = zid | node(__ldg(cols + k0 * 32 + j * 32 + lane));
            }
            __syncwarp();  // the stage is free
        }
    }
}

// The finished sources' words in source order: L lanes copy a source's (16, or 2
// where a source has fewer than four on average: 8M words of 16M sources 0.64 -> 0.10 ms).
struct SegmentWords {
    const u64 *seg;
    __device__ __forceinline__ u64 operator()(u64 i) const { return seg[i] & 0xFFFFu; }
};
template <u32 L>
__global__ void segments_kernel(const u64 *__restrict__ in, const u64 *__restrict__ seg, const u64 *__restrict__ at,
                                u64 n, u64 *__restrict__ out) {
    const u32 l = threadIdx.x % L;
    const u64 step = (u64) gridDim.x * blockDim.x / L;
    for (u64 i = ((u64) blockIdx.x * blockDim.x + threadIdx.x) / L; i < n; i += step) {
        const u64 sg = seg[i];
        const u32 c = (u32) sg & 0xFFFFu;
        const u64 *src = in + (sg >> 16);
        u64 *dst = out + at[i];
#pragma unroll 4
        for (u32 k = l; k < c; k += L) dst[k] = __ldcs(src + k);
    }
}

template <class K>
u64 resident_blocks(Context &ctx, K kern, int threads, size_t smem) {
    if (smem > 48 * 1024)
        DL_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int per_sm = 0;
    DL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    return (u64) ctx.sm_count * std::max(per_sm, 1);
}

// Keeps the first `keep` bytes of buf while it grows to `bytes`.
void grow_keeping(Context &ctx, DevBuf &buf, u64 bytes, u64 keep) {
    if (buf.p && buf.cap >= bytes) return;
    DevBuf nb;
    ctx.reserve(nb, bytes);
    if (keep) DL_CUDA(cudaMemcpyAsync(nb.p, buf.p, keep, cudaMemcpyDeviceToDevice, ctx.stream));
    ctx.give_back(buf);
    buf = nb;
}

}  // namespace

ClosureLight closure_search(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const u64 *inst_lo, u64 n_inst,
                            u64 k0, u64 k1, u64 stride, u64 max_level, u64 *cnt, u64 *deg) {
    Workspace &ws = ctx.ws;
    ClosureLight res;
    const u64 ns = hi - lo;
    if (ns == 0) return res;
    const u64 table = n_inst * stride * 8;
    const u32 ml = (u32) std::min<u64>(max_level, 0xFFFFFFFFull);
    DL_CUDA(cudaMemsetAsync(cnt, 0, table, ctx.stream));
    if (deg) DL_CUDA(cudaMemsetAsync(deg, 0, table, ctx.stream));
    ctx.reserve(ws.cl_levels, 2 * table);
    auto *c2 = ws.cl_levels.as<unsigned long long>();
    auto *d2 = c2 + table / 8;
    SearchCounters *ctr = reinterpret_cast<SearchCounters *>(&ctx.ctrl->scalar[40]);
    ctx.reserve(ws.cl_left, ns * 8);
    ctx.reserve(ws.cl_seg, ns * 8);
    DL_CUDA(cudaMemsetAsync(ws.cl_seg.p, 0, ns * 8, ctx.stream));
    DevBuf &out = ws.jbuf[0];
    // room for 96 targets a source at first, up to a GiB (nothing is known of the result
    // yet); eight-lane searches go on with more where it was full, the others are repeated
    ctx.reserve(out, std::min<u64>(std::max<u64>(96 * ns, 1 << 16), 1ull << 27) * 8);
    SearchCounters got{};
    // What a launch found: its words are kept, its level counts are added to cnt / deg.
    auto account = [&] {
        ctx.prof_add_bytes(K_BITMAP_EXPAND, 8.0 * got.words);
        res.n_words += got.words;
        res.levels = (u32) std::max<u64>(res.levels, got.levels);
        if (!got.words) return;
        const unsigned ag = grid_for(table / 8, T256, ctx);
        DL_LAUNCH(ctx, K_PREP, 0, add_counts_kernel<<<ag, T256, 0, ctx.stream>>>(cnt, c2, table / 8));
        if (deg) DL_LAUNCH(ctx, K_PREP, 0, add_counts_kernel<<<ag, T256, 0, ctx.stream>>>(deg, d2, table / 8));
    };
    // One stage of warp or CTA searches: `launch(where to)` with zeroed counters; repeated when
    // its words outgrow the room.
    auto stage = [&](auto launch) {
        for (;;) {
            DL_CUDA(cudaMemsetAsync(ctr, 0, sizeof(got), ctx.stream));
            DL_CUDA(cudaMemsetAsync(c2, 0, 2 * table, ctx.stream));
            const u64 room = out.cap / 8 - res.n_words;
            launch(SearchOut{out.as<u64>() + res.n_words, room, res.n_words, ws.cl_seg.as<u64>()});
            DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, ctr, sizeof(got), cudaMemcpyDeviceToHost, ctx.stream));
            ctx.sync();
            std::memcpy(&got, ctx.host_scalars, sizeof(got));
            if (got.words <= room) break;
            grow_keeping(ctx, out, (res.n_words + got.words) * 8, res.n_words * 8);
        }
        account();
    };
    // Few sources go to the warps at once: one launch and one wait instead of two
    // (3.6K sources of a 5.5K-edge DAG: 0.78 -> 0.67 ms for the whole run; the line above it, at
    // CL_FEW, was not timed on both sides).
    const bool groups = ns > CL_FEW && k1 - k0 < CG_MAX_EDGES;
    u64 nl = ns;
    if (groups) {
        const u64 m = k1 - k0;
        ctx.reserve(ws.cl_rec, std::max<u64>(m, 1) * 8);
        ctx.reserve(ws.cl_act, ns * 4);
        DL_CUDA(cudaMemsetAsync(ws.cl_act.p, 0, ns * 4, ctx.stream));
        DL_LAUNCH(ctx, K_PREP, 8.0 * m,
                  in_edges_kernel<<<grid_for(m, T256, ctx), T256, 0, ctx.stream>>>(csr.val, k0, k1, lo,
                                                                                  ws.cl_act.as<u32>()));
        DL_LAUNCH(ctx, K_PREP, 24.0 * m,
                  edge_records_kernel<<<grid_for(m, T256, ctx), T256, 0, ctx.stream>>>(
                      csr.off, csr.val, k0, k1, lo, ws.cl_act.as<u32>(), ws.cl_rec.as<uint2>()));
        const size_t smem_g = sizeof(CgSmem) * (CG_THREADS / 8);
        const u64 wave_g = resident_blocks(ctx, closure_group_kernel, CG_THREADS, smem_g);
        const u64 warps_g = wave_g * (CG_THREADS / 32);
        const u32 batch = (u32) std::max<u64>(4, std::min<u64>(32, ns / (warps_g * 4)));
        const unsigned grid_g = (unsigned) std::max<u64>(
            1, std::min<u64>(wave_g, (ns + batch * (CG_THREADS / 32) - 1) / (batch * (CG_THREADS / 32))));
        // A launch whose room is full takes no further sources; the next one goes on from there.
        // The searches under way then (a few ten thousand) are left over, as those that
        // outgrew their slice.
        for (u64 begun = 0;;) {
            SearchCounters *at = reinterpret_cast<SearchCounters *>(ctx.host_scalars + 8);
            *at = SearchCounters{begun, 0, got.left, 0, ~0ull};
            DL_CUDA(cudaMemcpyAsync(ctr, at, sizeof(got), cudaMemcpyHostToDevice, ctx.stream));
            DL_CUDA(cudaMemsetAsync(c2, 0, 2 * table, ctx.stream));
            const SearchOut to{out.as<u64>() + res.n_words, out.cap / 8 - res.n_words, res.n_words, ws.cl_seg.as<u64>()};
            DL_LAUNCH(ctx, K_BITMAP_EXPAND, 8.0 * (ns - begun),
                      closure_group_kernel<<<grid_g, CG_THREADS, smem_g, ctx.stream>>>(
                          csr.off, ws.cl_rec.as<uint2>(), (u32) k0, lo, hi, batch, bits, inst_lo, (u32) n_inst,
                          (u32) stride, ml, c2, deg ? d2 : nullptr, to, ctr, ws.cl_left.as<u64>()));
            DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, ctr, sizeof(got), cudaMemcpyDeviceToHost, ctx.stream));
            ctx.sync();
            std::memcpy(&got, ctx.host_scalars, sizeof(got));
            got.words = std::min(got.words, got.kept);
            account();
            if (got.fetch >= ns) break;
            begun = got.fetch;
            // the others find as much, or the 96 targets a source that the first room was short of
            const u64 rest = ns - begun;
            const u64 more = (u64) (1.25 * (double) res.n_words / (double) begun * (double) rest);
            grow_keeping(ctx, out, (res.n_words + std::max(more, 96 * rest)) * 8, res.n_words * 8);
        }
        nl = got.left;
        if (nl == 0) return res;
    }
    ctx.reserve(ws.cl_heavy, nl * 8);
    grow_keeping(ctx, out, (res.n_words + std::min<u64>(nl * 512, 1ull << 27)) * 8, res.n_words * 8);
    const size_t smem_w = sizeof(CwSmem) * (CW_THREADS / 32);
    const u64 wave_w = resident_blocks(ctx, closure_warp_kernel, CW_THREADS, smem_w);
    const unsigned grid_w = (unsigned) std::min<u64>(wave_w, (nl + CW_THREADS / 32 - 1) / (CW_THREADS / 32));
    stage([&](SearchOut to) {
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 8.0 * nl,
                  closure_warp_kernel<<<grid_w, CW_THREADS, smem_w, ctx.stream>>>(
                      csr.off, csr.val, groups ? ws.cl_left.as<u64>() : nullptr, lo, nl, bits, inst_lo, (u32) n_inst,
                      (u32) stride, ml, c2, deg ? d2 : nullptr, to, ctr, ws.cl_heavy.as<u64>()));
    });
    if (got.left == 0) return res;
    // What the warps left over: CTA searches, unless there are so many that
    // bit rows are the cheaper form. A CTA search that fails has cost up to
    // `reach` targets' edges, and one that finds thousands of targets more than its column. Measured
    // with 10^8 of them / 4 * 10^7 (on the matrix): five layers of 5,000 nodes and 6 edges a node
    // 0.98 / 1.42 (1.06) ms, 7 and 8 edges 1.72 / 1.18 (1.13) and 1.89 / 1.23 (1.17); 20 layers of 1,000
    // 2.60 / 1.95 (5.02); citations, 30K nodes and 90K edges, 5.24 / 4.17 (25.3); the Chung-Lu
    // graph of 317K nodes 11.9 / 11.5 (45.2).
    nl = got.left;
    const double mean_deg = std::max(1.0, (double) csr.n_vals / std::max<u64>(csr.n_keys, 1));
    u32 reach = CC_REACH;
    if (!inst_lo) {
        const double fit = 4e7 / (mean_deg * (double) nl);
        if (fit < CC_REACH) reach = (u32) fit;
        if (reach < CW_REACH + CW_REACH / 2) reach = 0;
    }
    if (reach == 0) {
        res.n_heavy = nl;
        return res;
    }
    std::swap(ws.cl_left, ws.cl_heavy);  // the sources to search are now in cl_left
    const u64 wave_c = resident_blocks(ctx, closure_cta_kernel, CC_THREADS, sizeof(CcSmem));
    const unsigned grid_c = (unsigned) std::min<u64>(wave_c, nl);
    ctx.reserve(ws.cl_heavy, nl * 8);
    ctx.reserve(ws.cl_act, (u64) grid_c * 2 * CL_LEVELS * 4);
    grow_keeping(ctx, out, (res.n_words + std::min<u64>(nl * 2048, 1ull << 27)) * 8, res.n_words * 8);
    stage([&](SearchOut to) {
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 8.0 * nl,
                  closure_cta_kernel<<<grid_c, CC_THREADS, sizeof(CcSmem), ctx.stream>>>(
                      csr.off, csr.val, ws.cl_left.as<u64>(), lo, nl, reach, bits, inst_lo, (u32) n_inst, (u32) stride, ml,
                      c2, deg ? d2 : nullptr, ws.cl_act.as<u32>(), to, ctr, ws.cl_heavy.as<u64>()));
    });
    res.n_heavy = got.left;
    return res;
}

// Measured on B200, 12.8M words of 100K sources: the passes over the source field
// (two of five) 235 us, lining up 115 us; in a batch's union, whose rank fields are
// wider, three of six passes go: 4.3 -> 2.4 ms for 45M words, 13.7 -> 11.5 ms for the
// whole batch.
u64 *closure_order(Context &ctx, u64 n_sources, u64 n_words, int bits, int used_bits) {
    Workspace &ws = ctx.ws;
    ctx.reserve(ws.jbuf[1], n_words * 8);
    ctx.reserve(ws.cl_seg_at, n_sources * 8);
    u64 *at = ws.cl_seg_at.as<u64>();
    const u64 tiles = (n_sources + SCAN_TILE - 1) / SCAN_TILE;
    u64 *lb = ctx.lookback_words(tiles);
    u32 *ctr = ctx.tile_counter(48);
    DL_CUDA(cudaMemsetAsync(ctr, 0, sizeof(u32), ctx.stream));
    DL_LAUNCH(ctx, K_JOIN_COUNT, 16.0 * n_sources,
              scan_kernel<SegmentWords><<<(unsigned) tiles, SCAN_THREADS, 0, ctx.stream>>>(
                  SegmentWords{ws.cl_seg.as<u64>()}, n_sources, at, lb, ctr, ctx.next_epoch(), &ctx.ctrl->err,
                  &ctx.ctrl->scalar[2]));
    const bool thin = n_words < 4 * n_sources;
    auto copy = thin ? segments_kernel<2> : segments_kernel<16>;
    DL_LAUNCH(ctx, K_SELECT, 16.0 * n_words,
              copy<<<grid_for(n_sources * (thin ? 2 : 16), T256, ctx, 8), T256, 0, ctx.stream>>>(
                  ws.jbuf[0].as<u64>(), ws.cl_seg.as<u64>(), at, n_sources, ws.jbuf[1].as<u64>()));
    int w[8], nw = 0;
    for (int b = 0; b < std::min(used_bits, bits); b += 8) w[nw++] = bits + b;
    return radix_sort_windows(ctx, ws.jbuf[1].as<u64>(), ws.jbuf[0].as<u64>(), n_words, w, nw);
}

static u64 pull_words(u64 h) { return (h + 1023) / 1024 * 32; }

u64 closure_pull_bytes(u64 n, u64 h) { return n * (3 * pull_words(h) * 4 + pull_words(h) / 4); }

ClosureHeavy closure_pull(Context &ctx, const Csr &csr, const u64 *edges, u64 ne, int bits, u64 n, const u64 *src,
                          u64 h, u64 max_level, DevBuf &t, DevBuf &cols) {
    Workspace &ws = ctx.ws;
    ClosureHeavy res;
    res.h = h;
    res.words = pull_words(h);
    PullShape sh{n, (u32) res.words, 0};
    while ((32u << sh.shift) < res.words / 32) ++sh.shift;
    const u64 *rev = edges_by_other(ctx, edges, ne, bits, ws.full[0], ws.full[1]);  // in-neighbours
    ctx.reserve(ws.cl_roff, (n + 1) * 4);
    ctx.reserve(ws.cl_rval, ne * 4);
    u32 *roff = ws.cl_roff.as<u32>(), *rval = ws.cl_rval.as<u32>();
    DL_LAUNCH(ctx, K_PREP, 0,
              key_offsets_kernel<u32><<<grid_for(n + 1, T256, ctx), T256, 0, ctx.stream>>>(rev, ne, bits, n, roff));
    DL_LAUNCH(ctx, K_PREP, 12.0 * ne,
              low_field_kernel<<<grid_for(ne, T256, ctx), T256, 0, ctx.stream>>>(rev, ne, (1ull << bits) - 1, rval));
    // targets with many in-edges
    auto *found = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[44]);
    ctx.reserve(ws.cl_segs, (ne / PU_SEG * 2 + 1) * 8);  // a hub's segments are at most twice its in-edges / 32
    ctx.reserve(ws.cl_hub_at, n * 4);
    DL_CUDA(cudaMemsetAsync(found, 0, 16, ctx.stream));
    DL_LAUNCH(ctx, K_PREP, 4.0 * n,
              pull_hubs_kernel<<<grid_for(n, T256, ctx), T256, 0, ctx.stream>>>(roff, n, ws.cl_hub_at.as<u32>(),
                                                                               ws.cl_segs.as<uint2>(), found));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, found, 16, cudaMemcpyDeviceToHost, ctx.stream));
    // rows: T starts empty; a row of newest bits is read only when its tag says so
    const u64 row_bytes = n * res.words * 4;
    ctx.reserve(t, row_bytes);
    ctx.reserve(ws.cl_rows[0], row_bytes);
    ctx.reserve(ws.cl_rows[1], row_bytes);
    ctx.reserve(ws.cl_act, 8 * n * 4);
    ctx.reserve(cols, (res.words * 32 + n) * 4);
    DL_CUDA(cudaMemsetAsync(t.p, 0, row_bytes, ctx.stream));
    // levels: at most one per node (a shortest path), counted on the device
    const u64 top = max_level ? std::min(max_level, n) : n;
    ctx.reserve(ws.cl_levels, 3 * (top + 2) * 8);
    DL_CUDA(cudaMemsetAsync(ws.cl_levels.p, 0, 3 * (top + 2) * 8, ctx.stream));
    u32 *p = ws.cl_act.as<u32>();
    DL_CUDA(cudaMemsetAsync(p, 0xFF, 4 * n * 4, ctx.stream));          // tags: no level
    DL_CUDA(cudaMemsetAsync(p + 4 * n, 0, 2 * n * 4, ctx.stream));     // todo
    auto view = [&](u64 level) {
        const u64 in = (level + 1) & 1, out = level & 1;  // buffers by parity; at level 0 only the outputs are used
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
        v.count = ws.cl_levels.as<unsigned long long>();
        v.cnt = v.count + top + 2;
        v.deg = v.cnt + top + 2;
        return v;
    };
    DL_LAUNCH(ctx, K_PREP, 128.0 * h,
              pull_init_kernel<<<grid_for(res.words * 32 * 32, T256, ctx), T256, 0, ctx.stream>>>(
                  sh, view(0), src, h, cols.as<u32>()));
    auto push = [&](u64 level) {
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                  closure_push_kernel<<<grid_for(ne, PU_THREADS, ctx, 8), PU_THREADS, 0, ctx.stream>>>(
                      view(level), edges, ne, bits));
    };
    push(0);
    ctx.sync();
    const u64 n_hubs = ctx.host_scalars[0], n_seg = ctx.host_scalars[1];
    if (n_hubs) {
        ctx.reserve(ws.cl_hub_acc, n_hubs * res.words * 4);
        DL_CUDA(cudaMemsetAsync(ws.cl_hub_acc.p, 0, n_hubs * res.words * 4, ctx.stream));
    }
    u32 *hub_acc = ws.cl_hub_acc.as<u32>();
    auto level_step = [&](auto kc, u64 level) {
        constexpr int K = decltype(kc)::value;
        const u64 passes = (res.words + K * 128 - 1) / (K * 128);
        if (n_hubs)
            DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                      closure_pull_hub_kernel<K><<<grid_for(n_seg * passes * 32, PU_THREADS, ctx, 8), PU_THREADS, 0,
                                                   ctx.stream>>>(sh, view(level), roff, rval, ws.cl_segs.as<uint2>(),
                                                                 n_seg, ws.cl_hub_at.as<u32>(), hub_acc));
        // lanes for a target: 8 for rows of one or two chunks, else a warp
        auto kern = res.words == 32 ? closure_pull_thin_kernel<1>
                    : res.words == 64 ? closure_pull_thin_kernel<2> : closure_pull_kernel<K>;
        const u64 per = PU_THREADS / (res.words <= 64 ? 8 : 32);
        const u64 wave = resident_blocks(ctx, kern, PU_THREADS, 0);
        DL_LAUNCH(ctx, K_BITMAP_EXPAND, 0,
                  kern<<<(unsigned) std::min<u64>(wave, (n + per - 1) / per), PU_THREADS, 0, ctx.stream>>>(
                      sh, view(level), csr.off, roff, rval, ws.cl_hub_at.as<u32>(), hub_acc, t.as<u32>()));
        push(level);
    };
    // Levels are launched eight at a time: one after the fixpoint finds its
    // list empty and returns.
    res.cnt.assign(1, 0);
    res.deg.assign(1, 0);
    bool done = false;
    for (u64 level = 1; !done && level <= top;) {
        const u64 batch = std::min<u64>(8, top - level + 1);
        for (u64 k = 0; k < batch; ++k) {
            if (res.words <= 128) level_step(std::integral_constant<int, 1>(), level + k);
            else if (res.words <= 256) level_step(std::integral_constant<int, 2>(), level + k);
            else level_step(std::integral_constant<int, 3>(), level + k);
        }
        u64 *hs = ctx.host_scalars;
        DL_CUDA(cudaMemcpyAsync(hs, view(0).cnt + level, batch * 8, cudaMemcpyDeviceToHost, ctx.stream));
        DL_CUDA(cudaMemcpyAsync(hs + 8, view(0).deg + level, batch * 8, cudaMemcpyDeviceToHost, ctx.stream));
        ctx.sync();
        for (u64 k = 0; k < batch; ++k) {
            if (hs[k] == 0) {
                done = true;
                break;
            }
            res.cnt.push_back(hs[k]);
            res.deg.push_back(hs[8 + k]);
            ctx.prof_add_bytes(K_BITMAP_EXPAND, 4.0 * hs[8 + k]);
        }
        level += batch;
    }
    return res;
}

void bit_rows_count(Context &ctx, Run &r, u64 n, u64 words, u64 n_light, int bits, const u32 *place, u64 *counts) {
    ctx.reserve(r.cl_loff, (n + 1) * 8);
    ctx.reserve(r.cl_start, n * (words / 32) * 8);
    if (n_light)
        DL_LAUNCH(ctx, K_BITMAP_COLUMNS, 8.0 * n,
                  key_offsets_kernel<u64><<<grid_for(n + 1, T256, ctx), T256, 0, ctx.stream>>>(
                      r.words.as<u64>(), n_light, bits, n, r.cl_loff.as<u64>()));
    else
        DL_CUDA(cudaMemsetAsync(r.cl_loff.p, 0, (n + 1) * 8, ctx.stream));
    DL_LAUNCH(ctx, K_BITMAP_COLUMNS, 4.0 * n * words,
              closure_counts_kernel<<<grid_for(n * 32, T256, ctx), T256, 0, ctx.stream>>>(
                  r.bm_t.as<u32>(), n, (u32) words, r.words.as<u64>(), r.cl_loff.as<u64>(), (1ull << bits) - 1, place,
                  r.cl_start.as<uint2>(), counts));
}

u64 bit_rows_finish(Context &ctx, Run &r, u64 n, u64 words, const u64 *counts) {
    ctx.reserve(r.bm_first, (n + 1) * 8);
    const u64 tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    u64 *lb = ctx.lookback_words(tiles);
    u32 *tc = ctx.tile_counter(62);
    u64 *tot = &ctx.ctrl->scalar[49];
    DL_CUDA(cudaMemsetAsync(tc, 0, sizeof(u32), ctx.stream));
    DL_LAUNCH(ctx, K_BITMAP_EXTRACT, 16.0 * n,
              scan_kernel<SumValue><<<(unsigned) tiles, SCAN_THREADS, 0, ctx.stream>>>(
                  SumValue{counts}, n, r.bm_first.as<u64>(), lb, tc, ctx.next_epoch(), &ctx.ctrl->err, tot));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, tot, sizeof(u64), cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    r.from_bitmat = true;
    r.cl_rows = true;
    r.bm_n = n;
    r.bm_stride = r.bm_words = words;
    return ctx.host_scalars[0];
}

void closure_heavy_words(Context &ctx, const Csr &csr, u64 lo, u64 hi, int bits, const std::vector<u64> &src,
                         u64 max_level, std::vector<u64> &cnt, u64 &n_words) {
    Workspace &ws = ctx.ws;
    const u64 n = hi - lo;
    const int lb = bits_for(std::max<u64>(n, 2));
    // the instance's own edges and CSR over ranks from 0
    u32 ends[2];
    DL_CUDA(cudaMemcpyAsync(&ends[0], csr.off + lo, 4, cudaMemcpyDeviceToHost, ctx.stream));
    DL_CUDA(cudaMemcpyAsync(&ends[1], csr.off + hi, 4, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    const u64 ne = ends[1] - ends[0];
    ctx.reserve(ws.w0, ne * 8);
    ctx.reserve(ws.csr_off, (n + 1) * 4);
    ctx.reserve(ws.csr_val, ne * 4);
    u64 *e = ws.w0.as<u64>();
    DL_LAUNCH(ctx, K_PREP, 0,
              local_edges_kernel<<<grid_for(n, T256, ctx), T256, 0, ctx.stream>>>(csr.off, csr.val, lo, hi, lb, e));
    Csr local;
    local.off = ws.csr_off.as<u32>();
    local.val = ws.csr_val.as<u32>();
    local.n_keys = (u32) n;
    local.n_vals = ne;
    DL_LAUNCH(ctx, K_PREP, 0,
              key_offsets_kernel<u32><<<grid_for(n + 1, T256, ctx), T256, 0, ctx.stream>>>(e, ne, lb, n, local.off));
    DL_LAUNCH(ctx, K_PREP, 0,
              low_field_kernel<<<grid_for(ne, T256, ctx), T256, 0, ctx.stream>>>(e, ne, (1ull << lb) - 1, local.val));
    // as many sources at a time as 8 GiB of rows hold (sources are independent)
    const u64 at_once = std::max<u64>(1024, (8ull << 30) / (closure_pull_bytes(n, 1024) / 1024 + 1) / 1024 * 1024);
    DevBuf t, cols;
    try {
        for (u64 s0 = 0; s0 < src.size(); s0 += at_once) {
            const u64 h = std::min<u64>(at_once, src.size() - s0);
            std::vector<u64> l(h);
            for (u64 i = 0; i < h; ++i) l[i] = src[s0 + i] - lo;
            ctx.reserve(ws.cl_left, h * 8);
            DL_CUDA(cudaMemcpyAsync(ws.cl_left.p, l.data(), h * 8, cudaMemcpyHostToDevice, ctx.stream));
            ctx.sync();  // l is a host temporary
            const ClosureHeavy hv = closure_pull(ctx, local, e, ne, lb, n, ws.cl_left.as<u64>(), h, max_level, t, cols);
            u64 total = 0;
            if (hv.cnt.size() > cnt.size()) cnt.resize(hv.cnt.size(), 0);
            for (size_t d = 1; d < hv.cnt.size(); ++d) {
                cnt[d] += hv.cnt[d];
                total += hv.cnt[d];
            }
            grow_keeping(ctx, ws.jbuf[0], (n_words + total) * 8, n_words * 8);
            auto *count = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[46]);
            DL_CUDA(cudaMemsetAsync(count, 0, 8, ctx.stream));
            DL_LAUNCH(ctx, K_BITMAP_EXTRACT, 4.0 * n * hv.words + 8.0 * total,
                      heavy_words_kernel<<<grid_for(n * 32, T256, ctx), T256, 0, ctx.stream>>>(
                          t.as<u32>(), n, (u32) hv.words, cols.as<u32>(), lo, bits, ws.jbuf[0].as<u64>() + n_words,
                          total, count));
            n_words += total;
        }
    } catch (...) {
        ctx.give_back(t);
        ctx.give_back(cols);
        throw;
    }
    ctx.give_back(t);
    ctx.give_back(cols);
}

static bool tc_closure_run(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt,
                           PhaseTimer &pt, u64 &nfull) {
    Workspace &ws = ctx.ws;
    const u64 n = g.n_ids;
    const u64 max_level = opt.max_iterations > 0 ? (u64) opt.max_iterations + 1 : 0;
    pt.mark(PH_JOIN);
    ctx.reserve(ws.offsets, 2 * (CL_LEVELS + 1) * 8);
    u64 *cnt = ws.offsets.as<u64>(), *deg = cnt + CL_LEVELS + 1;
    ClosureLight light = closure_search(ctx, g.csr, 0, n, g.bits, nullptr, 1, 0, ne, CL_LEVELS + 1,
                                       max_level, cnt, deg);
    if (light.n_heavy) {
        const u64 need = closure_pull_bytes(n, light.n_heavy);
        if (need > ((u64) ctx.tune.bitmap_max_gib << 30)) return false;
        const u64 rows = n * pull_words(light.n_heavy) * 4;
        if (!ctx.room_for({{&r.bm_t, rows}, {&ws.cl_rows[0], rows}, {&ws.cl_rows[1], rows}, {&ws.cl_act, 8 * n * 4}},
                          {&ws.bitmat[0], &ws.bitmat[1]}))
            return false;
        // (now, before smaller requests take the cached buffers that were counted on)
        ctx.reserve(r.bm_t, rows);
        ctx.reserve(ws.cl_rows[0], rows);
        ctx.reserve(ws.cl_rows[1], rows);
        ctx.reserve(ws.cl_act, 8 * n * 4);
    }
    // host copies of the level counts (index d)
    std::vector<u64> hc(light.levels + 1, 0), hd(light.levels + 1, 0);
    if (light.levels) {
        DL_CUDA(cudaMemcpyAsync(hc.data(), cnt, (light.levels + 1) * 8, cudaMemcpyDeviceToHost, ctx.stream));
        DL_CUDA(cudaMemcpyAsync(hd.data(), deg, (light.levels + 1) * 8, cudaMemcpyDeviceToHost, ctx.stream));
    }
    pt.mark(PH_DEDUP);
    // light pairs in result order
    u64 *lw = ws.jbuf[0].as<u64>();
    if (light.n_words) {
        lw = closure_order(ctx, n, light.n_words, g.bits, g.bits);
    }
    adopt_words(ctx, r, lw, light.n_words);
    nfull = light.n_words;
    if (light.n_heavy) {
        ctx.reserve(ws.cl_left, light.n_heavy * 8);
        const u64 *src = radix_sort(ctx, ws.cl_heavy.as<u64>(), ws.cl_left.as<u64>(), light.n_heavy, Codec::Raw, g.bits);
        pt.mark(PH_MERGE);
        const ClosureHeavy heavy =
            closure_pull(ctx, g.csr, edges, ne, g.bits, n, src, light.n_heavy, max_level, r.bm_t, r.cl_cols);
        if (heavy.cnt.size() > hc.size()) {
            hc.resize(heavy.cnt.size(), 0);
            hd.resize(heavy.cnt.size(), 0);
        }
        for (size_t d = 1; d < heavy.cnt.size(); ++d) {
            hc[d] += heavy.cnt[d];
            hd[d] += heavy.deg[d];
            nfull += heavy.cnt[d];
        }
        pt.mark(PH_FINAL);
        u32 *place = r.cl_cols.as<u32>() + heavy.words * 32;
        DL_LAUNCH(ctx, K_BITMAP_COLUMNS, 4.0 * n,
                  heavy_below_kernel<<<grid_for(n, T256, ctx), T256, 0, ctx.stream>>>(r.cl_cols.as<u32>(), heavy.h, n,
                                                                                     place));
        ctx.reserve(ws.w0, (n + 1) * 8);
        bit_rows_count(ctx, r, n, heavy.words, light.n_words, g.bits, place, ws.w0.as<u64>());
        const u64 total = bit_rows_finish(ctx, r, n, heavy.words, ws.w0.as<u64>());
        if (total != nfull)
            throw Error(DL_ERR_INTERNAL, "closure holds " + std::to_string(total) + " tuples, expected " +
                                             std::to_string(nfull));
    } else {
        pt.mark(PH_FINAL);
        ctx.sync();  // hc, hd are host memory
    }
    // iteration k joins level k + 1 and finds level k + 2 (tc.cu:216-314); the
    // last one finds nothing, unless max_iterations ends the loop before
    u64 full = hc.size() > 1 ? hc[1] : 0;
    for (u64 k = 0;; ++k) {
        const u64 nnew = k + 2 < hc.size() ? hc[k + 2] : 0;
        const u64 join = k + 1 < hd.size() ? hd[k + 1] : 0;
        full += nnew;
        r.deltas.push_back((i64) nnew);
        r.joins.push_back((i64) join);
        r.fulls.push_back((i64) full);
        ctx.run_join_total += join;
        ctx.run_join_max = std::max(ctx.run_join_max, join);
        if (nnew == 0 || (opt.max_iterations > 0 && k + 1 >= (u64) opt.max_iterations)) break;
    }
    return true;
}

bool tc_closure(Context &ctx, Run &r, const Graph &g, const u64 *edges, u64 ne, const dl_options &opt,
                PhaseTimer &pt, u64 &nfull) {
    bool done = false;
    try {
        done = tc_closure_run(ctx, r, g, edges, ne, opt, pt, nfull);
    } catch (const Error &err) {
        if (err.status != DL_ERR_OUT_OF_MEMORY) throw;
    }
    if (!done) {
        r.deltas.clear();
        r.joins.clear();
        r.fulls.clear();
        r.from_bitmat = r.cl_rows = false;
        for (DevBuf *b : {&r.words, &r.bm_t, &r.bm_first, &r.cl_cols, &r.cl_loff, &r.cl_start}) ctx.give_back(*b);
        // the searches' buffers too: the form that runs instead may need their memory
        Workspace &ws = ctx.ws;
        for (DevBuf *b : {&ws.jbuf[0], &ws.jbuf[1], &ws.cl_rec, &ws.cl_left, &ws.cl_heavy, &ws.cl_seg, &ws.cl_seg_at,
                          &ws.cl_levels, &ws.cl_roff, &ws.cl_rval, &ws.cl_segs, &ws.cl_hub_at, &ws.cl_hub_acc,
                          &ws.cl_rows[0], &ws.cl_rows[1], &ws.cl_act})
            ctx.give_back(*b);
        r.n_words = nfull = 0;
        ctx.run_join_total = ctx.run_join_max = 0;
    }
    return done;
}

}  // namespace detail

void closure_extract_rows(Context &ctx, const Run &r, int32_t *out, u64 z0, u64 z1) {
    using namespace detail;
    const u32 *cols = r.cl_cols.as<u32>();
    const u64 chunks = r.bm_words / 32;
    const bool dense = (u64) r.info.output_rows >= r.bm_n * r.bm_words * 32 / 3;
    auto kern = r.bm_row_first ? (dense ? closure_rows_kernel<true, true> : closure_rows_kernel<false, true>)
                               : (dense ? closure_rows_kernel<true, false> : closure_rows_kernel<false, false>);
    const u64 wave = resident_blocks(ctx, kern, 256, 0);
    const unsigned grid = (unsigned) std::max<u64>(1, std::min<u64>(wave, ((z1 - z0) * chunks + 7) / 8));
    DL_LAUNCH(ctx, K_BITMAP_EXTRACT, 4.0 * (z1 - z0) * r.bm_words,
              kern<<<grid, 256, 0, ctx.stream>>>(
                  r.bm_t.as<u32>(), (u32) r.bm_words, cols, cols + r.bm_words * 32, r.cl_start.as<uint2>(), z0, z1,
                  r.bm_first.as<u64>(), r.words.as<u64>(), r.cl_loff.as<u64>(), (1ull << r.bits) - 1,
                  r.ids.as<int32_t>(), r.ids_affine, r.id_base, reinterpret_cast<u64 *>(out)));
    if (r.n_words <= MERGE_PAIRS) return;
    const u64 parts = (z1 - z0) * chunks;
    const unsigned mg = grid_for(parts * 32, 256, ctx, 8);
    const u32 take = (u32) std::max<u64>(1, std::min<u64>(32, parts / (mg * 8)));
    DL_LAUNCH(ctx, K_BITMAP_EXTRACT, 0,
              closure_merge_kernel<<<mg, 256, 0, ctx.stream>>>(
                  r.bm_t.as<u32>(), (u32) r.bm_words, cols, cols + r.bm_words * 32, r.cl_start.as<uint2>(), z0, z1,
                  r.bm_first.as<u64>(), r.words.as<u64>(), r.cl_loff.as<u64>(), (1ull << r.bits) - 1,
                  r.ids.as<int32_t>(), r.ids_affine, r.id_base, take, reinterpret_cast<u64 *>(out)));
}

}  // namespace dl
