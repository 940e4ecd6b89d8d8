// single_join as a union of neighbour lists per output key.
//
// The reference joins R with itself, sorts the output and drops the
// duplicates (single_join.cu:135-309): 1.1e9 join words of 8 bytes through a
// sort for 10M rows over 90K ids. The rows of one output key z are the union of
// the in-neighbour lists of z's in-neighbours, so a CTA builds that union as a
// bitmap over the node ranks in shared memory -- no word of the join output
// ever reaches HBM -- and stores it as one row of a bit matrix; the result rows
// are written from the matrix when they are copied out (dl_closure.cu).
//
// Measured on B200, 10M rows over 90K ids, 1.04e9 result rows: 52.7 ms by the
// sort, 5.8 ms here (unions 1.5, rows 3.4, the input's sort 0.4).
#include "dl_closure.h"
#include "dl_pull.cuh"

namespace dl {
namespace detail {
namespace {

constexpr int SJ_THREADS = 256;
constexpr int SJ_WARPS = SJ_THREADS / 32;

__global__ void __launch_bounds__(256) degree_total_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val,
                                                           u64 n, unsigned long long *__restrict__ sum) {
    u64 s = 0;
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64) gridDim.x * blockDim.x) {
        const u32 y = val[i];
        s += off[y + 1] - off[y];
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(sum, (unsigned long long) s);
}

__global__ void identity_kernel(u32 *__restrict__ cols, u64 n, u64 padded) {
    for (u64 i = (u64) blockIdx.x * blockDim.x + threadIdx.x; i < padded; i += (u64) gridDim.x * blockDim.x)
        cols[i] = i < n ? (u32) i : 0xFFFFFFFFu;
}

// A CTA per output key z (persistent, next key from a counter). Warps take 32
// in-neighbours b of z at a time and OR the members of b's list into the
// bitmap; lists of 16 members or more on average are read list by list (128
// bytes a load, four loads in flight), shorter ones in windows of 32 members
// of consecutive lists. The row is then stored 16 bytes a thread, counted by chunk
// of 1024 columns, and cleared. Bound by the shared-memory atomics and the list
// reads from L2 (4 bytes a join word).
__global__ void __launch_bounds__(SJ_THREADS)
self_join_kernel(const u32 *__restrict__ off, const u32 *__restrict__ val, u64 n, u32 words, u32 *__restrict__ t,
                 uint2 *__restrict__ start, u64 *__restrict__ counts, unsigned long long *__restrict__ next) {
    extern __shared__ __align__(16) u32 smem[];
    u32 *row = smem;                 // words
    u32 *chunk = row + words;        // set bits of each chunk
    __shared__ u32 s_z, s_group;
    const u32 tid = threadIdx.x, lane = tid & 31;
    const u32 lt = lanemask_lt(), le = lane == 31 ? ~0u : (2u << lane) - 1;
    const u32 chunks = words / 32;
    __shared__ u32 wbeg[SJ_WARPS][32], wpre[SJ_WARPS][32];
    const u32 warp = tid >> 5;
    for (u32 k = tid; k < words; k += SJ_THREADS) row[k] = 0;
    for (;;) {
        if (tid == 0) {
            const u64 z = atomicAdd(next, 1ull);
            s_z = z < n ? (u32) z : 0xFFFFFFFFu;
            s_group = 0;
        }
        __syncthreads();  // the key; the row is clear
        const u32 z = s_z;
        if (z == 0xFFFFFFFFu) break;
        const u32 b0 = __ldg(off + z), nb = __ldg(off + z + 1) - b0;
        auto put = [&](u32 x) { atomicOr(&row[x >> 5], 1u << (x & 31)); };
        for (;;) {
            u32 g = 0;
            if (lane == 0) g = atomicAdd(&s_group, 32u);
            g = __shfl_sync(0xffffffffu, g, 0);
            if (g >= nb) break;
            u32 beg = 0, deg = 0;
            if (g + lane < nb) {
                const u32 b = __ldg(val + b0 + g + lane);
                beg = __ldg(off + b);
                deg = __ldg(off + b + 1) - beg;
            }
            const u32 nz = __ballot_sync(0xffffffffu, deg != 0);
            if (!nz) continue;
            const u32 incl = warp_inclusive_sum(deg);
            const u32 total = __shfl_sync(0xffffffffu, incl, 31);
            if (total >= 16u * __popc(nz)) {
                for (u32 m = nz; m; m &= m - 1) {
                    const u32 j = __ffs(m) - 1;
                    const u32 *list = val + __shfl_sync(0xffffffffu, beg, j);
                    const u32 d = __shfl_sync(0xffffffffu, deg, j);
                    for (u32 i = lane; i < d; i += 128) {
                        u32 x[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (i + 32 * q < d) x[q] = __ldg(list + i + 32 * q);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (i + 32 * q < d) put(x[q]);
                    }
                }
            } else {
                const u32 rk = __popc(nz & lt);
                if (deg) {
                    wbeg[warp][rk] = beg;
                    wpre[warp][rk] = incl - deg;
                }
                __syncwarp();
                const u32 nrows = __popc(nz);
                const u32 cb = lane < nrows ? wbeg[warp][lane] : 0u;
                const u32 pre = lane < nrows ? wpre[warp][lane] : 0xFFFFFFFFu;
                __syncwarp();
                int base = -1;  // last list started before the window
                for (u32 i0 = 0; i0 < total; i0 += 32) {
                    const u32 st = (pre - i0) < 32u ? 1u << (pre - i0) : 0u;
                    const u32 starts = __reduce_or_sync(0xffffffffu, st);
                    const int o = base + __popc(starts & le);
                    base += __popc(starts);
                    const u32 ob = __shfl_sync(0xffffffffu, cb, o), op = __shfl_sync(0xffffffffu, pre, o);
                    if (i0 + lane < total) put(__ldg(val + ob + (i0 + lane - op)));
                }
            }
        }
        __syncthreads();  // the row is complete
        // store, count and clear: eight threads to a chunk
        u32 *dst = t + (u64) z * words;
        for (u32 k0 = 0; k0 < words; k0 += SJ_THREADS * 4) {
            const u32 k = k0 + tid * 4;
            u32 c = 0;
            if (k < words) {
                uint4 *p = reinterpret_cast<uint4 *>(row + k);
                const uint4 v = *p;
                *p = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4 *>(dst + k) = v;
                c = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if ((lane & 7) == 0 && k < words) chunk[k >> 5] = c;
        }
        __syncthreads();  // chunk counts
        if (warp == 0) {
            u32 run = 0;
            for (u32 c0 = 0; c0 < chunks; c0 += 32) {
                const u32 c = c0 + lane < chunks ? chunk[c0 + lane] : 0u;
                const u32 in = warp_inclusive_sum(c);
                if (c0 + lane < chunks) start[(u64) z * chunks + c0 + lane] = make_uint2(run + in - c, 0u);
                run += __shfl_sync(0xffffffffu, in, 31);
            }
            if (lane == 0) counts[z] = run;
        }
        // (the next key is taken by thread 0 after its share of this)
    }
}

}  // namespace

u64 *edges_by_other(Context &ctx, const u64 *edges, u64 ne, int bits, DevBuf &a, DevBuf &b) {
    ctx.reserve(a, ne * 8);
    ctx.reserve(b, ne * 8);
    DL_LAUNCH(ctx, K_PREP, 16.0 * ne,
              pull_swap_kernel<<<grid_for(ne, T256, ctx), T256, 0, ctx.stream>>>(edges, ne, bits, a.as<u64>()));
    int w[8], nw = 0;
    for (int k = 0; k < bits; k += 8) w[nw++] = bits + k;
    return radix_sort_windows(ctx, a.as<u64>(), b.as<u64>(), ne, w, nw);
}

u64 self_join_total(Context &ctx, const Csr &in) {
    auto *sum = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[24]);
    DL_CUDA(cudaMemsetAsync(sum, 0, 8, ctx.stream));
    DL_LAUNCH(ctx, K_JOIN_COUNT, 4.0 * in.n_vals,
              degree_total_kernel<<<grid_for(in.n_vals, T256, ctx, 8), T256, 0, ctx.stream>>>(in.off, in.val, in.n_vals,
                                                                                             sum));
    DL_CUDA(cudaMemcpyAsync(ctx.host_scalars, sum, 8, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    return ctx.host_scalars[0];
}

bool self_join_rows(Context &ctx, Run &r, const Csr &in, u64 total, PhaseTimer &pt, u64 &rows) {
    Workspace &ws = ctx.ws;
    const u64 n = in.n_keys, words = (n + 1023) / 1024 * 32, chunks = words / 32;
    const size_t smem = (words + chunks) * 4;
    const u64 bytes = n * words * 4;
    // The matrix is written and read once, the join words through the sort a
    // dozen times: worth it up to 16 bytes of matrix per join word (a result
    // row per 1K bits or so).
    if (smem + 4096 > 227 * 1024 || bytes > 16 * total || bytes > ((u64) ctx.tune.bitmap_max_gib << 30)) return false;
    if (!ctx.room_for({{&r.bm_t, bytes}}, {&ws.bitmat[0], &ws.bitmat[1], &ws.cl_rows[0], &ws.cl_rows[1]})) return false;
    pt.mark(PH_JOIN);
    try {
        ctx.reserve(r.bm_t, bytes);
        ctx.reserve(r.cl_start, n * chunks * 8);
        ctx.reserve(r.cl_cols, (words * 32 + n) * 4);
        ctx.reserve(r.cl_loff, (n + 1) * 8);
        ctx.reserve(r.bm_first, (n + 1) * 8);
        ctx.reserve(ws.offsets, (n + 1) * 8);
    } catch (const Error &err) {
        if (err.status != DL_ERR_OUT_OF_MEMORY) throw;
        for (DevBuf *b : {&r.bm_t, &r.cl_start, &r.cl_cols, &r.cl_loff, &r.bm_first}) ctx.give_back(*b);
        return false;
    }
    DL_CUDA(cudaMemsetAsync(r.cl_loff.p, 0, (n + 1) * 8, ctx.stream));  // no light pairs
    DL_LAUNCH(ctx, K_PREP, 4.0 * words * 32,
              identity_kernel<<<grid_for(words * 32, T256, ctx), T256, 0, ctx.stream>>>(r.cl_cols.as<u32>(), n,
                                                                                       words * 32));
    auto *next = reinterpret_cast<unsigned long long *>(&ctx.ctrl->scalar[24]);
    DL_CUDA(cudaMemsetAsync(next, 0, 8, ctx.stream));
    DL_CUDA(cudaFuncSetAttribute(self_join_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    int per_sm = 0;
    DL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, self_join_kernel, SJ_THREADS, smem));
    const u64 wave = (u64) ctx.sm_count * std::max(per_sm, 1);
    DL_LAUNCH(ctx, K_BITMAP_EXPAND, 4.0 * total + (double) bytes,
              self_join_kernel<<<(unsigned) std::min<u64>(wave, n), SJ_THREADS, smem, ctx.stream>>>(
                  in.off, in.val, n, (u32) words, r.bm_t.as<u32>(), r.cl_start.as<uint2>(), ws.offsets.as<u64>(), next));
    pt.mark(PH_DEDUP);
    rows = bit_rows_finish(ctx, r, n, words, ws.offsets.as<u64>());
    return true;
}

}  // namespace detail
}  // namespace dl
