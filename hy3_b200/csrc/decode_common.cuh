/*
 * decode_common.cuh -- helpers of the decode kernel: the argument block, the unit schedule
 * (segment / locate), shared-memory, mbarrier and bulk-copy primitives with bounded waits, and the
 * receiving side of the sequence-shard exchange.  Everything lives in an unnamed namespace: each
 * translation unit gets its own copy.
 */
#ifndef HY3A_DECODE_COMMON_CUH
#define HY3A_DECODE_COMMON_CUH

#include <cuda_fp16.h>
#include <math.h>

#include "ctx.h"
#include "decode_plan.h"

/* Argument block of the decode kernels (filled by hy3a_launch_decode / hy3a_decode_noalloc in decode.cu). */
struct hy3a_decode_args {
    const float *q;
    size_t q_stride;
    float *out;
    size_t out_stride;
    float *user_partials; /* NULL or [n][8*kv_heads][130] */
    /* sequence sharding with the exchange inside the kernel (n_dest = world size > 0): the CTA that completes a
     * (row, KV head) segment stores its 8 records, as 16-byte lines {value, flag, value, flag}, into every other
     * rank's gather buffer (dest[r], already offset to this rank's slice there), then polls the lines the other
     * ranks store into its own buffer, folds all ranks' records in rank order and writes the final output.
     * flag = use count of the (slot, segment) + 1, kept in shard_round on every rank.                          */
    int n_dest, my_rank;
    uint4 *dest[8];
    const uint4 *gathered;        /* local: [n_dest][n*kv_heads*8][65] lines of the slot */
    unsigned *shard_round;        /* local: [n*kv_heads*8] uses of the slot so far, per head */
    float *scratch;       /* merge records: [(gridDim.x + n*kv_heads)][8][HY3A_REC_FLOATS] */
    unsigned int *counters; /* [n_counters][8]: arrivals per (row, KV head) segment and query head (a spread fold counts in the first), then [n_counters]: finished folds */
    int n_counters;
    int spread;           /* > 0: CTA-aligned segments spread their fold over up to this many of their CTAs (the whole grid is resident) */
    unsigned int *err;
    int layer;
    int cluster;          /* 0: the grid; 2, 4, 8: a cluster of that many CTAs per (row, KV head) */
    /* fused step (fused != 0): the kernel itself normalises + rotates the queries read from q_in and
     * the CTA that streams the page of the newest slot quantises and appends the new K / V row   */
    int fused;
    int wait_first;       /* the preceding kernel may be the one that writes the batch descriptor */
    int early_prefetch;   /* pages below the newest slots may be fetched before griddepcontrol.wait */
    const float *q_in, *k_in, *v_in;
    size_t qi_stride, ki_stride, vi_stride;
    float *q_out;         /* optional: normalised + rotated queries, fp32 [n][64][128] */
    size_t q_out_stride;
    const float *norm_w;  /* [2][128] of this layer */
    float eps;
    hy3a_rope_params rope;
    int stages;           /* staged variant: stages of the shared-memory ring (2..8) */
    int prefix_bytes;     /* bytes reserved for the page-count prefix */
};

/* the INT8 decode kernel (decode_umma.cu) */
int hy3a_decode_umma_cluster_cap(hy3a_ctx *ctx, int cl);
/* clusters of cl CTAs (decode.cu): a launch, and how many of a kernel fit on the current device at once */
cudaError_t hy3a_launch_cluster(hy3a_ctx *ctx, const void *fn, int cl, int clusters, int threads, size_t smem, void **args);
int hy3a_cluster_cap(const void *fn, int cl, int threads, size_t smem);
cudaError_t hy3a_launch_decode_umma(hy3a_ctx *ctx, const hy3a_cache_view &cv, const hy3a_batch_view &bv, hy3a_decode_args &a);

namespace {

constexpr int kSmemMax = 232448 - 128;                 /* opt-in limit per block minus the 128 bytes that hy3a_decode_kernel declares statically */
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

typedef hy3a_decode_args decode_args;

struct segment {
    int row, hl, pages, p_begin, p_end, sidx, len, seq;
    long long seg_u0, seg_u1;
};

/* Locate the (row, local head) segment that contains unit u and the page range of it that
 * falls into [u, u_end).                                                                   */
__device__ __forceinline__ segment locate_pages(const int *s_prefix, int n, int G, long long u, long long u_end) {
    segment sg;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if ((long long)G * s_prefix[mid] <= u) lo = mid; else hi = mid - 1;
    }
    sg.row = lo;
    sg.pages = s_prefix[lo + 1] - s_prefix[lo];
    const long long row_u0 = (long long)G * s_prefix[lo];
    sg.hl = (int)((unsigned)(u - row_u0) / (unsigned)sg.pages);   /* both fit 32 bits: a 64-bit division costs hundreds of cycles */
    sg.seg_u0 = row_u0 + (long long)sg.hl * sg.pages;
    sg.seg_u1 = sg.seg_u0 + sg.pages;
    sg.p_begin = (int)(u - sg.seg_u0);
    sg.p_end = (int)((sg.seg_u1 < u_end ? sg.seg_u1 : u_end) - sg.seg_u0);
    sg.sidx = lo * G + sg.hl;
    return sg;
}
__device__ __forceinline__ segment locate(const int *s_prefix, const hy3a_batch_view &batch, int n, int G, long long u, long long u_end) {
    segment sg = locate_pages(s_prefix, n, G, u, u_end);
    sg.len = batch.slot[sg.row] + 1;
    sg.seq = batch.seq[sg.row];
    return sg;
}
/* the rows of the producer's warp: lane = row, up to 32 of them; its segments then wait for no load */
struct lane_rows { int slot, seq; };
__device__ __forceinline__ lane_rows load_rows(const hy3a_batch_view &batch, int n, int lane) {
    lane_rows r = {-1, 0};
    if (n <= 32 && lane < n) { r.slot = batch.slot[lane]; r.seq = batch.seq[lane]; }
    return r;
}
__device__ __forceinline__ segment locate(const int *s_prefix, const hy3a_batch_view &batch, const lane_rows &rows, int n, int G, long long u, long long u_end) {
    if (n > 32) return locate(s_prefix, batch, n, G, u, u_end);
    segment sg = locate_pages(s_prefix, n, G, u, u_end);
    sg.len = __shfl_sync(0xffffffffu, rows.slot, sg.row) + 1;
    sg.seq = __shfl_sync(0xffffffffu, rows.seq, sg.row);
    return sg;
}

/* 2 to 32 rows with fewer than four CTAs per segment: the least number of pages L for which pieces of at most L pages fit the
 * grid (sum of ceil(pages / L) over the rows <= CTAs per head), a lane per row; 0: not this case.  Shares in proportion (plan_cta, below)
 * round down, and a row that just misses its second CTA holds the launch up: 8 rows of 22 to 56 pages x 8 heads on 148 CTAs get at
 * most 24 pages a CTA that way, 19 this way (INT4: 27.3 -> 21.1 us a layer with the straddling split that 24 pages fall back to;
 * 12 rows of up to 2 646 tokens 27.1 -> 17.7, FP16 24.9 -> 20.6).  The FP16 / INT4 kernel only: the INT8 kernel would gain
 * as much there (8 rows of 300 to 8 000 x 8 heads 26.6 -> 18.4, 12 up to 2 646 28.2 -> 15.8, 30 up to 16 000 x 2 38.4 -> 32.8), but its batch-1
 * launch loses 1 % with this code in the planning warp (32 768 tokens 17.60 -> 17.78, 16 000 12.94 -> 13.11), at the same registers and
 * spills.  Called by a whole warp, the result is the same in every lane. */
__device__ __noinline__ unsigned even_piece_search(const int *s_prefix, int n, int G, unsigned grid, int lane) {
    const unsigned P = (unsigned)s_prefix[n], cap = grid / (unsigned)G, p = lane < n ? (unsigned)(s_prefix[lane + 1] - s_prefix[lane]) : 0u;
    if (P == 0u) return 0u;
    return hy3a_least_piece((P + cap - 1u) / cap, hy3a_piece_bound(P, cap, (unsigned)n, __reduce_max_sync(0xffffffffu, p)), cap,
                            [&](unsigned L) { return __reduce_add_sync(0xffffffffu, (p + L - 1u) / L); });
}
/* the pages of a cluster's CTA, in units */
template <int CL>
__device__ __forceinline__ void cluster_share(const int *s_prefix, int G, int cta, long long &u_begin, long long &u_end) {
    const int seg = cta / CL, k = cta - seg * CL, row = seg / G, hl = seg - row * G;
    const int p = s_prefix[row + 1] - s_prefix[row];
    const long long seg0 = (long long)G * s_prefix[row] + (long long)hl * p;
    u_begin = seg0 + (long long)k * p / CL;
    u_end = seg0 + (long long)(k + 1) * p / CL;
}
/* ---- the CTA's range of units.  One warp (the producer's, which then starts its copies without a word from the others) plans for the CTA.
 *  - few segments (n G < grid): every segment gets its own whole number of CTAs, for pieces of at most L pages or (1 row, more than 32,
 *    INT8) roughly in proportion to its pages, so that no CTA straddles two segments (a straddling CTA pays the query set-up and the
 *    fold twice and becomes the critical path of a small batch).  In proportion is balanced to a page with few segments; when the
 *    segments are about as many as the CTAs the rounding leaves some with far more pages than the even share (64 rows of one KV head
 *    on 148 CTAs: up to 1.75 x), so with fewer than four CTAs per segment it is kept only within 5/4 of the even share;
 *  - else one contiguous, equally sized range per CTA over all units.
 * In both, never more CTAs than units, and the CTAs sharing a segment are contiguous.  A lane takes a row, 32 at a time, and the
 * arithmetic is 32-bit (T) unless the units are too many for it: this stands in front of every launch's first copy.  Planned by
 * every warp for itself, row by row and with 64-bit divisions, it took 1.1 us of a launch of one row, 3.3 of 8 rows, 2.3 of 64. */
struct cta_plan { long long u0, u1; int first, pieces, aligned; };
template <int DT, class T>
__device__ __noinline__ void plan_cta(cta_plan *out, const int *s_prefix, int n, int G, unsigned grid, unsigned cta, int lane) {
    const unsigned Pn = (unsigned)s_prefix[n], g = (unsigned)G;
    const T U = (T)Pn * g;
    auto pages = [&](int r) { return r < n ? (unsigned)(s_prefix[r + 1] - s_prefix[r]) : 0u; };
    unsigned ne = 0, L = 0;
    for (int r = lane; r < n; r += 32) ne += pages(r) != 0u;
    ne = __reduce_add_sync(0xffffffffu, ne);
    const T spare = (T)grid - (T)ne * g;
    auto pieces = [&](unsigned p) {
        const unsigned c = L ? (p + L - 1u) / L : min(1u + (unsigned)(spare * p / U), hy3a_most_pieces(p));
        return c < p ? c : p;
    };
    bool aligned = Pn != 0u && (unsigned)n * g < grid;
    if (aligned && DT != 1 && hy3a_even_applies(n, G, grid)) {
        L = even_piece_search(s_prefix, n, G, grid, lane);
        aligned = hy3a_even_accepted(L, Pn, G, grid);
    } else if (aligned && (unsigned)n * g * 4u > grid) {
        unsigned worst = 0;
        for (int r = lane; r < n; r += 32) {
            const unsigned p = pages(r), c = p ? pieces(p) : 1u;
            worst = max(worst, (p + c - 1u) / c);
        }
        worst = __reduce_max_sync(0xffffffffu, worst);
        aligned = (T)worst * 4u <= (U + grid - 1u) / grid * 5u + 4u;
    }
    if (lane == 0) {
        const T C = U < grid ? U : (T)grid;
        const bool mine = !aligned && cta < C;
        out->u0 = mine ? (long long)(cta * U / C) : 0;
        out->u1 = mine ? (long long)((cta + 1u) * U / C) : 0;
        out->first = 0; out->pieces = 1; out->aligned = aligned;
    }
    __syncwarp();
    unsigned base0 = 0;
    for (int r0 = 0; aligned && r0 < n && base0 <= cta; r0 += 32) {
        const unsigned p = pages(r0 + lane), c = p ? pieces(p) : 0u;
        unsigned end = c * g;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += t;
        }
        const unsigned base = base0 + end - c * g;
        if (c && cta >= base && cta < base0 + end) {      /* one lane at most */
            const unsigned idx = cta - base, hl = idx / c, k = idx - hl * c, k1 = k + 1u;
            const long long seg0 = (long long)g * s_prefix[r0 + lane] + (long long)hl * p;
            T b = (T)k * p / c, e = (T)k1 * p / c;
            /* The CTAs with the highest indices are dispatched last, onto the SMs that the preceding launch's folding CTAs held
             * longest: they start their ring fill late and would finish last (and then fold, and hold their SMs again).  In a
             * single-row grid the last HY3A_LATE pieces of the INT8 kernel therefore take HY3A_LATE_CUT pages less each and the other
             * pieces of that segment share them: 18.83 instead of 19.02 us per launch on the benchmark. */
            if (DT == 1 && ne == 1u && hl == g - 1u && c > 2u * HY3A_LATE && p >= 8u * c && Pn < (1u << 23)) {
                const unsigned pp = p + HY3A_LATE * HY3A_LATE_CUT, late = c - HY3A_LATE;
                b = (T)k * pp / c - HY3A_LATE_CUT * (k > late ? k - late : 0u);
                e = (T)k1 * pp / c - HY3A_LATE_CUT * (k1 > late ? k1 - late : 0u);
            }
            out->u0 = seg0 + (long long)b; out->u1 = seg0 + (long long)e;
            out->first = (int)(base + hl * c); out->pieces = (int)c;
        }
        base0 += __shfl_sync(0xffffffffu, end, 31);
    }
}
__device__ __forceinline__ int pages_of_slot(int slot) { return slot >= 0 ? slot / HY3A_PT + 1 : 0; }
/* the planning warp: prefix of pages per row (rows beyond 32 come as page counts in s_prefix), then the plan, in shared memory */
template <int DT, int CL>
__device__ __forceinline__ void plan(cta_plan *out, int *s_prefix, int slot /* of row `lane`, -1 behind the last */, int n, int G, unsigned grid, int cta, int lane) {
    int carry = 0;
    for (int base = 0; base < n; base += 32) {
        const int i = base + lane;
        int v = n <= 32 ? pages_of_slot(slot) : (i < n ? s_prefix[i + 1] : 0);
        if (n > 1) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
        }
        if (i < n) s_prefix[i + 1] = v + carry;
        carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) s_prefix[0] = 0;
    __syncwarp();
    if (CL) {
        if (lane == 0) {
            cluster_share<CL ? CL : 1>(s_prefix, G, cta, out->u0, out->u1);
            out->first = 0; out->pieces = 1; out->aligned = 1;
        }
    } else if ((unsigned long long)(unsigned)s_prefix[n] * (unsigned)G * (grid + 1u) >> 32) {
        plan_cta<DT, unsigned long long>(out, s_prefix, n, G, grid, (unsigned)cta, lane);
    } else {
        plan_cta<DT, unsigned>(out, s_prefix, n, G, grid, (unsigned)cta, lane);
    }
    __syncwarp();
}
/* pieces of a segment where units are dealt in equal ranges: CTA of unit u is the least c with (c + 1) U / C > u */
__device__ __forceinline__ int cta_of_unit(long long u, long long U, int C) {
    const unsigned long long x = (unsigned long long)(u + 1) * (unsigned)C + (unsigned long long)U - 1ull;
    return (int)((x >> 32 ? x / (unsigned long long)U : (unsigned)x / (unsigned)U) - 1ull);
}

/* ---- shared-memory / mbarrier / bulk-copy primitives ---------------------------------- */
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint4 lds16(unsigned addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned lds4(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
/* Blocking flavour of the wait: mbarrier.try_wait suspends the thread in hardware (up to the hinted time) instead of
 * spinning, so that waiting warps do not take issue slots from working ones.  Bounded in time (about half a second)
 * through the global timer; on expiry same protocol as mbar_wait below. */
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity, unsigned hint_ns) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(hint_ns) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_blocking(unsigned bar, unsigned parity, volatile int *abort_flag, unsigned *err, unsigned where) {
    if (mbar_try(bar, parity, 2000u)) return true;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (unsigned i = 0; i < (1u << 22); i++) {
        if (mbar_try(bar, parity, 20000u)) return true;
        if (*abort_flag) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        /* both a real amount of waiting and the clock must agree: the global timer can step (it is re-synchronised with the
         * host clock), and a try_wait may return long before its hint */
        if (i >= (1u << 13) && t1 - t0 > 500000000ull) break;
    }
    *abort_flag = 1;
    if (atomicCAS(err, 0u, 1u) == 0u) { err[1] = where; err[2] = blockIdx.x; err[3] = bar; }
    return false;
}
/* The KV stream is read once per step: its lines are marked evict-first in L2, so that what is small and re-read by every
 * launch (queries, batch descriptor, block table, norm weights, merge records) stays resident beside 68 MB of pages per launch. */
__device__ __forceinline__ unsigned long long l2_evict_first_policy() {
    unsigned long long pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void bulk_g2s(unsigned dst, const void *src, unsigned bytes, unsigned bar, unsigned long long policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
}
/* Bounded wait: gives up after ~2^22 polls (far beyond any legitimate wait), records the
 * failure in the device error word and raises the CTA-wide abort flag; once the flag is up
 * every later wait returns at once, so all warps keep the same control flow and the kernel
 * runs to its end (with a meaningless result that the host discards on seeing the error). */
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int *abort_flag, unsigned *err, unsigned where) {
    if (mbar_test(bar, parity)) return true;
    for (unsigned i = 0; i < (1u << 22); i++) {
        if (mbar_test(bar, parity)) return true;
        if ((i & 63u) == 63u) { if (*abort_flag) return false; __nanosleep(32); }
    }
    *abort_flag = 1;
    if (atomicCAS(err, 0u, 1u) == 0u) err[1] = where;
    return false;
}
/* ---- pieces both decode kernels use */
/* Folds skip a record only where its denominator is 0, the mark of a piece without keys, and divide by whatever else it is: a NaN score
 * reaches the output on every route, whichever piece its key is in (a test for l > 0 would drop that piece's other keys too). */
__device__ __forceinline__ float inv_sum(float l) { return l == 0.f ? 0.f : 1.f / l; }
/* a row without keys: zero output, or empty partial records {-inf, 0, 0...} (hy3_gpu.cu:197-199); `out`, `partials`: the row's owned heads */
__device__ __forceinline__ void write_empty_row(float *out, float *partials, int G, int t, int threads) {
#pragma unroll 1
    for (int e = t; e < G * 8 * HY3A_D; e += threads) {
        if (partials) {
            float *rec = partials + (e / HY3A_D) * HY3A_PARTIAL_FLOATS;
            rec[2 + e % HY3A_D] = 0.f;
            if (e % HY3A_D == 0) { rec[0] = -INFINITY; rec[1] = 0.f; }
        } else {
            out[e] = 0.f;
        }
    }
}
#define HY3A_EMPTY_ROW(i, t, threads) \
    write_empty_row(a.out + (size_t)(i) * a.out_stride + (size_t)cache.kv_head_begin * 8 * HY3A_D, \
                    a.user_partials ? a.user_partials + (size_t)(i) * G * 8 * HY3A_PARTIAL_FLOATS : nullptr, G, t, threads)
/* ---- a segment that several CTAs share, one warp per query head.  Records in memory: {acc[128], m, l, -, -}.  A piece without keys (l = 0)
 * leaves acc = 0, and its weight in the fold is 0: the sums of a piece whose scores are all -inf may hold 0 x infinity (a V scale). */
__device__ __forceinline__ void store_record(float *rec, int lane, float M, float L, const float (&acc)[4]) {
    *reinterpret_cast<float4 *>(rec + 4 * lane) = L != 0.f ? make_float4(acc[0], acc[1], acc[2], acc[3]) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane == 0) *reinterpret_cast<float2 *>(rec + HY3A_D) = make_float2(M, L);
}
__device__ __forceinline__ float warp_max(float x) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
/* One warp folds the np records of its head, in their order, with the rule of hy3_gpu.cu:233-247; rec0: record of piece 0, records 8 heads
 * apart.  A lane holds one record's {m, l}, so that the maximum, the weights and the denominator are one step instead of a dependent
 * one per record; their acc land in `slots` (at most 32) places of 512 bytes in shared memory, `stride` bytes apart, which are this
 * warp's own (a lane reads back what it copied).  How many there are does not change a bit of the result. */
__device__ __forceinline__ void fold_records(const float *rec0, int np, uint8_t *zone, unsigned stride, int slots, int lane, float &M, float &L, float (&acc)[4]) {
    constexpr size_t kStep = 8 * HY3A_REC_FLOATS;
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    auto fetch = [&](int c0, int nc) {
        const float *rec = rec0 + c0 * kStep + 4 * lane;
        unsigned dst = smem_u32(zone) + 16u * (unsigned)lane;
#pragma unroll 4
        for (int c = 0; c < nc; c++, dst += stride, rec += kStep) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rec) : "memory");
    };
    auto ml_of = [&](int c) {      /* {m, l} of a record; l = 0: a piece without keys */
        return c < np ? __ldcg(reinterpret_cast<const float2 *>(rec0 + c * kStep + HY3A_D)) : make_float2(-INFINITY, 0.f);
    };
    fetch(0, min(slots, np));
    const float2 ml0 = ml_of(lane);
    float mx = ml0.y != 0.f ? ml0.x : -INFINITY;
#pragma unroll 1
    for (int c = lane + 32; c - lane < np; c += 32) {
        const float2 ml = ml_of(c);
        mx = fmaxf(mx, ml.y != 0.f ? ml.x : -INFINITY);
    }
    M = warp_max(mx);
    auto weight = [&](float2 ml) { return ml.y != 0.f ? ex2(ml.x - M) : 0.f; };
    const float w0 = weight(ml0);
    L = ml0.y * w0;
#pragma unroll 1
    for (int c = lane + 32; c - lane < np; c += 32) {
        const float2 ml = ml_of(c);
        L += ml.y * weight(ml);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
#pragma unroll 1
    for (int c0 = 0; c0 < np; c0 += slots) {
        const int nc = min(slots, np - c0);
        if (c0) fetch(c0, nc);
        const float w = c0 ? weight(ml_of(lane < nc ? c0 + lane : np)) : w0;
        asm volatile("cp.async.wait_all;" ::: "memory");
        const uint8_t *src = zone + 16 * lane;
#pragma unroll 4
        for (int c = 0; c < nc; c++, src += stride) {
            const float f = __shfl_sync(0xffffffffu, w, c);
            const float4 v = *reinterpret_cast<const float4 *>(src);
            acc[0] = fmaf(v.x, f, acc[0]); acc[1] = fmaf(v.y, f, acc[1]); acc[2] = fmaf(v.z, f, acc[2]); acc[3] = fmaf(v.w, f, acc[3]);
        }
    }
}
/* The warp leaves its piece's record and counts its head's arrivals; true: it came last and has folded all pieces.  Nothing but the
 * head's own chain of trips to L2 is waited for: no barrier of the CTA, which the other heads and the next segment's pages need not
 * wait for.  us a layer with barriers and one CTA for all heads / so: FP16 4 096 tokens 10.3 / 9.7, 32 768 27.7 / 26.8; INT4 16 000 14.0 / 13.4,
 * 32 768 17.8 / 17.1; INT8 32 768 19.0 / 18.9. */
__device__ __forceinline__ bool fold_last(float *rec0, int piece, int np, unsigned *arrivals, uint8_t *zone, unsigned stride, int slots, int lane, float &M, float &L, float (&acc)[4]) {
    store_record(rec0 + (size_t)piece * 8 * HY3A_REC_FLOATS, lane, M, L, acc);
    __syncwarp();      /* the record is complete in the warp; the release publishes it */
    unsigned old = 0;
    if (lane == 0) asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(arrivals) : "memory");
    if (__shfl_sync(0xffffffffu, old, 0) != (unsigned)(np - 1)) return false;
    __syncwarp();      /* lane 0 has acquired the other pieces' records; a shuffle orders no memory, and every lane reads them */
    if (lane == 0) *arrivals = 0u;      /* for the next launch */
    fold_records(rec0, np, zone, stride, slots, lane, M, L, acc);
    return true;
}
/* Clusters: the CL CTAs of a (row, KV head) segment take an equal share of its pages each and meet in shared memory.  Rank r finishes
 * heads [r 8 / CL, (r + 1) 8 / CL): every CTA stores its records of these heads into r's landing zone with st.async, whose bytes
 * r's mbarrier counts, so that there is no record in memory, no counter and no fetch. */
constexpr int kCluRec = (HY3A_D + 4) * 4;               /* {acc[128], m, l, -, -} */
constexpr int kCluBytes = 8 * kCluRec;                  /* a CTA's zone: [CL sources][8 / CL heads] */
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_addr(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async16(unsigned addr, float a, float b, float c, float d, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
/* thread (head h of a warp, 4 dims): this CTA's piece to the CTA that finishes the head */
template <int CL>
__device__ __forceinline__ void cluster_send(unsigned zone, unsigned bar, int rank, int h, int lane, float M, float L, const float (&acc)[4]) {
    constexpr int HPC = 8 / CL;
    const unsigned to = (unsigned)h / HPC, rec = zone + (unsigned)((rank * HPC + h % HPC) * kCluRec), rb = cluster_addr(bar, to);
    st_async16(cluster_addr(rec + 16u * (unsigned)lane, to), acc[0], acc[1], acc[2], acc[3], rb);
    if (lane == 0) st_async16(cluster_addr(rec + 512u, to), M, L, 0.f, 0.f, rb);
}
/* warp w < 8 / CL folds its head's pieces in their order (rule of hy3_gpu.cu:233-247); a piece without keys has l = 0 */
template <int CL>
__device__ __forceinline__ void cluster_fold(const uint8_t *zone, int w, int lane, float &M, float &L, float (&acc)[4]) {
    M = -INFINITY; L = 0.f; acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
    for (int c = 0; c < CL; c++) {
        const uint8_t *rec = zone + (c * (8 / CL) + w) * kCluRec;
        const float2 ml = *reinterpret_cast<const float2 *>(rec + 512);
        const float4 v = *reinterpret_cast<const float4 *>(rec + 16 * lane);
        if (ml.y == 0.f) continue;
        const float nm = fmaxf(M, ml.x), os = ex2(M - nm), rs = ex2(ml.x - nm);
        L = L * os + ml.y * rs;
        acc[0] = acc[0] * os + v.x * rs; acc[1] = acc[1] * os + v.y * rs; acc[2] = acc[2] * os + v.z * rs; acc[3] = acc[3] * os + v.w * rs;
        M = nm;
    }
}
/* head hq (of the context's heads) of a row: final output, or the caller's record */
__device__ __forceinline__ void cluster_write(const hy3a_decode_args &a, int kv_heads, int kv_head_begin, int row, int hq, int lane, float M, float L, const float (&acc)[4]) {
    const int d4 = 4 * lane;
    if (a.user_partials) {
        float *rec = a.user_partials + ((size_t)row * kv_heads * 8 + hq) * HY3A_PARTIAL_FLOATS;
        if (lane == 0) { rec[0] = M * kLn2; rec[1] = L; }
        rec[2 + d4] = acc[0]; rec[3 + d4] = acc[1]; rec[4 + d4] = acc[2]; rec[5 + d4] = acc[3];
    } else {
        const float inv = inv_sum(L);
        *reinterpret_cast<float4 *>(a.out + (size_t)row * a.out_stride + (size_t)(kv_head_begin * 8 + hq) * HY3A_D + d4) = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
    }
}
__device__ __forceinline__ void imma16832(int c[4], const uint4 &a, unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float2 unpack_h2(unsigned v) {
    __half2 h = *reinterpret_cast<__half2 *>(&v);
    return __half22float2(h);
}
/* Sequence sharding: lines of one head's record in a gather buffer: line 0 = {m, l}, line 1 + j = acc[2j], acc[2j+1]. */
constexpr int kShardLines = HY3A_PARTIAL_FLOATS / 2;   /* 65 */
__device__ __forceinline__ void shard_store_line(uint4 *p, float x, float y, unsigned flag) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(p), "r"(__float_as_uint(x)), "r"(flag), "r"(__float_as_uint(y)) : "memory");
}
__device__ __forceinline__ uint4 shard_load_line(const uint4 *p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

/* Sequence sharding, receiving side; run by the first 8 warps of one CTA for one (row, KV head) segment: thread
 * (h, d4) polls the three lines it needs of every other rank's record (all ranks' loads are issued before any is
 * checked, so the usual cost is one L2 round trip), takes its own rank's values from registers, folds in rank
 * order with the rule of hy3_gpu.cu:233-247 (same order on every rank: identical bits) and writes the normalised
 * output.  The wait is bounded in polls and in time (about a second); when it runs out a code goes into the
 * error word, later waits return at once and the kernel runs to its end.                                      */
struct shard_fold_args {
    const uint4 *rec0;     /* line 0 of rank 0's record of this thread's (segment, head) */
    size_t rank_stride;    /* lines between consecutive ranks' records */
    unsigned *err;
    float *out;            /* this thread's 4 output floats */
    const uint4 *stage;    /* shared memory, [kShardBatch][8 heads][65] lines: landing zone of the polls */
    int n_ranks, my_rank, line_a, h, lane;
    unsigned flag;
    float own_m, own_l, own_acc[4];
};

/* Run by the first 8 warps (all lanes) for one segment.  Polling costs no registers: every thread copies the three
 * lines it needs of each pending rank's record into shared memory with 16-byte asynchronous copies (L2 -> shared),
 * all ranks of a batch in flight at once, and checks the flags there; the usual cost is one L2 round trip per batch.
 * Own rank: values from registers.  Fold in rank order (hy3_gpu.cu:233-247): identical bits on every rank.
 * The wait is bounded in polls and in time (about a second); when it runs out a code goes into the error word, the
 * missing records count as empty, later waits return at once and the kernel runs to its end.                       */
template <int kShardBatch>   /* ranks polled at once: kShardBatch x 8 320 bytes of landing zone */
__device__ __forceinline__ void shard_fold(const shard_fold_args &a) {
    float ms = -INFINITY, ss = 0.f, ov[4] = {0.f, 0.f, 0.f, 0.f};
    const unsigned stage_u32 = smem_u32(a.stage);
#pragma unroll 1
    for (int base = 0; base < a.n_ranks; base += kShardBatch) {
        const int cnt = min(kShardBatch, a.n_ranks - base);
        unsigned pending = 0u;   /* bit j: rank base + j not complete yet (per thread) */
        for (int j = 0; j < cnt; j++) if (base + j != a.my_rank) pending |= 1u << j;
        unsigned long long t0 = 0;
        bool gave_up = false;
#pragma unroll 1
        for (unsigned i = 0; __any_sync(0xffffffffu, pending != 0u); i++) {
#pragma unroll 1
            for (int j = 0; j < cnt; j++)
                if (pending & (1u << j)) {
                    const uint4 *rec = a.rec0 + (size_t)(base + j) * a.rank_stride;
                    const unsigned dst = stage_u32 + (unsigned)((j * 8 + a.h) * kShardLines) * 16u;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (unsigned)a.line_a), "l"(rec + a.line_a) : "memory");
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (unsigned)(a.line_a + 1)), "l"(rec + a.line_a + 1) : "memory");
                    if (a.lane == 0) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(rec) : "memory");
                }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
#pragma unroll 1
            for (int j = 0; j < cnt; j++)
                if (pending & (1u << j)) {
                    const uint4 *st = a.stage + (j * 8 + a.h) * kShardLines;
                    const uint4 l0 = st[0];
                    if (l0.y != a.flag || l0.w != a.flag) continue;
                    if (__uint_as_float(l0.z) != 0.f) {
                        const uint4 la = st[a.line_a], lb = st[a.line_a + 1];
                        if (la.y != a.flag || la.w != a.flag || lb.y != a.flag || lb.w != a.flag) continue;
                    }
                    pending &= ~(1u << j);
                }
            __syncwarp();   /* lane 0 may overwrite line 0 in the next round */
            if ((i & 15u) == 15u) {
                bool stop = *reinterpret_cast<volatile unsigned *>(a.err) != 0u;
                if (!stop && pending) {
                    unsigned long long t1;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
                    if (t0 == 0) t0 = t1;
                    if (t1 - t0 > 1000000000ull || i > (1u << 24)) {
                        if (atomicCAS(a.err, 0u, 3u) == 0u) a.err[1] = 41u;
                        stop = true;
                    }
                }
                if (__any_sync(0xffffffffu, stop && pending)) { gave_up = true; break; }
                __nanosleep(32);
            }
        }
#pragma unroll 1
        for (int j = 0; j < cnt; j++) {
            float pm, pl, pv[4];
            if (base + j == a.my_rank) {
                pm = a.own_m; pl = a.own_l; pv[0] = a.own_acc[0]; pv[1] = a.own_acc[1]; pv[2] = a.own_acc[2]; pv[3] = a.own_acc[3];
                if (pl == 0.f) continue;
            } else {
                if (gave_up && (pending & (1u << j))) continue;
                const uint4 *st = a.stage + (j * 8 + a.h) * kShardLines;
                const uint4 l0 = st[0];
                pm = __uint_as_float(l0.x); pl = __uint_as_float(l0.z);
                if (pl == 0.f) continue;
                const uint4 la = st[a.line_a], lb = st[a.line_a + 1];
                pv[0] = __uint_as_float(la.x); pv[1] = __uint_as_float(la.z); pv[2] = __uint_as_float(lb.x); pv[3] = __uint_as_float(lb.z);
            }
            const float nm = fmaxf(ms, pm), os = __expf(ms - nm), rs = __expf(pm - nm);
            ss = ss * os + pl * rs;
            ov[0] = ov[0] * os + pv[0] * rs; ov[1] = ov[1] * os + pv[1] * rs; ov[2] = ov[2] * os + pv[2] * rs; ov[3] = ov[3] * os + pv[3] * rs;
            ms = nm;
        }
        __syncwarp();   /* the landing zone is reused by the next batch of ranks */
    }
    const float inv = inv_sum(ss);
    *reinterpret_cast<float4 *>(a.out) = make_float4(ov[0] * inv, ov[1] * inv, ov[2] * inv, ov[3] * inv);
}

} /* namespace */
#endif
