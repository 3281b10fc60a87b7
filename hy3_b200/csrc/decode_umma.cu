/*
 * decode_umma.cu -- split-KV GQA decode attention for INT8 caches: scores on mma.sync, P.V on tcgen05 / TMEM.
 *
 * Same job, schedule, records and merge as decode.cu (replaces attention_split_kv_kernel + attention_reduce_kernel,
 * hy3_gpu.cu:183-247); what changes is who multiplies by V.  In decode.cu every warp converts the V codes of its 16
 * tokens to fp16 and keeps a 16 x 128 output tile in registers: 64 conversions + 16 MMAs per 16 tokens, 64 accumulator
 * registers per lane, a shared-memory fold of all warps at the end -- the CUDA cores, not HBM, set the pace of a page.
 * Here the V area of a page is stored TRANSPOSED (row = head dim, 128 token bytes, 128-byte swizzle: layout.h), so the
 * copy that lands in shared memory IS a tensor-core operand, and the head dims, not the heads, are the M dimension:
 *
 *   S[16 x 32]        = Qd . K^T         mma.sync m16n8k32.s8 on the stored codes, as in decode.cu: rows 0-7 = high int8
 *                                        digit of the 8 queries, rows 8-15 = low digit (q ~ sq (hi + lo / 254))
 *   O^T[128 dim x 16] = V^T . Pd^T       tcgen05.mma kind::i8, M = 128, N = 16, K = 32 tokens: the 16 columns are the
 *                                        8 heads x {high, low} int8 digit of w = p * vscale(token) / wb, wb = the largest
 *                                        V scale of the 32 tokens; products and sums are exact integers
 *
 * Roles (19 warps, coupled by mbarriers only):
 *   warps 0-7   accumulators: thread = (head dim = TMEM lane, 4 of the 8 heads).  Per page they read the four groups' integer
 *               results from TMEM (tcgen05.ld) and add them, scaled, to 4 fp32 registers.  Before the stream starts they
 *               also run the fused append (one warp per new row).
 *   warp 8      page producer (one lane): bulk copies (cp.async.bulk + mbarrier transaction counts, evict-first in L2) into a
 *               ring of pages; the first ring fill runs before the preceding kernel is known to be complete (pages below
 *               the newest slot are immutable).  It plans for the CTA first (decode_common.cuh).
 *   warp 9      MMA issuer (one lane): when the four groups' digits of a page are in shared memory it issues the four
 *               tcgen05.mma back to back, one tcgen05.commit for the accumulators and one that frees the ring stage.  It
 *               does nothing else: scalar code between two MMAs of a lane costs more than the MMA.
 *   warp 10     bookkeeper (lane = (group, head)): the online-softmax bookkeeping of the page -- running max, rescale factor,
 *               denominator, the factor of every (group, head) -- once for all accumulators, while the tensor core works.
 *   warps 11-18 score warps: a warp takes a 32-token group: 16 integer MMAs, scales, the group's own max (2 shuffles),
 *               8 exponentials per lane, digits, 8 two-byte stores into the P^T tile, {max, sum, wb} for the bookkeeper.
 *               No output accumulators, no conversion of V: about 250 instructions per 32 tokens instead of 860.
 *               The same warps run the query set-up and the epilogue (records, merge, exchange).
 *   Every waiter of an mbarrier waits for every phase of it, in order (a wait only knows a phase's parity).
 *
 * Every wait is bounded; a wait that runs out raises a CTA-wide abort flag and records a code in the context's error
 * word, every later wait returns at once, all roles keep their control flow to the end and TMEM is released.
 *
 * Roofline: HBM; algorithmic bytes per (token, KV head) = 260.
 */
#include <cuda_fp16.h>
#include <math.h>
#include <stddef.h>
#include <string.h>

#include "ctx.h"
#include "decode_common.cuh"
#include "rowops.cuh"

namespace {

constexpr int kAccWarps = 8, kProdWarp = 8, kIssWarp = 9, kBkWarp = 10, kQkWarp0 = 11, kQkWarps = 8;
constexpr int kAccThreads = kAccWarps * 32;
constexpr int kQkThreads = kQkWarps * 32;
constexpr int kUThreads = (kQkWarp0 + kQkWarps) * 32;
constexpr int kSlots = 8;                        /* pages in flight between the score warps and the accumulators (8 x 64 TMEM columns) */
constexpr int kStages = HY3A_UMMA_STAGES;        /* pages in the ring */
constexpr int kStageBytes = 33792;               /* an INT8 page (33 280 B) rounded up to 1 KB: every V^T tile 1024-byte aligned */
constexpr int kVtOff = 16384, kKsOff = 32768, kVsOff = 33024;
constexpr int kRecFloats = HY3A_REC_FLOATS;
constexpr int kShardBatchU = 1;                  /* ranks polled at once by the sharded epilogue when the ring is not idle (8 320 B of landing zone each) */
constexpr float kDigits = 32258.f;               /* 127 * 254: the largest two-digit value */

struct u_misc {
    unsigned long long rfull[8], rempty[8], pfull[kSlots], ofull[kSlots], bk[kSlots], sfree[kSlots], clu;
    unsigned tmem;
    int abort_flag, flag, app_ready;         /* app_ready: the fused appends of this CTA are in HBM */
    cta_plan plan;
    float qf[8];
    float ml[8][2];                              /* {M, L} of the segment piece the accumulators just finished */
    float meta_m[kSlots][4][8], meta_l[kSlots][4][8], meta_wb[kSlots][4];
    /* read as float4 by the accumulators */
    __align__(16) float fa[kSlots][32];
    __align__(16) float rr[kSlots][8];
};
static_assert(offsetof(u_misc, fa) % 16 == 0 && offsetof(u_misc, rr) % 16 == 0 && offsetof(u_misc, rfull) % 8 == 0, "alignment of the vector-loaded members");
/* shared-memory map, bytes from a 1024-byte aligned base.  The P^T tiles double as the hand-over area of a finished piece
 * and as the landing zone of the epilogue: all three uses follow one another (the accumulators hand a piece over when every
 * MMA of it is done; the score warps copy it into registers, run the epilogue, and only then start the next piece's digits). */
constexpr int kOffPt = 0;                            /* kSlots x [16 rows][128 B]: P digits, transposed, 128-byte swizzle */
constexpr int kOffAcc = 0;                           /* [8 heads][128 dims] fp32: the finished piece, handed to the epilogue */
constexpr int kOffLand = 0;                          /* landing zone of records / exchange lines when the page ring is not idle */
constexpr int kLandBytes = kSlots * 2048;
constexpr int kOffQ = kOffPt + kSlots * 2048;        /* Q fragments [4 k-steps][32 lanes] x 16 B */
constexpr int kOffMisc = kOffQ + 2048;
constexpr int kOffClu = kOffMisc + ((sizeof(u_misc) + 127) / 128) * 128;      /* a cluster's landing zone, at the cost of two pages of the ring */
constexpr int kStagesClu = kStages - 2;
template <int CL> constexpr int kOffPrefix = kOffClu + (CL ? (kCluBytes + 127) / 128 * 128 : 0);
static_assert(kShardBatchU * 8 * (HY3A_PARTIAL_FLOATS / 2) * 16 <= kLandBytes, "landing zone too small for the exchange");
static_assert(8 * HY3A_D * 4 == 4096 && kLandBytes >= 2 * 4096, "the hand-over area, and behind it places for every head's records");
/* score warps 0-3 take the even pages and 4-7 the odd ones: with an even ring each waits for every phase of its stages */
static_assert(kStages >= 4 && kStages <= 8 && kStages % 2 == 0 && kStagesClu % 2 == 0 && kSlots % 2 == 0, "ring depth");

/* descriptors: K-major, 128-byte swizzle, 8-row groups 1024 B apart (version 1, layout type 2) */
__device__ __forceinline__ unsigned long long make_desc(unsigned saddr) {
    return (unsigned long long)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
/* instruction descriptor, kind::i8: D = s32 (2 at bit 4), A = B = signed 8-bit (1 at bits 7 and 10), both K-major,
 * N = 16 (>> 3 at bit 17), M = 128 (>> 4 at bit 24) */
constexpr unsigned kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
__device__ __forceinline__ void umma_i8(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, 0, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(kIdescI8) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16_nowait(unsigned taddr, int *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(unsigned taddr, int *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void qk_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kQkThreads) : "memory"); }
/* hand-over of a finished piece: the accumulators arrive, the score warps wait */
__device__ __forceinline__ void epi_arrive() { asm volatile("bar.arrive 3, %0;" ::"n"(kAccThreads + kQkThreads) : "memory"); }
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 3, %0;" ::"n"(kAccThreads + kQkThreads) : "memory"); }
__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b, unsigned sel) {
    unsigned r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ void sts16(unsigned addr, unsigned v) { asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((unsigned short)v) : "memory"); }
#define UBAR(field) smem_u32(&(field))
/* every wait of this kernel: blocking try_wait, bounded, a no-op once the CTA has given up */
#define UWAIT(field, parity, where) mbar_wait_blocking(UBAR(field), (parity), &mi.abort_flag, a.err, (where))

/* One 32-token group of one score warp: S = Qd . K^T, the group's max / sum, digits of w into the P^T tile.
 * FULL: all 32 tokens are valid.  spage: shared address of the page; pt: shared address of the slot's P^T tile. */
template <bool FULL>
__device__ __forceinline__ void score_group(u_misc &mi, int slot, unsigned sq, float qf, unsigned spage, unsigned pt, int k_off0, int k_off1, int gi, int g, int tig, int lane, int valid) {
    unsigned ksw[4], vsw[4];
#pragma unroll
    for (int nb = 0; nb < 4; nb++) {
        ksw[nb] = lds4(spage + kKsOff + gi * 64 + nb * 16 + 4 * tig);
        vsw[nb] = lds4(spage + kVsOff + gi * 64 + nb * 16 + 4 * tig);
    }
    int c[4][4];
#pragma unroll
    for (int nb = 0; nb < 4; nb++) c[nb][0] = c[nb][1] = c[nb][2] = c[nb][3] = 0;
    /* two 8-token blocks at a time: two independent chains of four dependent MMAs, 16 registers of K codes in flight */
#pragma unroll
    for (int half = 0; half < 2; half++) {
        uint4 kr[2][2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            kr[j][0] = lds16(spage + gi * 4096 + (2 * half + j) * 1024 + k_off0);
            kr[j][1] = lds16(spage + gi * 4096 + (2 * half + j) * 1024 + k_off1);
        }
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const uint4 qa = lds16(sq + kk * 512);
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const unsigned b0 = kk == 0 ? kr[j][0].x : (kk == 1 ? kr[j][0].y : (kk == 2 ? kr[j][0].z : kr[j][0].w));
                const unsigned b1 = kk == 0 ? kr[j][1].x : (kk == 1 ? kr[j][1].y : (kk == 2 ? kr[j][1].z : kr[j][1].w));
                imma16832(c[2 * half + j], qa, b0, b1);
            }
        }
    }
    /* logits (base 2) of head g for tokens 32 gi + 8 nb + 2 tig + e, and the V scales of those tokens */
    float s[4][2], vs[4][2];
#pragma unroll
    for (int nb = 0; nb < 4; nb++) {
        const float2 kf = unpack_h2(ksw[nb]), vf = unpack_h2(vsw[nb]);
        const float r0 = (float)(c[nb][0] * 254 + c[nb][2]) * qf, r1 = (float)(c[nb][1] * 254 + c[nb][3]) * qf;
        const int t0 = 32 * gi + 8 * nb + 2 * tig;
        s[nb][0] = (FULL || t0 < valid) ? r0 * kf.x : -INFINITY;
        s[nb][1] = (FULL || t0 + 1 < valid) ? r1 * kf.y : -INFINITY;
        vs[nb][0] = (FULL || t0 < valid) ? vf.x : 0.f;
        vs[nb][1] = (FULL || t0 + 1 < valid) ? vf.y : 0.f;
    }
    float mx = fmaxf(fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1])), fmaxf(fmaxf(s[2][0], s[2][1]), fmaxf(s[3][0], s[3][1])));
    float wb = fmaxf(fmaxf(fmaxf(vs[0][0], vs[0][1]), fmaxf(vs[1][0], vs[1][1])), fmaxf(fmaxf(vs[2][0], vs[2][1]), fmaxf(vs[3][0], vs[3][1])));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    wb = fmaxf(wb, __shfl_xor_sync(0xffffffffu, wb, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    wb = fmaxf(wb, __shfl_xor_sync(0xffffffffu, wb, 2));
    const float msafe = mx == -INFINITY ? 0.f : mx;
    const float inv = wb > 0.f ? __fdividef(kDigits, wb) : 0.f;
    /* two int8 digits per w through the 1.5 * 2^23 trick: the low mantissa byte of (x + magic) is round(x) as int8 */
    const float magic = 12582912.f;
    float lsum = 0.f;
    const unsigned pt_row = pt + (unsigned)g * 128u;
#pragma unroll
    for (int nb = 0; nb < 4; nb++) {
        unsigned hb[2], lb[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float p = ex2(s[nb][e] - msafe);               /* -inf -> 0 */
            lsum += p;
            const float d = p * vs[nb][e] * inv;                 /* 0 .. 32258 */
            const float t = fmaf(d, 1.f / 254.f, magic);
            const float hf = t - magic;
            const float u = fmaf(hf, -254.f, d + magic);
            hb[e] = __float_as_uint(t);
            lb[e] = __float_as_uint(u);
        }
        /* byte column 32 gi + 8 nb + 2 tig of rows g (high digit) and 8 + g (low digit); 16-byte chunk c of a row sits at
         * chunk c ^ (row & 7) = c ^ g */
        const unsigned col = (unsigned)(((2 * gi + (nb >> 1)) ^ g) << 4) + (unsigned)(8 * (nb & 1) + 2 * tig);
        sts16(pt_row + col, prmt(hb[0], hb[1], 0x0040u));
        sts16(pt_row + 1024u + col, prmt(lb[0], lb[1], 0x0040u));
    }
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
    lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
    if (tig == 0) { mi.meta_m[slot][gi][g] = mx; mi.meta_l[slot][gi][g] = lsum; }
    if (lane == 0) mi.meta_wb[slot][gi] = wb;
    /* the digits were written through the generic proxy; the tensor core reads through the async proxy */
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_arrive(UBAR(mi.pfull[slot]));
}

/* CL: 0 = any grid, 2 / 4 / 8 = a cluster of CL CTAs per (row, KV head) */
template <bool SHARD, int CL = 0>
__global__ void __launch_bounds__(kUThreads, 1) hy3a_decode_umma_kernel(hy3a_cache_view cache, hy3a_batch_view batch, decode_args a) {
    constexpr int kStages = CL ? kStagesClu : HY3A_UMMA_STAGES;
    extern __shared__ __align__(128) uint8_t s_raw[];
    uint8_t *s_dyn = s_raw + ((1024u - (smem_u32(s_raw) & 1023u)) & 1023u);   /* 1024-aligned in the shared window */
    const unsigned s_base = smem_u32(s_dyn);
    u_misc &mi = *reinterpret_cast<u_misc *>(s_dyn + kOffMisc);
    int *s_prefix = reinterpret_cast<int *>(s_dyn + kOffPrefix<CL>);
    const hy3a_geom geom = hy3a_make_geom(1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int n = batch.n, G = cache.kv_heads;
    const int cta = blockIdx.x;
    int *s_pos = s_prefix + n + 1;                                   /* RoPE positions of the rows */
    const unsigned ring_off = (unsigned)((kOffPrefix<CL> + a.prefix_bytes + 1023) & ~1023);
    const unsigned ring_base = s_base + ring_off;
    const int qw = warp - kQkWarp0, qtid = tid - kQkWarp0 * 32;      /* score-warp numbering (negative for the other roles) */
    const bool is_qk = warp >= kQkWarp0;

    if (a.wait_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    /* ---- prologue: everything here reads only what the host wrote.  The loads are issued together. */
    const int rl_d0 = (lane >> 4) * 64 + (lane & 15) * 4;
    float4 pre_w = make_float4(1.f, 1.f, 1.f, 1.f), pre_f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.fused && is_qk && qw < 8) {
        pre_w = *reinterpret_cast<const float4 *>(a.norm_w + rl_d0);
        pre_f = hy3a_rowops::rope_freqs(a.rope, lane);
    }
    if (warp == kIssWarp) {
        /* TMEM: kSlots pages x 4 groups x 16 columns (allocated by every CTA up front: the allocation takes about a microsecond) */
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&mi.tmem)), "n"(kSlots * 64) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < n; i += kUThreads) {
        if (n > 32) s_prefix[i + 1] = pages_of_slot(batch.slot[i]);
        s_pos[i] = batch.pos[i];
    }
    if (n > 32) __syncthreads();
    const bool is_producer = warp == kProdWarp;
    lane_rows rows = {-1, 0};
    if (is_producer) {
        /* the planning warp sets the barriers up while its rows' slots are on the way */
        rows = load_rows(batch, n, lane);
        if (lane == 0) {
            mi.abort_flag = 0;
            mi.app_ready = 0;
            for (int i = 0; i < kStages; i++) { mbar_init(UBAR(mi.rfull[i]), 1); mbar_init(UBAR(mi.rempty[i]), 1); }
            for (int i = 0; i < kSlots; i++) {
                mbar_init(UBAR(mi.pfull[i]), 128);      /* the four score warps of a page, every lane */
                mbar_init(UBAR(mi.ofull[i]), 1);
                mbar_init(UBAR(mi.bk[i]), 1);
                mbar_init(UBAR(mi.sfree[i]), kAccWarps);
            }
            if (CL) mbar_init(UBAR(mi.clu), 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            if (CL) mbar_expect_tx(UBAR(mi.clu), kCluBytes);
        }
        plan<1, CL>(&mi.plan, s_prefix, rows.slot, n, G, gridDim.x, cta, lane);
    }
    if (CL) cluster_arrive();      /* every CTA of the cluster has set its barrier up; cluster_wait below */
    fence_before();
    /* the others need the plan; the copies need no one.  A barrier of its own: the producer may be at the CTA's last one before the others are here */
    if (is_producer) asm volatile("bar.arrive 4, %0;" ::"n"(kUThreads) : "memory");
    else asm volatile("bar.sync 4, %0;" ::"n"(kUThreads) : "memory");
    fence_after();
    const long long U = (long long)G * s_prefix[n], u_begin = mi.plan.u0, u_end = mi.plan.u1;
    const bool aligned = mi.plan.aligned, idle = u_begin == u_end;
    const int C = (long long)gridDim.x < U ? (int)gridDim.x : (int)U;
    const int al_first = mi.plan.first, al_pieces = mi.plan.pieces;
    if (idle && !SHARD && !CL) {
        /* No pages: give the tensor memory back and leave -- behind the rows without keys, which belong to idle CTAs as well, and, where
         * no CTA has pages, behind the wait of CTA 0, so that such a launch too ends after the one before it (hy3a_batch_kernel relies
         * on that).  (Sharded: idle CTAs may still own the fold of rows without local keys.) */
        if (cta < n) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
        for (int i = cta; i < n; i += gridDim.x)
            if (s_prefix[i + 1] == s_prefix[i]) HY3A_EMPTY_ROW(i, tid, kUThreads);
        fence_before();
        __syncthreads();
        if (warp == kIssWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(mi.tmem), "n"(kSlots * 64) : "memory");
        return;
    }
    segment sg0;                                                    /* the CTA's first piece */
    sg0.row = 0; sg0.hl = 0;
    if (!idle && !is_producer) sg0 = locate(s_prefix, batch, n, G, u_begin, u_end);

    /* fused step: cos / sin of the first segment's row (positions are in shared memory, the table in registers) */
    float pre_c[4] = {1.f, 1.f, 1.f, 1.f}, pre_s[4] = {0.f, 0.f, 0.f, 0.f};
    int pre_row = -1;
    auto rope_of_row = [&](int row) {
        hy3a_rowops::rope_coeffs(pre_c, pre_s, a.rope, pre_f, s_pos[row]);
        pre_row = row;
    };
    if (a.fused && !idle && is_qk && qw < 8) rope_of_row(sg0.row);
    /* The step's inputs may still be on their way from the preceding kernel, so they are read after the wait below; asking
     * L2 for their lines now is harmless (L2 is the point of coherence) and saves a trip to HBM when they are old. */
    if (!idle) {
        const int row0 = sg0.row, hl0 = sg0.hl;
        const int hd0 = (cache.kv_head_begin + hl0) * 8;
        if (is_qk && qw < 8 && (lane & 7) == 0) {
            const float *qp = (a.fused ? a.q_in + (size_t)row0 * a.qi_stride : a.q + (size_t)row0 * a.q_stride) + (size_t)(hd0 + qw) * HY3A_D + (lane >> 3) * 32;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(qp));
        }
        if (warp == 0 && a.fused && a.k_in && lane < 8) {
            const float *kp = (lane < 4 ? a.k_in + (size_t)row0 * a.ki_stride : a.v_in + (size_t)row0 * a.vi_stride) + (size_t)(cache.kv_head_begin + hl0) * HY3A_D + (lane & 3) * 32;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(kp));
        }
    }
    if (CL && !is_producer) cluster_wait();
    const unsigned tmem = is_producer ? 0u : mi.tmem;      /* the producer has not waited for it */

    /* From here on the kernel touches memory that the preceding kernel in the stream may produce (queries, the newest KV
     * slot, scratch records): wait for it -- except the producer lane, which first starts the copies of pages that lie
     * wholly below the newest slot (append-only cache: immutable). */
    if (!is_producer) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    /* rows with no keys on this rank: zero output / empty partial (hy3_gpu.cu:197-199) */
    if (is_qk && !CL)
        for (int i = cta; i < n; i += gridDim.x) {
            if (s_prefix[i + 1] != s_prefix[i]) continue;
            if (SHARD) {
                for (int e = qtid; e < G * 8; e += kQkThreads) {
                    const unsigned flag = a.shard_round[i * G * 8 + e] + 1u;
                    for (int r = 0; r < a.n_dest; r++)
                        if (r != a.my_rank) shard_store_line(a.dest[r] + ((size_t)i * G * 8 + e) * kShardLines, -INFINITY, 0.f, flag);
                }
                continue;
            }
            HY3A_EMPTY_ROW(i, qtid, kQkThreads);
        }

    if (!idle && warp == kProdWarp) {
        /* ================= producer: one lane streams the CTA's pages into the ring (the warp finds the segments).  Nothing is asked of L2 beyond the
         * ring: the first copies of a launch are what HBM has to bring first, and a request for the next 24 pages at once took
         * its bandwidth from the CTAs that start late (32 768 tokens 20.1 us a layer with it, 18.8 for 6 pages, 17.6 without; one page at a
         * time, each behind its block-table entry, 17.5 against 17.6 with all entries held by the warp's lanes). */
        unsigned it = 0;
        bool waited = false;   /* griddepcontrol.wait executed yet? */
        bool app_seen = false; /* the CTA's fused appends are known to be complete */
        const unsigned long long pol = l2_evict_first_policy();
        if (!a.early_prefetch) { asm volatile("griddepcontrol.wait;" ::: "memory"); waited = true; }
        for (long long u = u_begin; u < u_end;) {
            const segment sg = locate(s_prefix, batch, rows, n, G, u, u_end);
            const int *bt = cache.block_table + (size_t)sg.seq * cache.max_blocks_per_seq;
            if (lane == 0) {
                const uint8_t *page0 = cache.pool + hy3a_page_index(cache, 0, a.layer, sg.hl) * (size_t)cache.page_bytes;
                const size_t block_bytes = (hy3a_page_index(cache, 1, a.layer, sg.hl) - hy3a_page_index(cache, 0, a.layer, sg.hl)) * (size_t)cache.page_bytes;
                int block_next = bt[sg.p_begin];
                for (int p = sg.p_begin; p < sg.p_end; p++, it++) {
                    const uint8_t *page = page0 + block_next * block_bytes;
                    if (p + 1 < sg.p_end) block_next = bt[p + 1];   /* in flight while we wait for the stage */
                    const unsigned stage = it % (unsigned)kStages, phase = (it / (unsigned)kStages) & 1u;
                    /* before the preceding kernel is known to be complete only pages that lie wholly below the newest
                     * slot may be fetched, and only into stages that were never used */
                    if (!waited && (it >= (unsigned)kStages || (p + 1) * HY3A_PT > sg.len - 2)) { asm volatile("griddepcontrol.wait;" ::: "memory"); waited = true; }
                    const bool newest = a.fused && a.k_in && p == ((sg.len - 1) >> 7);
                    if (UWAIT(mi.rempty[stage], phase ^ 1u, 1u)) {      /* else gave up: issue nothing more */
                        if (newest && !app_seen) {
                            /* the page that holds a newest slot: the accumulator warps append those rows at the start of the
                             * kernel; their stores must be in HBM / L2 before the copy reads the page */
                            volatile int *ready = &mi.app_ready;
                            unsigned long long t0 = 0;
                            for (unsigned i = 0; !*ready && i < (1u << 24); i++) {
                                if ((i & 255u) == 255u) {
                                    unsigned long long t1;
                                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
                                    if (t0 == 0) t0 = t1;
                                    if (mi.abort_flag || (i >= (1u << 14) && t1 - t0 > 500000000ull)) { mi.abort_flag = 1; if (atomicCAS(a.err, 0u, 5u) == 0u) a.err[1] = 60u; break; }
                                }
                            }
                            app_seen = true;
                        }
                        mbar_expect_tx(UBAR(mi.rfull[stage]), (unsigned)geom.page_bytes);
                        bulk_g2s(ring_base + stage * (unsigned)kStageBytes, page, (unsigned)geom.page_bytes, UBAR(mi.rfull[stage]), pol);
                    }
                }
            }
            __syncwarp();
            u = sg.seg_u0 + sg.p_end;
        }
        if (lane == 0 && !waited) asm volatile("griddepcontrol.wait;" ::: "memory");
    } else if (!idle && warp == kIssWarp) {
        /* ================= MMA issuer: one lane; per page one wait, four MMAs back to back, one commit (the scalar code
         * between two tcgen05.mma of a thread costs more than the MMA itself, so this loop does nothing else) */
        if (lane == 0) {
            const unsigned n_pages = (unsigned)(u_end - u_begin);
            const unsigned long long dv0 = make_desc(ring_base + (unsigned)kVtOff), dp0 = make_desc(s_base + kOffPt);
            for (unsigned it = 0; it < n_pages; it++) {
                const unsigned stage = it % (unsigned)kStages, slot = it % (unsigned)kSlots, sph = (it / (unsigned)kSlots) & 1u;
                const unsigned long long dv = dv0 + (unsigned long long)(stage * (unsigned)(kStageBytes >> 4)), dp = dp0 + (unsigned long long)(slot * (2048u >> 4));
                const unsigned d = tmem + slot * 64u;
                UWAIT(mi.pfull[slot], sph, 20u);
                fence_after();
                /* a group's 32 tokens are bytes 32 gi .. 32 gi + 31 of every row of both tiles: + 32 B on the descriptors */
                umma_i8(d, dv, dp);
                umma_i8(d + 16u, dv + 2ull, dp + 2ull);
                umma_i8(d + 32u, dv + 4ull, dp + 4ull);
                umma_i8(d + 48u, dv + 6ull, dp + 6ull);
                umma_commit(UBAR(mi.ofull[slot]));
                umma_commit(UBAR(mi.rempty[stage]));    /* K was consumed by the scores, V^T by these MMAs: the stage can be refilled */
            }
        }
    } else if (!idle && warp == kBkWarp) {
        /* ================= bookkeeper: lane = (group, head).  Per page the online-softmax bookkeeping -- running max, rescale
         * factor, denominator, the factor of every (group, head) -- once for all accumulators, while the tensor core works. */
        const int bk_gi = lane >> 3, bk_h = lane & 7;
        float Mh = -INFINITY, Lh = 0.f;                 /* running max / denominator of head bk_h (replicated over the 4 group lanes) */
        unsigned it = 0;
        for (long long u = u_begin; u < u_end;) {
            const segment sg = locate(s_prefix, batch, n, G, u, u_end);
            Mh = -INFINITY; Lh = 0.f;
            for (int p = sg.p_begin; p < sg.p_end; p++, it++) {
                const unsigned slot = it % (unsigned)kSlots, sph = (it / (unsigned)kSlots) & 1u;
                UWAIT(mi.pfull[slot], sph, 25u);
                const float m = mi.meta_m[slot][bk_gi][bk_h], l = mi.meta_l[slot][bk_gi][bk_h], wbv = mi.meta_wb[slot][bk_gi];
                float mx = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float Mn = fmaxf(Mh, mx);
                const float r = Mn == -INFINITY ? 1.f : ex2(Mh - Mn);     /* 0 when Mh = -inf */
                const float f = m == -INFINITY ? 0.f : ex2(m - Mn);
                float ls = l * f;
                ls += __shfl_xor_sync(0xffffffffu, ls, 8);
                ls += __shfl_xor_sync(0xffffffffu, ls, 16);
                Lh = Lh * r + ls;
                Mh = Mn;
                mi.fa[slot][lane] = f * wbv * (1.f / kDigits);
                if (bk_gi == 0) {
                    mi.rr[slot][bk_h] = r;
                    if (p + 1 == sg.p_end) { mi.ml[bk_h][0] = Mh; mi.ml[bk_h][1] = Lh; }   /* the piece is complete */
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(UBAR(mi.bk[slot]));
            }
            u = sg.seg_u0 + sg.p_end;
        }
    } else if (!idle && warp < kAccWarps) {
        /* ================= accumulators: thread = (head dim = TMEM lane, 4 of the 8 heads) */
        const unsigned lane_base = (unsigned)((warp & 3) * 32) << 16;
        const int hq0 = 4 * (warp >> 2), dim = (warp & 3) * 32 + lane;
        float acc[4];
        unsigned it = 0;
        if (a.fused && a.k_in) {
            /* ---- fused append, up front: the newest token of every segment whose last page lies in this CTA's range is
             * normalised, rotated, quantised and stored exactly as the append kernel does (hy3_gpu.cu:750-756), one warp
             * per row, while the score warps prepare the queries.  The page is copied into the ring afterwards (the
             * producer waits for app_ready), so the kernel attends over the new token from the same bytes later steps read. */
            int j = 0;
            for (long long u2 = u_begin; u2 < u_end;) {
                const segment sg = locate(s_prefix, batch, n, G, u2, u_end);
                const int last_page = (sg.len - 1) >> 7;
                if (last_page >= sg.p_begin && last_page < sg.p_end) {
                    if ((j & (kAccWarps - 1)) == warp) {
                        const int tok = (sg.len - 1) & 127, kvh = cache.kv_head_begin + sg.hl;
                        const int block = cache.block_table[(size_t)sg.seq * cache.max_blocks_per_seq + last_page];
                        uint8_t *gp = cache.pool + hy3a_page_index(cache, block, a.layer, sg.hl) * (size_t)cache.page_bytes;
                        float4 kv4 = *reinterpret_cast<const float4 *>(a.k_in + (size_t)sg.row * a.ki_stride + (size_t)kvh * HY3A_D + rl_d0);
                        const float4 vv4 = *reinterpret_cast<const float4 *>(a.v_in + (size_t)sg.row * a.vi_stride + (size_t)kvh * HY3A_D + rl_d0);
                        float y[4] = {kv4.x, kv4.y, kv4.z, kv4.w};
                        float kc[4], ks[4];
                        hy3a_rowops::rope_coeffs(kc, ks, a.rope, s_pos[sg.row], lane);
                        hy3a_rowops::norm_rope_apply(y, *reinterpret_cast<const float4 *>(a.norm_w + HY3A_D + rl_d0), a.eps, kc, ks, lane);
                        hy3a_rowops::store_row<1>(gp, geom, tok, false, y, rl_d0, lane);
                        y[0] = vv4.x; y[1] = vv4.y; y[2] = vv4.z; y[3] = vv4.w;
                        const unsigned sb = hy3a_rowops::store_row<1>(gp, geom, tok, true, y, rl_d0, lane);
                        if (lane == 0) atomicMax(cache.vs_max + a.layer * G + sg.hl, sb);
                    }
                    j++;
                }
                u2 = sg.seg_u0 + sg.p_end;
            }
            /* the rows were stored through the generic proxy, the bulk copy reads through the async proxy */
            asm volatile("fence.proxy.async.global;" ::: "memory");
            asm volatile("bar.sync 2, %0;" ::"n"(kAccThreads) : "memory");
            if (tid == 0) { __threadfence_block(); *reinterpret_cast<volatile int *>(&mi.app_ready) = 1; }
        }
        for (long long u = u_begin; u < u_end;) {
            const segment sg = locate(s_prefix, batch, n, G, u, u_end);
            acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
            for (int p = sg.p_begin; p < sg.p_end; p++, it++) {
                const unsigned slot = it % (unsigned)kSlots, sph = (it / (unsigned)kSlots) & 1u;
                UWAIT(mi.ofull[slot], sph, 30u);
                fence_after();
                int c[4][8];   /* [group][high digits of the 4 heads | low digits] */
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    tmem_ld4_nowait(tmem + lane_base + slot * 64u + q * 16u + hq0, &c[q][0]);
                    tmem_ld4_nowait(tmem + lane_base + slot * 64u + q * 16u + 8u + hq0, &c[q][4]);
                }
                UWAIT(mi.bk[slot], sph, 31u);
                const float4 rv = *reinterpret_cast<const float4 *>(&mi.rr[slot][hq0]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                acc[0] *= rv.x; acc[1] *= rv.y; acc[2] *= rv.z; acc[3] *= rv.w;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 fv = *reinterpret_cast<const float4 *>(&mi.fa[slot][8 * q + hq0]);
                    acc[0] = fmaf((float)(c[q][0] * 254 + c[q][4]), fv.x, acc[0]);
                    acc[1] = fmaf((float)(c[q][1] * 254 + c[q][5]), fv.y, acc[1]);
                    acc[2] = fmaf((float)(c[q][2] * 254 + c[q][6]), fv.z, acc[2]);
                    acc[3] = fmaf((float)(c[q][3] * 254 + c[q][7]), fv.w, acc[3]);
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(UBAR(mi.sfree[slot]));          /* TMEM slot, P^T tile, meta and factors of the slot are free */
            }
            /* hand the finished piece to the epilogue (score warps) */
            float *s_acc = reinterpret_cast<float *>(s_dyn + kOffAcc);
#pragma unroll
            for (int h = 0; h < 4; h++) s_acc[(hq0 + h) * HY3A_D + dim] = acc[h];
            epi_arrive();
            u = sg.seg_u0 + sg.p_end;
        }
    } else if (is_qk) {
        /* ================= score warps (+ query set-up, fused append, epilogue) */
        const int k_off0 = hy3a_k_chunk_off<1>(g, tig), k_off1 = hy3a_k_chunk_off<1>(g, tig + 4);
        const unsigned sq = s_base + kOffQ + 16u * (unsigned)lane;
        uint4 (*s_q)[32] = reinterpret_cast<uint4 (*)[32]>(s_dyn + kOffQ);
        unsigned it = 0;
        long long u = u_begin;
        while (u < u_end) {
            const segment sg = locate(s_prefix, batch, n, G, u, u_end);
            const int row = sg.row, hl = sg.hl, sidx = sg.sidx;
            const int head0 = (cache.kv_head_begin + hl) * 8;
            /* ---- Q digits of the segment's 8 heads as MMA A fragments, straight from the registers of the warp that prepared the row */
            if (qw < 8) {
                float x[4];
                if (a.fused) {
                    const float4 xv = *reinterpret_cast<const float4 *>(a.q_in + (size_t)row * a.qi_stride + (size_t)(head0 + qw) * HY3A_D + rl_d0);
                    x[0] = xv.x; x[1] = xv.y; x[2] = xv.z; x[3] = xv.w;
                    if (row != pre_row) rope_of_row(row);
                    hy3a_rowops::norm_rope_apply(x, pre_w, a.eps, pre_c, pre_s, lane);
                    if (a.q_out && sg.p_begin == 0)
                        *reinterpret_cast<float4 *>(a.q_out + (size_t)row * a.q_out_stride + (size_t)(head0 + qw) * HY3A_D + rl_d0) = make_float4(x[0], x[1], x[2], x[3]);
                } else {
                    const float4 xv = *reinterpret_cast<const float4 *>(a.q + (size_t)row * a.q_stride + (size_t)(head0 + qw) * HY3A_D + rl_d0);
                    x[0] = xv.x; x[1] = xv.y; x[2] = xv.z; x[3] = xv.w;
                }
                float m = fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3])));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                const float sqv = m > 0.f ? m * (1.f / 127.f) : 1.f, inv = 1.f / sqv;
                unsigned hw = 0, lw = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float hi = fminf(127.f, fmaxf(-127.f, rintf(x[j] * inv)));
                    const float lo = fminf(127.f, fmaxf(-127.f, rintf((x[j] - hi * sqv) * (254.f * inv))));
                    hw |= ((unsigned)(int)hi & 0xFFu) << (8 * j);
                    lw |= ((unsigned)(int)lo & 0xFFu) << (8 * j);
                }
                /* MMA k-step kk, k-slots 4tig..4tig+3 / 16+4tig..16+4tig+3 of thread-in-group tig carry head dims 16 tig + 4 kk + 0..3 /
                 * 64 + the same: exactly what a thread gets out of its own 16-byte loads of a K row.  The lane's four dims are one of these
                 * halves, kk = lane & 3, tig = (lane & 15) >> 2: words 2 (lane >> 4) (high digits, rows 0-7) and the one behind it (low
                 * digits, rows 8-15) of that fragment.  (Gathered from a staged copy: a second barrier and 16 byte loads; no
                 * difference beyond noise at 700 tokens, 7.45 and 7.39 us a layer.) */
                *reinterpret_cast<uint2 *>(reinterpret_cast<unsigned *>(&s_q[lane & 3][4 * qw + ((lane & 15) >> 2)]) + 2 * (lane >> 4)) = make_uint2(hw, lw);
                if (lane == 0) mi.qf[qw] = sqv * (1.f / 254.f) * 0.08838834764831845f * kLog2e;
            }
            qk_sync();
            const float qf = mi.qf[g];

            /* group X = 4 * (ring position of the page) + group-in-page; warp w takes X = w (mod kQkWarps) */
            const unsigned it_end = it + (unsigned)(sg.p_end - sg.p_begin);
            for (unsigned X = it * 4u + ((unsigned)qw + kQkWarps - (it * 4u) % kQkWarps) % kQkWarps; X < it_end * 4u; X += kQkWarps) {
                const unsigned pit = X >> 2;
                const int gi = (int)(X & 3u), p = sg.p_begin + (int)(pit - it);
                const int valid = min(HY3A_PT, sg.len - p * HY3A_PT);
                const unsigned stage = pit % (unsigned)kStages, rph = (pit / (unsigned)kStages) & 1u;
                const unsigned slot = pit % (unsigned)kSlots, sph = (pit / (unsigned)kSlots) & 1u;
                const unsigned spage = ring_base + stage * (unsigned)kStageBytes;
                UWAIT(mi.rfull[stage], rph, 2u);
                UWAIT(mi.sfree[slot], sph ^ 1u, 3u);        /* the accumulators are through with the page that used this slot before */
                const unsigned pt = s_base + kOffPt + slot * 2048u;
                if (32 * gi + 32 <= valid) score_group<true>(mi, (int)slot, sq, qf, spage, pt, k_off0, k_off1, gi, g, tig, lane, valid);
                else score_group<false>(mi, (int)slot, sq, qf, spage, pt, k_off0, k_off1, gi, g, tig, lane, valid);
            }
            it = it_end;

            /* ---- the piece of this CTA, from the accumulators: thread -> (head, 4 dims) */
            epi_sync();
            const int h = (qtid >> 5) & 7, d4 = (qtid & 31) * 4;
            float M = mi.ml[h][0], L = mi.ml[h][1], acc[4];
            {
                const float4 o4 = *reinterpret_cast<const float4 *>(s_dyn + kOffAcc + (h * HY3A_D + d4) * 4);
                acc[0] = o4.x; acc[1] = o4.y; acc[2] = o4.z; acc[3] = o4.w;
            }
            if (CL) {
                cluster_send<CL ? CL : 1>(s_base + kOffClu, UBAR(mi.clu), cta % (CL ? CL : 1), h, lane, M, L, acc);
                break;
            }
            if (SHARD) qk_sync();   /* everybody holds its share: the hand-over area is a landing zone below; else it is written again behind the next piece's queries */

            /* ---- how many CTAs share this segment? */
            const int c_first = aligned ? al_first : cta_of_unit(sg.seg_u0, U, C);
            const int npieces = aligned ? al_pieces : cta_of_unit(sg.seg_u1 - 1, U, C) - c_first + 1;
            const int rec_base = aligned ? 0 : sidx;   /* record index = CTA (+ segment when CTAs may hold several pieces) */
            const size_t head_q = (size_t)(cache.kv_head_begin + hl) * 8 + h; /* global query head */
            u = sg.seg_u0 + sg.p_end;

            int h_lo = 0, h_hi = 8;
            bool last = true;      /* this warp has its head's final record */
            float *const recs = a.scratch + ((size_t)(c_first + rec_base) * 8 + h) * kRecFloats;      /* of the segment's piece 0 */
            if (npieces > 1) {
                if (aligned && a.spread) {
                    /* CTA-aligned segments: the fold is spread over the first F pieces (see decode.cu) */
                    const int Fmax = a.spread, F = npieces >= Fmax ? Fmax : (npieces >= 4 && Fmax >= 4 ? 4 : (npieces >= 2 && Fmax >= 2 ? 2 : 1)), hpf = 8 / F, piece = cta - c_first;
                    store_record(recs + (size_t)piece * 8 * kRecFloats, lane, M, L, acc);
                    qk_sync();   /* the record is complete in CTA scope; the release publishes it */
                    if (qtid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counters + 8 * sidx) : "memory");
                    if (piece >= F) continue;   /* CTA-uniform */
                    if (qtid == 0) {
                        unsigned seen = 0;
                        unsigned long long t0 = 0;
                        bool ok = false;
                        for (unsigned i = 0; i < (1u << 24); i++) {
                            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.counters + 8 * sidx) : "memory");
                            if (seen >= (unsigned)npieces) { ok = true; break; }
                            if ((i & 255u) == 255u) {
                                unsigned long long t1;
                                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
                                if (t0 == 0) t0 = t1;
                                if (mi.abort_flag || (i >= (1u << 14) && t1 - t0 > 500000000ull)) break;
                            }
                        }
                        if (!ok) { mi.abort_flag = 1; if (atomicCAS(a.err, 0u, 4u) == 0u) { a.err[1] = 50u; a.err[2] = blockIdx.x; a.err[3] = seen; } }
                        mi.flag = ok;
                    }
                    qk_sync();
                    h_lo = piece * hpf; h_hi = h_lo + hpf;
                    const bool mine = h >= h_lo && h < h_hi;
                    M = -INFINITY; L = 0.f; acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                    if (mi.flag && mine) {
                        constexpr int kRing = kStages * kStageBytes;      /* idle: this CTA's pages are consumed */
                        const int slots = min(32, kRing / (hpf * 512));
                        fold_records(recs, npieces, s_dyn + ring_off + (h - h_lo) * slots * 512, 512u, slots, lane, M, L, acc);
                    }
                    qk_sync();   /* every landing zone is read (the sharded exchange lands its lines in the ring too) */
                    if (qtid == 0) {
                        unsigned *done = a.counters + 8 * a.n_counters + sidx;
                        const unsigned old = atomicAdd(done, 1u);
                        if (old == (unsigned)(F - 1)) { a.counters[8 * sidx] = 0u; *done = 0u; }
                    }
                } else {
                    /* The last CTA to arrive folds, nobody waits.  The records land in the page ring where it is idle (whole CTAs to a segment:
                     * this CTA's pages are consumed), else behind the hand-over area. */
                    constexpr int kRingSlots = kStages * kStageBytes / 4096 < 32 ? kStages * kStageBytes / 4096 : 32;
                    uint8_t *const zone = s_dyn + (aligned ? ring_off + h * (kRingSlots * 512) : kOffLand + 4096 + h * 512);
                    last = fold_last(recs, cta - c_first, npieces, a.counters + 8 * sidx + h, zone, aligned ? 512u : 4096u, aligned ? kRingSlots : kLandBytes / 4096 - 1, lane, M, L, acc);
                    if (SHARD) qk_sync();      /* the exchange lands its lines there too */
                }
            }
            const bool fin = last && h >= h_lo && h < h_hi;   /* this thread finishes its (head, 4 dims) of the segment */
            if (SHARD) {
                /* sequence sharding: this rank's records go into every other rank's gather buffer as flagged lines, then
                 * the same threads collect the other ranks' lines and finish the segment (see decode.cu) */
                const int seg = row * G + hl;
                if (fin) {
                    const unsigned flag = a.shard_round[seg * 8 + h] + 1u;
                    const float m_nat = M * kLn2;
                    const size_t ro = ((size_t)seg * 8 + h) * kShardLines;
                    for (int r = 0; r < a.n_dest; r++) {
                        if (r == a.my_rank) continue;
                        uint4 *rec = a.dest[r] + ro;
                        if (d4 == 0) shard_store_line(rec, m_nat, L, flag);
                        shard_store_line(rec + 1 + (d4 >> 1), acc[0], acc[1], flag);
                        shard_store_line(rec + 2 + (d4 >> 1), acc[2], acc[3], flag);
                    }
                    shard_fold_args fa;
                    fa.rec0 = a.gathered + ro; fa.rank_stride = (size_t)n * G * 8 * kShardLines; fa.err = a.err;
                    fa.out = a.out + (size_t)row * a.out_stride + ((size_t)(cache.kv_head_begin + hl) * 8 + h) * HY3A_D + d4;
                    fa.n_ranks = a.n_dest; fa.my_rank = a.my_rank; fa.line_a = 1 + (d4 >> 1); fa.flag = flag; fa.h = h; fa.lane = lane;
                    fa.own_m = m_nat; fa.own_l = L; fa.own_acc[0] = acc[0]; fa.own_acc[1] = acc[1]; fa.own_acc[2] = acc[2]; fa.own_acc[3] = acc[3];
                    if (aligned) {
                        /* the page ring is idle by now and holds all 8 ranks' records at once: one round of polls */
                        fa.stage = reinterpret_cast<const uint4 *>(s_dyn + ring_off);
                        shard_fold<8>(fa);
                    } else {
                        fa.stage = reinterpret_cast<const uint4 *>(s_dyn + kOffLand);
                        shard_fold<kShardBatchU>(fa);
                    }
                    __syncwarp();
                    if (d4 == 0) a.shard_round[seg * 8 + h] = flag;
                }
                qk_sync();
                continue;
            }
            if (!fin) continue;
            if (a.user_partials) {
                float *rec = a.user_partials + ((size_t)row * G * 8 + (size_t)hl * 8 + h) * HY3A_PARTIAL_FLOATS;
                if (d4 == 0) { rec[0] = M * kLn2; rec[1] = L; } /* m in natural-log units like the reference record */
                rec[2 + d4] = acc[0]; rec[3 + d4] = acc[1]; rec[4 + d4] = acc[2]; rec[5 + d4] = acc[3];
            } else {
                const float inv = inv_sum(L);
                *reinterpret_cast<float4 *>(a.out + (size_t)row * a.out_stride + head_q * HY3A_D + d4) = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
            }
        }
        if (CL) {
            constexpr int C1 = CL ? CL : 1, HPC = 8 / C1;
            const int rank = cta % C1, seg = cta / C1, row = seg / G, hl = seg - row * G;
            const float none[4] = {0.f, 0.f, 0.f, 0.f};
            if (idle) cluster_send<C1>(s_base + kOffClu, UBAR(mi.clu), rank, qw, lane, -INFINITY, 0.f, none);
            if (qw < HPC) {
                UWAIT(mi.clu, 0u, 70u);
                float M, L, acc[4];
                cluster_fold<C1>(s_dyn + kOffClu, qw, lane, M, L, acc);
                cluster_write(a, G, cache.kv_head_begin, row, hl * 8 + rank * HPC + qw, lane, M, L, acc);
            }
        }
        /* sharded: rows without keys on this rank were announced at the top; the other ranks' records are folded here */
        if (SHARD)
            for (int i = cta; i < n; i += gridDim.x) {
                if (s_prefix[i + 1] != s_prefix[i]) continue;
                for (int hl = 0; hl < G; hl++) {
                    const int seg = i * G + hl;
                    if (qtid < 256) {
                        const int h = (qtid >> 5) & 7, d4 = (qtid & 31) * 4;
                        shard_fold_args fa;
                        fa.rec0 = a.gathered + ((size_t)seg * 8 + h) * kShardLines; fa.rank_stride = (size_t)n * G * 8 * kShardLines; fa.err = a.err;
                        fa.out = a.out + (size_t)i * a.out_stride + ((size_t)(cache.kv_head_begin + hl) * 8 + h) * HY3A_D + d4;
                        fa.n_ranks = a.n_dest; fa.my_rank = a.my_rank; fa.line_a = 1 + (d4 >> 1); fa.flag = a.shard_round[seg * 8 + h] + 1u;
                        fa.stage = reinterpret_cast<const uint4 *>(s_dyn + kOffLand); fa.h = h; fa.lane = lane;
                        fa.own_m = -INFINITY; fa.own_l = 0.f; fa.own_acc[0] = fa.own_acc[1] = fa.own_acc[2] = fa.own_acc[3] = 0.f;
                        shard_fold<kShardBatchU>(fa);
                        __syncwarp();
                        if (d4 == 0) a.shard_round[seg * 8 + h] = fa.flag;
                    }
                    qk_sync();
                }
            }
    }
    /* ---- common exit: every role arrives here, also after a wait ran out */
    {
        if (warp == kProdWarp && lane == 0 && mi.abort_flag) {
            /* copies already issued must land before the shared memory goes away */
            for (int st = 0; st < kStages; st++)
                for (unsigned ph = 0; ph < 2; ph++)
                    for (unsigned spin = 0; spin < (1u << 14) && !mbar_test(UBAR(mi.rfull[st]), ph); spin++) __nanosleep(64);
        }
        fence_before();
        __syncthreads();
        if (warp == kIssWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kSlots * 64) : "memory");
        /* a CTA's shared memory stays until every CTA of the cluster has sent (they have, unless a wait ran out) */
        if (CL) { __syncwarp(); if (is_producer) cluster_wait(); cluster_arrive(); cluster_wait(); }
    }
}

} /* namespace */

/* Bytes of dynamic shared memory for a batch capacity (prefix = page counts + positions of the rows). */
static size_t umma_prefix_bytes(int n) { return ((size_t)(2 * n + 2) * sizeof(int) + 127) & ~(size_t)127; }

/* the launch's shared memory: CL = 0 or any cluster */
template <int CL>
static size_t umma_smem(size_t prefix) { return 1024 + ((kOffPrefix<CL> + prefix + 1023) & ~(size_t)1023) + (size_t)(CL ? kStagesClu : kStages) * kStageBytes; }

int hy3a_decode_umma_fits(int max_batch) {
    return umma_smem<0>(umma_prefix_bytes(max_batch)) <= (size_t)kSmemMax;
}

static const void *umma_cluster_fn(int cl) {
    return cl == 2 ? (const void *)hy3a_decode_umma_kernel<false, 2> : cl == 4 ? (const void *)hy3a_decode_umma_kernel<false, 4> : (const void *)hy3a_decode_umma_kernel<false, 8>;
}

/* clusters of cl CTAs that fit on the device at once */
int hy3a_decode_umma_cluster_cap(hy3a_ctx *ctx, int cl) {
    return hy3a_cluster_cap(umma_cluster_fn(cl), cl, kUThreads, umma_smem<1>(umma_prefix_bytes(ctx->cfg.max_batch)));
}

cudaError_t hy3a_launch_decode_umma(hy3a_ctx *ctx, const hy3a_cache_view &cv, const hy3a_batch_view &bv, hy3a_decode_args &a) {
    const size_t prefix = umma_prefix_bytes(ctx->batch_n);
    a.prefix_bytes = (int)prefix;
    a.stages = kStages;
    const size_t smem = umma_smem<0>(prefix);
    const bool shard = a.n_dest > 0;
    if (a.cluster) {
        void *args[3] = {(void *)&cv, (void *)&bv, (void *)&a};
        return hy3a_launch_cluster(ctx, umma_cluster_fn(a.cluster), a.cluster, ctx->batch_n * ctx->cfg.kv_head_count, kUThreads, umma_smem<1>(prefix), args);
    }
    static bool attr_dev[64][2];   /* function attributes are per device */
    bool *attr_set = attr_dev[ctx->device & 63];
    if (!attr_set[shard ? 1 : 0]) {
        cudaError_t e = shard ? cudaFuncSetAttribute(hy3a_decode_umma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax)
                              : cudaFuncSetAttribute(hy3a_decode_umma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
        if (e != cudaSuccess) return e;
        attr_set[shard ? 1 : 0] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctx->decode_ctas); cfg.blockDim = dim3(kUThreads); cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = ctx->use_pdl ? 1 : 0;
    if (shard) return cudaLaunchKernelEx(&cfg, hy3a_decode_umma_kernel<true>, cv, bv, a);
    return cudaLaunchKernelEx(&cfg, hy3a_decode_umma_kernel<false>, cv, bv, a);
}
