/*
 * decode.cu -- split-KV GQA decode attention over the paged FP16 and INT4 caches (INT8 caches: decode_umma.cu),
 * the launch entry points of all three, and the merge kernel.
 *
 * Replaces attention_split_kv[_int4]_kernel + attention_reduce_kernel of the reference
 * (hy3_gpu.cu:183-247, :274-325).  The reference runs one warp per (query head, split),
 * so every KV byte is fetched once per query head of its group (8x) with 4-byte loads at
 * an 83 KB stride.  Here a warp processes 16 or 32 tokens of one KV head for ALL 8 query heads
 * of the group at once, on tensor cores, so each KV byte is read exactly once:
 *
 *   S[16 x 8]   = Q2[16 x 128] . K^T    rows 0-7 = the 8 heads, rows 8-15 = a residual of the
 *                                       same 8 queries (M=16 is the MMA minimum, so the second
 *                                       half of the tile buys near-fp32 queries for free).
 *                                       INT4 cache: integer MMA (m16n8k32.s8) directly on the
 *                                       stored nibbles -- Q is split into two int8 digits
 *                                       (q ~ sq*(hi + lo/254)), the products are exact, and no
 *                                       per-element conversion of K is needed at all.
 *                                       FP16 cache: m16n8k16.f16 with Q = fp16 + fp16 residual.
 *   O[16 x 128] += P[16 x 16] . V       m16n8k16.f16; INT4 codes become fp16 exactly with one lop3 +
 *                                       one fp16 subtract (or fma) per pair.
 *
 * The per-token scales are applied once per score (K) and once per probability (V), never
 * per element.  The contraction dimension of Q.K^T and the output dimension of P.V are
 * permuted so that every thread's MMA operands are exactly the 16-byte chunks it loads.
 *
 * Scheduling: unit = one 128-token page of one (batch row, KV head); units are laid out
 * row-major, head, page and cut into contiguous ranges, one per CTA, so one grid
 * serves every length (lengths come from device memory; nothing is baked into a captured
 * graph, cf. hy3_gpu.cu:774-789).  A producer warp streams the CTA's pages into a shared-
 * memory ring with bulk asynchronous copies (cp.async.bulk + mbarrier transaction counts);
 * the consumer warps take the 16- or 32-token granules of the pages round-robin.  The piece a CTA
 * computes for a (row, head) segment is folded in shared memory; if the segment spans
 * several CTAs each writes an {acc, m, l} record per query head and the LAST warp to arrive
 * (atomic counter per head) folds them -- the LSE-merge epilogue, no second launch.  Steps of few segments with few pages run as clusters
 * instead (cluster_size below).
 *
 * Roofline: HBM.  Algorithmic bytes per (token, KV head): 512 (FP16), 132 (INT4); per token and
 * layer x8.
 */
#include <cuda_fp16.h>
#include <math.h>
#include <string.h>

#include <algorithm>

#include "ctx.h"
#include "decode_common.cuh"
#include "rowops.cuh"

namespace {

constexpr int kWarps = HY3A_DECODE_WARPS;              /* consumer warps */
static_assert(kWarps >= 11, "eight warps for the queries and the reductions, one each for the new V row's scale and the new K and V rows");
constexpr int kThreads = kWarps * 32;
constexpr int kFixedO = kWarps * 8 * HY3A_D * 4;
constexpr int kFixedML = kWarps * 8 * 2 * 4;
constexpr int kFixedQ = 8 * 32 * 16;
constexpr int kFixedNew = 2 * HY3A_D * 4;
constexpr int kFixedHead = kFixedO + kFixedML + kFixedQ + kFixedNew;      /* every variant's; a cluster's landing zone follows */
/* bytes of shared memory in front of the page-count prefix (a multiple of 128), and of the mbarriers behind it: the page ring's empty[8]
 * and full[16], a cluster's meeting.  The ring starts on 128 bytes.  Nothing is padded further: a context's largest batch is what
 * the prefix has room for beside two pages (FP16: 12 543 rows). */
template <int CL> constexpr int kFixed = kFixedHead + (CL ? kCluBytes : 0);
template <int CL> constexpr int kBarBytes = CL ? 320 : 192;
constexpr int kBarClu = 192;
static_assert(kFixedML % 16 == 0 && kFixedHead % 16 == 0 && (kFixed<0> + kBarBytes<0>) % 128 == 0 && (kFixed<2> + kBarBytes<2>) % 128 == 0, "alignment of the shared-memory map");
static_assert(16 / 8 * 8 >= 8 + 3 && 16 / 7 * 7 >= 7 + 3 && 16 / 6 * 6 >= 6 + 3 && kWarps <= 12, "rounds of the full barriers: see the consumer loop");
constexpr bool kPSplit = true;                         /* carry the fp16 residual of P in MMA rows 8-15 */
constexpr int kRecFloats = HY3A_REC_FLOATS;             /* floats per head record in the merge scratch (130 used) */
constexpr int kShardBatch = 5;                          /* ranks polled at once by the sharded epilogue */
static_assert(kShardBatch * 8 * (HY3A_PARTIAL_FLOATS / 2) * 16 <= kFixedO, "landing zone of the rank records exceeds the staging area");
constexpr float kRescaleThreshold = 8.f;               /* lazy rescale: the running max may lag by 2^8 */

__device__ __forceinline__ uint4 ld16(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned ld4(const uint8_t *p) {
    unsigned v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned prmt(unsigned a, unsigned b, unsigned sel) {
    unsigned r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ unsigned hsub2(unsigned a, unsigned b) {
    unsigned r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ unsigned hfma2(unsigned a, unsigned b, unsigned c) {
    unsigned r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ unsigned pack_h2(float lo, float hi) {
    unsigned r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void mma16816(float c[4], const unsigned a[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

/* ---- exact integer-code -> fp16x2 conversions of V --------------------------------------
 * INT4 V codes are stored offset-binary (n+8; see append.cu), so that no sign fix-up is needed here. */
/* INT4: nibbles (i, i+4) become one fp16x2.  Low positions: (x & 0x000f000f) | 0x6400 =
 * 1024 + (n+8), minus 1032.  High positions: (x & 0x00f000f0) | 0x6400 = 1024 + 16(n+8);
 * times 1/16 minus 72 = n.                                                               */
__device__ __forceinline__ unsigned cvt_u4_lo(unsigned x) {
    unsigned v;
    asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(v) : "r"(x));
    return hsub2(v, 0x64086408u);
}
__device__ __forceinline__ unsigned cvt_u4_hi(unsigned x) {
    unsigned v;
    asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xea;" : "=r"(v) : "r"(x));
    return hfma2(v, 0x2c002c00u /* 1/16 */, 0xd480d480u /* -72 */);
}

/* ---- contraction-dimension maps of Q.K^T: exactly the dims whose codes a thread gets out of its own 16-byte loads of a K row.
 * FP16 cache (m16n8k16): for k-step j (0..7) the four MMA k-slots (2tig, 2tig+1, 2tig+8, 2tig+9) of thread-in-group tig
 * carry head dims 8 (tig + 4 (j >> 1)) + 4 (j & 1) + 0..3.
 * INT4 cache (m16n8k32): for k-step kk (0..3) the eight k-slots (4tig..4tig+3, 16+4tig..16+4tig+3) carry head dims
 * 32 tig + 8 kk + {0, 2, 4, 6} (even nibbles of word kk) and + {1, 3, 5, 7}. */
/* ---- output-dimension map of P.V: n-block jn (0..15), column n (0..7) -> head dim 16 n + jn (INT4) or 8 n + 64 (jn >> 3) + (jn & 7) (FP16):
 * a lane (columns 2 tig, 2 tig + 1) holds 32 (INT4) or twice 16 (FP16) consecutive dims of its head. */

/* Where a warp's piece keeps 16-byte chunk `chunk` (of 32) of head h's row while the warps of a CTA are folded.  The eight lanes of a
 * store (two heads, four tig) hold the same chunk of dims that are 128 or 64 bytes apart: unswizzled they met in one (INT4) or
 * two (FP16) groups of four banks and went out one or two at a time, 256 or 128 wavefronts for each of 11 warps.  us a layer before / with it:
 * 700 tokens (INT4 clusters) 7.5 -> 6.7 together with the fragments that the queries' warps write themselves, 8 ragged INT4 rows 19.6 -> 18.9,
 * FP16 32 768 28.1 -> 27.9. */
template <int DT> __device__ __forceinline__ int stage_chunk(int h, int chunk) {
    return DT == 2 ? chunk ^ ((chunk >> 3) + 4 * (h & 1)) : chunk ^ (((chunk >> 3) & 1) + 2 * (h & 1));
}

/* ---- packed fp32 pairs, one instruction for two values (the same bits): the softmax of INT4 32-token granules, us a layer 68.6 -> 66.5 at 262 144
 * tokens, 8 ragged rows 17.1 -> 17.0 */
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 x, y, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 w, x, y;\n mov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 x, y, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mul.rn.f32x2 w, x, y;\n mov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
struct warp_state {
    float m;      /* reference max (base-2 logits), identical in the 4 lanes of a head; may lag the true max by 2^8 */
    float l;      /* this lane's share of the denominator */
    float o[16][4];
};

__device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

/* Tokens a consumer warp takes at a time.  An INT4 page costs instructions, not bytes (16.9 KB per 128 tokens): with 32 tokens
 * the Q fragments, the maximum's shuffles, the rescale test and the ring bookkeeping are paid half as often and four
 * independent score chains cover each other's latency: 262 144 positions 82.9 -> 73.8 us a layer (3.3 -> 3.75 TB/s), 8 ragged
 * sequences of up to 8 000 tokens 27.3 -> 26.2 us.  FP16 keeps 16: its K and V registers would not fit twice. */
template <int DT> constexpr int kGran = DT == 2 ? 32 : 16;
/* A stage of the ring: an INT4 page, half an FP16 page (64 tokens: K and V rows in one copy each).  Halves fill what two whole pages leave
 * of the shared memory (5 x 32 KB instead of 2 x 64), come and go in smaller steps, and the half behind a row's last token is not fetched: 16 000
 * tokens 17.3 -> 16.5 us a layer, 32 768 26.6 -> 25.8. */
template <int DT> constexpr int kStageTok = DT == 0 ? 64 : 128;
template <int DT> constexpr int kStageBytes = DT == 0 ? 32768 : 16896;
template <int DT> constexpr int kStageV = DT == 0 ? 16384 : 8192;      /* V area of a stage */
template <int DT, bool STAGED> constexpr int kGranStage = (STAGED ? kStageTok<DT> : HY3A_PT) / kGran<DT>;

/* One granule of one warp: loads, S = Q.K^T, online softmax, O += P.V.
 * SM: operands come from a shared-memory copy of the page (32-bit shared addresses) instead
 * of global memory.  FULL: all 16 tokens are valid (no masking).  sq: shared address of this
 * lane's Q fragments; qf: score factor of this lane's head (integer-MMA path).             */
template <int DT, bool SM, bool FULL>
__device__ __forceinline__ void granule(warp_state &st, unsigned sq, float qf, const uint8_t *gpage, unsigned spage, const hy3a_geom &geom,
                                        const int (&k_off)[2][4], const int (&v_off)[8], const int (&sc_off)[2], int gi, int tig, int valid,
                                        float pscale) {
    static_assert(DT == 0 || DT == 2, "INT8 caches are served by decode_umma.cu");
    constexpr int NK = DT == 0 ? 4 : 1;
    constexpr int NV = DT == 0 ? 8 : 2;                      /* V chunks per 16 tokens */
    constexpr int NB = kGran<DT> / 8, NT = kGran<DT> / 16;   /* 8-token blocks, 16-token halves */
    /* byte offsets of granule gi in the stage (or page) */
    const int gk = gi * kGran<DT> * geom.k_row, gv = (SM ? kStageV<DT> : geom.v_off) + gi * (DT == 0 ? 16 : 8 * NT) * geom.v_prow, gs = gi * 2 * kGran<DT>;
    uint4 kr[NB][NK];
#pragma unroll
    for (int nb = 0; nb < NB; nb++) {
        const int o = gk + (nb >> 1) * 16 * geom.k_row;
#pragma unroll
        for (int i = 0; i < NK; i++) kr[nb][i] = SM ? lds16(spage + o + k_off[nb & 1][i]) : ld16(gpage + o + k_off[nb & 1][i]);
    }
    unsigned ksw[NB], vsw[NB];
#pragma unroll
    for (int nb = 0; nb < NB; nb++) ksw[nb] = vsw[nb] = 0;
    if (DT != 0) {
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
            const int o = gs + (nb >> 1) * 32 + sc_off[nb & 1];
            ksw[nb] = SM ? lds4(spage + geom.ks_off + o) : ld4(gpage + geom.ks_off + o);
            vsw[nb] = SM ? lds4(spage + geom.vs_off + o) : ld4(gpage + geom.vs_off + o);
        }
    }
    uint4 vr[NT * NV];
#pragma unroll
    for (int i = 0; i < NT * NV; i++) {
        const int o = gv + (i / NV) * 8 * geom.v_prow + v_off[i % NV];
        vr[i] = SM ? lds16(spage + o) : ld16(gpage + o);
    }

    /* ---- raw scores r[nb][e] of head g for tokens kGran gi + 8nb + 2tig + e (before the K scale) */
    float r[NB][2];
    if (DT == 0) {
        unsigned qa[8][4];
#pragma unroll
        for (int j = 0; j < 8; j++) { uint4 t = lds16(sq + j * 512); qa[j][0] = t.x; qa[j][1] = t.y; qa[j][2] = t.z; qa[j][3] = t.w; }
        float sc[2][4], sd[2][4];   /* even / odd k-steps accumulate separately: four independent MMA chains */
#pragma unroll
        for (int nb = 0; nb < 2; nb++) { sc[nb][0] = sc[nb][1] = sc[nb][2] = sc[nb][3] = 0.f; sd[nb][0] = sd[nb][1] = sd[nb][2] = sd[nb][3] = 0.f; }
#pragma unroll
        for (int i = 0; i < NK; i++) {
#pragma unroll
            for (int nb = 0; nb < 2; nb++) {
                mma16816(sc[nb], qa[2 * i], kr[nb][i].x, kr[nb][i].y);
                mma16816(sd[nb], qa[2 * i + 1], kr[nb][i].z, kr[nb][i].w);
            }
        }
#pragma unroll
        for (int nb = 0; nb < 2; nb++) { r[nb][0] = (sc[nb][0] + sd[nb][0]) + (sc[nb][2] + sd[nb][2]); r[nb][1] = (sc[nb][1] + sd[nb][1]) + (sc[nb][3] + sd[nb][3]); }
    } else {
        uint4 qa[4];
#pragma unroll
        for (int kk = 0; kk < 4; kk++) qa[kk] = lds16(sq + kk * 512);
        int c[NB][4];               /* four independent integer-MMA chains */
#pragma unroll
        for (int nb = 0; nb < NB; nb++) c[nb][0] = c[nb][1] = c[nb][2] = c[nb][3] = 0;
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
#pragma unroll
            for (int nb = 0; nb < NB; nb++) {
                /* two's-complement nibbles: moving a nibble to the top of its byte gives 16 x code as int8 */
                const unsigned w = kk == 0 ? kr[nb][0].x : (kk == 1 ? kr[nb][0].y : (kk == 2 ? kr[nb][0].z : kr[nb][0].w));
                const unsigned b0 = (w << 4) & 0xF0F0F0F0u, b1 = w & 0xF0F0F0F0u;
                imma16832(c[nb], qa[kk], b0, b1);
            }
        }
        /* rows 0-7 carry the high digit of q, rows 8-15 the low digit: q ~ sq*(hi + lo/254) */
#pragma unroll
        for (int nb = 0; nb < NB; nb++) {
            const float2 x = mul2(make_float2((float)(c[nb][0] * 254 + c[nb][2]), (float)(c[nb][1] * 254 + c[nb][3])), make_float2(qf, qf));
            r[nb][0] = x.x; r[nb][1] = x.y;
        }
    }
    /* ---- logits (base 2) and V scales */
    float s[NB][2], vs[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; nb++) {
        float2 kf = make_float2(1.f, 1.f), vf = make_float2(1.f, 1.f);
        if (DT != 0) { kf = unpack_h2(ksw[nb]); vf = unpack_h2(vsw[nb]); }
        const int t0 = kGran<DT> * gi + 8 * nb + 2 * tig;
        const float2 x = mul2(make_float2(r[nb][0], r[nb][1]), kf), y = mul2(vf, make_float2(pscale, pscale));
        s[nb][0] = (FULL || t0 < valid) ? x.x : -INFINITY;
        s[nb][1] = (FULL || t0 + 1 < valid) ? x.y : -INFINITY;
        vs[nb][0] = (FULL || t0 < valid) ? y.x : 0.f;
        vs[nb][1] = (FULL || t0 + 1 < valid) ? y.y : 0.f;
    }
    /* ---- online softmax with a lazily updated reference max: O and l are only rescaled when
     * the granule's max exceeds the reference by more than 2^8; until then p <= 2^8, which the
     * fp16 range of P has room for (pscale leaves 2^8 of headroom).                           */
    float mx = fmaxf(fmaxf(s[0][0], s[0][1]), fmaxf(s[1][0], s[1][1]));
#pragma unroll
    for (int nb = 2; nb < NB; nb += 2) mx = fmaxf(mx, fmaxf(fmaxf(s[nb][0], s[nb][1]), fmaxf(s[nb + 1][0], s[nb + 1][1])));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));   /* the first token of this granule is valid */
    const bool grow = mx > st.m + kRescaleThreshold;       /* also true while st.m == -inf */
    if (__any_sync(0xffffffffu, grow)) {
        const float m_new = grow ? mx : st.m;
        const float alpha = ex2(st.m - m_new);             /* 0 on the first granule (m = -inf), 1 if unchanged */
        st.l *= alpha;
#pragma unroll
        for (int jn = 0; jn < 16; jn++) { st.o[jn][0] *= alpha; st.o[jn][1] *= alpha; st.o[jn][2] *= alpha; st.o[jn][3] *= alpha; }
        st.m = m_new;
    }
    const float mref = st.m == -INFINITY ? 0.f : st.m;     /* no finite score yet: -inf weighs 0, NaN stays NaN */
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {      /* 16 tokens: one k-step of P.V */
        unsigned pa[4];
        {
            float w[2][2], pe[2][2];
#pragma unroll
            for (int nb = 0; nb < 2; nb++) {
                const float2 t = add2(make_float2(s[2 * nt + nb][0], s[2 * nt + nb][1]), make_float2(-mref, -mref));
                pe[nb][0] = ex2(t.x); pe[nb][1] = ex2(t.y);      /* -inf -> 0 */
                const float2 wv = mul2(make_float2(pe[nb][0], pe[nb][1]), make_float2(vs[2 * nt + nb][0], vs[2 * nt + nb][1]));
                w[nb][0] = wv.x; w[nb][1] = wv.y;
            }
            st.l += (pe[0][0] + pe[0][1]) + (pe[1][0] + pe[1][1]);
            pa[0] = pack_h2(w[0][0], w[0][1]);
            pa[2] = pack_h2(w[1][0], w[1][1]);
            if (kPSplit) {
                float2 h0 = unpack_h2(pa[0]), h1 = unpack_h2(pa[2]);
                pa[1] = pack_h2(w[0][0] - h0.x, w[0][1] - h0.y);
                pa[3] = pack_h2(w[1][0] - h1.x, w[1][1] - h1.y);
            } else {
                pa[1] = pa[3] = 0u;
            }
        }
        /* ---- O += P.V over 16 n-blocks of 8 output dims */
        if (DT == 2) {
            const uint4 va = vr[nt * NV], vb = vr[nt * NV + 1];
            unsigned a4[4] = {va.x, va.y, va.z, va.w};
            unsigned b4[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned xa = a4[k], xb = b4[k], xah = xa >> 8, xbh = xb >> 8;
                mma16816(st.o[4 * k + 0], pa, cvt_u4_lo(xa), cvt_u4_lo(xb));
                mma16816(st.o[4 * k + 1], pa, cvt_u4_hi(xa), cvt_u4_hi(xb));
                mma16816(st.o[4 * k + 2], pa, cvt_u4_lo(xah), cvt_u4_lo(xbh));
                mma16816(st.o[4 * k + 3], pa, cvt_u4_hi(xah), cvt_u4_hi(xbh));
            }
        } else {
#pragma unroll
            for (int half = 0; half < 2; half++) {
                /* vr[2t + half]: token t (A,B = b0 pair; C,D = b1 pair), chunk g + 8*half */
                unsigned tA[4] = {vr[0 + half].x, vr[0 + half].y, vr[0 + half].z, vr[0 + half].w};
                unsigned tB[4] = {vr[2 + half].x, vr[2 + half].y, vr[2 + half].z, vr[2 + half].w};
                unsigned tC[4] = {vr[4 + half].x, vr[4 + half].y, vr[4 + half].z, vr[4 + half].w};
                unsigned tD[4] = {vr[6 + half].x, vr[6 + half].y, vr[6 + half].z, vr[6 + half].w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    mma16816(st.o[8 * half + 2 * k], pa, prmt(tA[k], tB[k], 0x5410u), prmt(tC[k], tD[k], 0x5410u));
                    mma16816(st.o[8 * half + 2 * k + 1], pa, prmt(tA[k], tB[k], 0x7632u), prmt(tC[k], tD[k], 0x7632u));
                }
            }
        }
    }
}

/* DIRECT variant (STAGED=false): operands fetched straight from global memory with 128-bit
 * loads (no ring, no producer).  STAGED variant: kWarps consumer warps + 1 producer warp.
 * Same arithmetic, same results.                                                          */
/* SHARD: the sequence-sharded variant (exchange + final fold in the epilogue); a separate instantiation so that the
 * single-GPU kernel's register allocation is untouched by it. */
/* CL: 0 = any grid, 2 / 4 / 8 = a cluster of CL CTAs per (row, KV head) */
template <int DT, bool STAGED, bool SHARD = false, int CL = 0>
__global__ void __launch_bounds__(kThreads + (STAGED ? 32 : 0), 1) hy3a_decode_kernel(hy3a_cache_view cache, hy3a_batch_view batch, decode_args a) {
    /* dynamic shared memory: [s_o | s_ml | s_q | s_new | a cluster's landing zone | page-count prefix | empty[8] full[16] meeting | ring of pages] */
    extern __shared__ __align__(128) uint8_t s_dyn[];
    float (*s_o)[8][HY3A_D] = reinterpret_cast<float (*)[8][HY3A_D]>(s_dyn);                       /* per-warp unnormalised outputs */
    float (*s_ml)[8][2] = reinterpret_cast<float (*)[8][2]>(s_dyn + kFixedO);                      /* per-warp {m, l} */
    uint4 (*s_q)[32] = reinterpret_cast<uint4 (*)[32]>(s_dyn + kFixedO + kFixedML);                /* Q fragments: [k-step][lane] */
    float (*s_new)[HY3A_D] = reinterpret_cast<float (*)[HY3A_D]>(s_dyn + kFixedO + kFixedML + kFixedQ);   /* fused step: the new K row (normalised, rotated) and V row */
    __shared__ float s_qf[8];
    __shared__ unsigned s_vnew;
    __shared__ int s_flag;
    __shared__ int s_abort;
    __shared__ cta_plan s_plan;

    const hy3a_geom geom = hy3a_make_geom(DT);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int n = batch.n, G = cache.kv_heads;
    const int cta = blockIdx.x;

    int *s_prefix = reinterpret_cast<int *>(s_dyn + kFixed<CL>);
    const unsigned bar_base = smem_u32(s_dyn + kFixed<CL> + a.prefix_bytes);
    const unsigned ring_base = bar_base + kBarBytes<CL>;

    if (a.wait_first) asm volatile("griddepcontrol.wait;" ::: "memory");
    /* ---- What the query set-up needs besides the queries (norm weights, RoPE table, positions) comes from the host: warps 0-7 (queries) and 9
     * (new K row) fetch it now, off the critical path; the planning warp sets the barriers up while its rows' slots are on the way. */
    constexpr int kPlanWarp = STAGED ? kWarps : 0;
    const int rl_d0 = (lane >> 4) * 64 + (lane & 15) * 4;
    float4 pre_w = make_float4(1.f, 1.f, 1.f, 1.f), pre_f = make_float4(0.f, 0.f, 0.f, 0.f);
    float pre_c[4] = {1.f, 1.f, 1.f, 1.f}, pre_s[4] = {0.f, 0.f, 0.f, 0.f};
    int pre_row = -1, pos_l = 0;           /* pos_l: position of row `lane`, up to 32 rows */
    const bool ropes = a.fused && (warp < 8 || warp == 9);
    if (ropes) {
        pre_w = *reinterpret_cast<const float4 *>(a.norm_w + (warp == 9 ? HY3A_D : 0) + rl_d0);
        pre_f = hy3a_rowops::rope_freqs(a.rope, lane);
        if (lane < n) pos_l = batch.pos[lane];
    }
    if (n > 32) {
        for (int i = tid; i < n; i += blockDim.x) s_prefix[i + 1] = pages_of_slot(batch.slot[i]);
        __syncthreads();
    }
    lane_rows rows = {-1, 0};
    if (warp == kPlanWarp) {
        rows = load_rows(batch, n, lane);
        if (lane == 0) {
            s_abort = 0;
            if (STAGED) {
                for (int i = 0; i < a.stages; i++) mbar_init(bar_base + 8 * i, 32 * kGranStage<DT, STAGED>);   /* empty[stage]: every thread of the warps that share it */
                for (int i = 0; i < 16; i++) mbar_init(bar_base + 64 + 8 * i, 1);   /* full[ring position mod n_full]: the producer's expect_tx */
                if (CL) mbar_init(bar_base + kBarClu, 1);
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                if (CL) mbar_expect_tx(bar_base + kBarClu, kCluBytes);
            }
        }
        plan<DT, CL>(&s_plan, s_prefix, rows.slot, n, G, gridDim.x, cta, lane);
    }
    if (CL) cluster_arrive();      /* every CTA of the cluster has set its barrier up; cluster_wait below */
    const bool is_producer = STAGED && warp == kWarps;
    if (is_producer) asm volatile("bar.arrive 2, %0;" ::"r"(blockDim.x) : "memory");      /* the others need the plan; the copies need no one */
    else asm volatile("bar.sync 2, %0;" ::"r"(blockDim.x) : "memory");

    const long long U = (long long)G * s_prefix[n], u_begin = s_plan.u0, u_end = s_plan.u1;
    const bool aligned = s_plan.aligned, idle = u_begin == u_end;
    const int C = (long long)gridDim.x < U ? (int)gridDim.x : (int)U;
    const int al_first = s_plan.first, al_pieces = s_plan.pieces;
    /* cos / sin of a row's position */
    auto rope_row = [&](int row) {
        hy3a_rowops::rope_coeffs(pre_c, pre_s, a.rope, pre_f, n <= 32 ? __shfl_sync(0xffffffffu, pos_l, row) : batch.pos[row]);
        pre_row = row;
    };
    if (ropes && !idle) rope_row(locate(s_prefix, batch, n, G, u_begin, u_end).row);
    /* Everything above reads only what the host wrote (batch descriptor).  From here on the kernel
     * touches memory that the preceding kernel in the stream may produce (queries, the newest KV
     * slot, scratch records), so wait for it -- except the producer lane, which first starts the
     * copies of pages that lie wholly below the newest slot (append-only cache: immutable).       */
    if (CL && !is_producer) cluster_wait();
    const unsigned n_full = STAGED ? 16u / (unsigned)a.stages * (unsigned)a.stages : 1u;   /* "full" barriers: a multiple of the stages */
    if (!is_producer) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        /* Only now may the NEXT kernel in the stream start its prologue: it then knows that everything
         * older than this kernel is complete, so the only writes it can race with are this kernel's
         * (the newest slot of each row), which its early page fetches stay clear of.                  */
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    /* rows with no keys on this rank: zero output / empty partial (hy3_gpu.cu:197-199) */
    for (int i = CL ? n : cta; i < n; i += gridDim.x) {
        if (s_prefix[i + 1] != s_prefix[i]) continue;
        if (SHARD) {
            /* sharded: the empty record {m = -inf, l = 0} of every head goes to every other rank now (one flagged line;
             * the fold skips it without reading acc); this rank's own fold of the row happens at the end of the kernel,
             * when the other ranks' records are due */
            if (is_producer) continue;
            for (int e = tid; e < G * 8; e += kThreads) {
                const unsigned flag = a.shard_round[i * G * 8 + e] + 1u;
                for (int r = 0; r < a.n_dest; r++)
                    if (r != a.my_rank) shard_store_line(a.dest[r] + ((size_t)i * G * 8 + e) * kShardLines, -INFINITY, 0.f, flag);
            }
            continue;
        }
        if (!is_producer) HY3A_EMPTY_ROW(i, tid, kThreads);
    }

    if (idle && !SHARD && !CL) return;   /* sharded: idle CTAs may still own the fold of rows without local keys */


    if (STAGED && warp == kWarps) {
        /* ================= producer warp: one lane streams the CTA's pages into the ring (the warp finds the segments).  It shares a
         * scheduler with two consumer warps, so the loop is short: stage, parity and barrier are carried along, addresses are a base and a
         * stride.  INT4 262 144 tokens 66.5 -> 62.5 us a layer, 8 ragged rows 17.0 -> 16.7; with every lane in the loop, each holding a
         * page's block-table entry, 71. */
        unsigned it = 0, stage = 0, phase = 1, fb = 0;      /* ring position, its stage, the parity to wait for there and its "full" barrier, carried along */
        bool ok = true;
        bool waited = false;   /* griddepcontrol.wait executed yet? */
        const unsigned long long pol = l2_evict_first_policy();
        if (!a.early_prefetch) { asm volatile("griddepcontrol.wait;" ::: "memory"); waited = true; }
        for (long long u = u_begin; u < u_end && ok;) {
            const segment sg = locate(s_prefix, batch, rows, n, G, u, u_end);
            const int *bt = cache.block_table + (size_t)sg.seq * cache.max_blocks_per_seq;
            if (lane == 0) {
                const uint8_t *page0 = cache.pool + hy3a_page_index(cache, 0, a.layer, sg.hl) * (size_t)cache.page_bytes;
                const size_t block_bytes = (hy3a_page_index(cache, 1, a.layer, sg.hl) - hy3a_page_index(cache, 0, a.layer, sg.hl)) * (size_t)cache.page_bytes;
                int block_next = bt[sg.p_begin];
                for (int p = sg.p_begin; p < sg.p_end; p++) {
                    const uint8_t *page = page0 + block_next * block_bytes;
                    if (p + 1 < sg.p_end) block_next = bt[p + 1];   /* in flight while we wait for the stage */
#pragma unroll
                    for (int half = 0; half < HY3A_PT / kStageTok<DT>; half++) {
                        const int t_end = p * HY3A_PT + (half + 1) * kStageTok<DT>;
                        if (half && t_end - kStageTok<DT> >= sg.len) break;
                        /* before the preceding kernel is known to be complete only tokens that lie wholly below
                         * the newest slot may be fetched, and only into stages that were never used            */
                        if (!waited && (it >= (unsigned)a.stages || t_end > sg.len - 2)) { asm volatile("griddepcontrol.wait;" ::: "memory"); waited = true; }
                        ok = mbar_wait(bar_base + 8 * stage, phase, &s_abort, a.err, 1u);
                        if (!ok) break;
                        const unsigned full = bar_base + 64 + 8 * fb, dst = ring_base + stage * (unsigned)kStageBytes<DT>;
                        mbar_expect_tx(full, (unsigned)kStageBytes<DT>);
                        if (DT == 0) {
                            bulk_g2s(dst, page + half * kStageV<DT>, kStageV<DT>, full, pol);
                            bulk_g2s(dst + kStageV<DT>, page + HY3A_PT * 256 + half * kStageV<DT>, kStageV<DT>, full, pol);
                        } else {
                            bulk_g2s(dst, page, (unsigned)kStageBytes<DT>, full, pol);
                        }
                        it++;
                        if (++stage == (unsigned)a.stages) { stage = 0; phase ^= 1u; }
                        if (++fb == n_full) fb = 0;
                    }
                    if (!ok) break;
                }
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            u = sg.seg_u0 + sg.p_end;
        }
        if (lane == 0 && !waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        if (lane == 0 && !ok) {
            /* gave up: let the copies already issued land before the CTA's shared memory goes away */
            const unsigned first = it > (unsigned)a.stages ? it - (unsigned)a.stages : 0u;
            for (unsigned j = first; j < it; j++) {
                const unsigned fb = j % n_full, fphase = (j / n_full) & 1u;
                for (unsigned spin = 0; spin < (1u << 20) && !mbar_test(bar_base + 64 + 8 * fb, fphase); spin++) __nanosleep(64);
            }
        }
        if (CL) { __syncwarp(); cluster_wait(); cluster_arrive(); cluster_wait(); }
        return;
    }

    /* ================= consumer warps */
    int k_off[2][4];   /* [n-block][chunk], relative to the granule, loop invariant */
    int v_off[8];
    int sc_off[2];
#pragma unroll
    for (int nb = 0; nb < 2; nb++) {
        int tok = 8 * nb + g;
        if (DT == 2) { k_off[nb][0] = hy3a_k_chunk_off<2>(tok, tig); k_off[nb][1] = k_off[nb][2] = k_off[nb][3] = 0; }
        else { for (int i = 0; i < 4; i++) k_off[nb][i] = hy3a_k_chunk_off<0>(tok, tig + 4 * i); }
        sc_off[nb] = 2 * (8 * nb + 2 * tig);
    }
    {
        int pr0 = tig, pr1 = pr0 + 4;
        if (DT == 2) {
            v_off[0] = hy3a_v_chunk_off<2>(pr0, g); v_off[1] = hy3a_v_chunk_off<2>(pr1, g);
            for (int i = 2; i < 8; i++) v_off[i] = 0;
        } else {
            int tA = 2 * tig;
            for (int t = 0; t < 4; t++) {
                int tok = tA + (t & 1) + 8 * (t >> 1);
                v_off[2 * t] = hy3a_v16_chunk_off(tok, g);
                v_off[2 * t + 1] = hy3a_v16_chunk_off(tok, g + 8);
            }
        }
    }
    const unsigned sq = smem_u32(&s_q[0][lane]);

    unsigned it = 0; /* pages consumed by this CTA so far (ring position) */
    long long u = u_begin;
    while (u < u_end) {
        const segment sg = locate(s_prefix, batch, n, G, u, u_end);
        const int row = sg.row, hl = sg.hl, sidx = sg.sidx;
        const int head0 = (cache.kv_head_begin + hl) * 8;   /* first of the segment's 8 query heads */

        /* ---- Q operand fragments of the segment's 8 heads, pre-packed per (k-step, lane).
         * Warp w < 8 owns head w as a row of 4 values per lane (dims d0..d0+3); in the fused step it
         * first applies the per-head RMSNorm and RoPE (same code as the append kernel).  The softmax
         * scale 1/sqrt(128) (hy3_gpu.cu:193) and log2(e) are folded into the fragments.  The warp writes the fragments
         * straight from its registers (gathering them from a staged copy cost a second barrier and 16 byte loads: 8 ragged INT4 rows
         * 18.9 -> 18.7 us a layer). */
        float qf = 1.f;
        /* what the scales of P and the append need from memory: issued with the loads of the queries */
        const unsigned vs_old = DT != 0 ? cache.vs_max[a.layer * G + hl] : 0u;
        const int new_page = (sg.len - 1) >> 7;
        const bool has_new = a.fused && a.k_in && new_page >= sg.p_begin && new_page < sg.p_end;
        int new_block = 0;
        if (has_new) new_block = cache.block_table[(size_t)sg.seq * cache.max_blocks_per_seq + new_page];
        if (warp < 8) {
            const int d0 = (lane >> 4) * 64 + (lane & 15) * 4;
            float x[4];
            if (a.fused) {
                const float4 xv = *reinterpret_cast<const float4 *>(a.q_in + (size_t)row * a.qi_stride + (size_t)(head0 + warp) * HY3A_D + d0);
                x[0] = xv.x; x[1] = xv.y; x[2] = xv.z; x[3] = xv.w;
                if (row != pre_row) rope_row(row);
                hy3a_rowops::norm_rope_apply(x, pre_w, a.eps, pre_c, pre_s, lane);
                if (a.q_out && sg.p_begin == 0)
                    *reinterpret_cast<float4 *>(a.q_out + (size_t)row * a.q_out_stride + (size_t)(head0 + warp) * HY3A_D + d0) = make_float4(x[0], x[1], x[2], x[3]);
            } else {
                const float4 xv = *reinterpret_cast<const float4 *>(a.q + (size_t)row * a.q_stride + (size_t)(head0 + warp) * HY3A_D + d0);
                x[0] = xv.x; x[1] = xv.y; x[2] = xv.z; x[3] = xv.w;
            }
            if (DT == 0) {
                /* fp16 value in rows 0-7, fp16 residual in rows 8-15.  The lane's dims d0..d0+3 are one thread-in-group's four k-slots
                 * of one k-step: it writes that fragment */
                const float qs = 0.08838834764831845f * kLog2e;
                float lo4[4];
#pragma unroll
                for (int j = 0; j < 4; j++) { x[j] *= qs; lo4[j] = x[j] - __half2float(__float2half_rn(x[j])); }
                const int c = d0 >> 3;
                s_q[2 * (c >> 2) + ((d0 >> 2) & 1)][4 * warp + (c & 3)] = make_uint4(pack_h2(x[0], x[1]), pack_h2(lo4[0], lo4[1]), pack_h2(x[2], x[3]), pack_h2(lo4[2], lo4[3]));
            } else {
                /* two int8 digits per query element: q ~ sq*(hi + lo/254), |hi|,|lo| <= 127, so the
                 * quantisation step is absmax/32258 per head                                       */
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
                /* rows 0-7 = hi, rows 8-15 = lo.  The lane's dims are half of the eight k-slots of k-step (d0 >> 3) & 3, thread-in-group
                 * d0 >> 5: two even ones (words 0, 1 of the fragment) and two odd ones (words 2, 3) */
                unsigned char *fr = reinterpret_cast<unsigned char *>(&s_q[(d0 >> 3) & 3][4 * warp + (d0 >> 5)]) + ((d0 & 7) >> 1);
                *reinterpret_cast<unsigned short *>(fr) = (unsigned short)prmt(hw, 0u, 0x0020u);
                *reinterpret_cast<unsigned short *>(fr + 4) = (unsigned short)prmt(lw, 0u, 0x0020u);
                *reinterpret_cast<unsigned short *>(fr + 8) = (unsigned short)prmt(hw, 0u, 0x0031u);
                *reinterpret_cast<unsigned short *>(fr + 12) = (unsigned short)prmt(lw, 0u, 0x0031u);
                if (lane == 0) s_qf[warp] = sqv * (1.f / 254.f) * 0.08838834764831845f * kLog2e * (DT == 2 ? 0.0625f : 1.f);
            }
        } else if (warp == 8) {
            /* fused step: the scale the new V row will get (hy3_gpu.cu:260-262), so that every CTA of the
             * segment sizes its P scale for it as well                                                 */
            unsigned vb = 0;
            if (DT != 0 && a.fused && a.k_in) {
                const float4 xv = *reinterpret_cast<const float4 *>(a.v_in + (size_t)row * a.vi_stride + (size_t)(cache.kv_head_begin + hl) * HY3A_D + 4 * lane);
                float m = fmaxf(fmaxf(fabsf(xv.x), fabsf(xv.y)), fmaxf(fabsf(xv.z), fabsf(xv.w)));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                vb = (unsigned)__half_as_ushort(__float2half(__fadd_rn(__fdiv_rn(m, 7.f), 1e-8f)));
            }
            if (lane == 0) s_vnew = vb;
        } else if (has_new) {
            /* the new rows, ready by the time their page is: the warp that holds the newest slot then only quantises and stores
             * (loading, normalising and rotating them there cost every launch 1 to 2 us behind the last page) */
            const size_t kvh = (size_t)(cache.kv_head_begin + hl) * HY3A_D + rl_d0;
            if (warp == 9) {
                const float4 k4 = *reinterpret_cast<const float4 *>(a.k_in + (size_t)row * a.ki_stride + kvh);
                float y[4] = {k4.x, k4.y, k4.z, k4.w};
                if (row != pre_row) rope_row(row);
                hy3a_rowops::norm_rope_apply(y, pre_w, a.eps, pre_c, pre_s, lane);
                *reinterpret_cast<float4 *>(&s_new[0][rl_d0]) = make_float4(y[0], y[1], y[2], y[3]);
            } else if (warp == 10) {
                *reinterpret_cast<float4 *>(&s_new[1][rl_d0]) = *reinterpret_cast<const float4 *>(a.v_in + (size_t)row * a.vi_stride + kvh);
            }
        }
        consumer_sync();
        if (DT != 0) qf = s_qf[g];
        const unsigned vnew = s_vnew;
        /* P scale: w = p * vscale * 2^E with vs_max * 2^E <= 2^6 and p <= 2^8, so fp16 P never
         * overflows and its subnormal floor sits 2^-30 below the reference max.               */
        float pscale;
        {
            int E = 6;
            if (DT != 0) {
                const unsigned vb = vs_old > vnew ? vs_old : vnew;   /* positive fp16 bit patterns order like the numbers */
                __half_raw hr; hr.x = (unsigned short)vb;
                float vmax = __half2float(__half(hr));
                int ex;
                frexpf(fmaxf(vmax, 1e-30f), &ex); /* vmax < 2^ex */
                E = 6 - ex;
                E = E > 60 ? 60 : (E < -60 ? -60 : E);
            }
            pscale = exp2f((float)E);
        }

        warp_state st;
        st.m = -INFINITY; st.l = 0.f;
#pragma unroll
        for (int jn = 0; jn < 16; jn++) { st.o[jn][0] = st.o[jn][1] = st.o[jn][2] = st.o[jn][3] = 0.f; }

        /* granule slot x = GP*(ring position of the stage) + granule-in-stage; warp w takes slots
         * x = w (mod kWarps), so any number of consumer warps shares the GP granules of a stage and
         * each stage is released by exactly GP warps (one arrival per thread per slot).  (Direct variant: stage = page.) */
        constexpr unsigned GP = kGranStage<DT, STAGED>;
        constexpr int GT = kGran<DT>, ST = STAGED ? kStageTok<DT> : HY3A_PT;
        /* stages of the piece, and of those in the sequence's last page */
        const int t_end = min(sg.len, sg.p_end * HY3A_PT), tail_t0 = (sg.pages - 1) * HY3A_PT;
        const unsigned it_end = it + (unsigned)((t_end - sg.p_begin * HY3A_PT + ST - 1) / ST);
        unsigned x = it * GP + ((unsigned)warp + kWarps - (it * GP) % kWarps) % kWarps, pit = x / GP;
        /* ring position of stage pit, its "full" barrier and that barrier's phase, carried along (no divisions per granule) */
        unsigned stage = STAGED ? pit % (unsigned)a.stages : 0u, fb = pit % n_full, fphase = (pit / n_full) & 1u;
        auto advance = [&]() {
            x += kWarps;
            const unsigned d = x / GP - pit;
            pit += d;
            if (STAGED) {
                stage += d;
                while (stage >= (unsigned)a.stages) stage -= (unsigned)a.stages;
                fb += d;
                if (fb >= n_full) { fb -= n_full; fphase ^= 1u; }
            }
        };
        if (STAGED) {
            /* A warp holds granules in GP of every 11 stages, so it may skip a use of a stage, and an mbarrier wait only knows
             * the parity of a phase: with one "full" barrier per stage the warp's next wait on that stage could pass on the
             * stale phase while the skipped copy is still landing (seen with a two-stage ring of FP16 pages).  So the
             * barriers are cycled over n_full ring positions: position pit - n_full, whose phase a wait for pit could mistake, has
             * long been consumed, because this warp's last position pit' >= pit - ceil(11 / GP) was issued after pit' - stages
             * had been consumed, and n_full >= stages + ceil(11 / GP). */
            auto page_wait = [&]() {
                mbar_wait(bar_base + 64 + 8 * fb, fphase, &s_abort, a.err, 2u);
                return ring_base + stage * (unsigned)kStageBytes<DT>;
            };
            /* The sequence's last page has its masks and the fused append; it stands behind the loop (a warp has one granule of it at most),
             * whose body is then one granule's code (INT4 8 ragged rows 18.0 -> 17.3 us a layer, 32 768 tokens 17.0 -> 16.5; FP16 32 768 26.8 -> 26.6). */
            const unsigned whole = it_end - (sg.p_end == sg.pages ? (unsigned)((sg.len - tail_t0 + ST - 1) / ST) : 0u);
            for (; x < whole * GP; advance()) {
                const unsigned spage = page_wait();
                granule<DT, true, true>(st, sq, qf, nullptr, spage, geom, k_off, v_off, sc_off, (int)(x % GP), tig, HY3A_PT, pscale);
                mbar_arrive(bar_base + 8 * stage); /* every thread of the warps that share a page releases it */
            }
            if (x < it_end * GP) {
                /* valid: tokens from the stage's first one on; the newest is number valid - 1 */
                const int gi = (int)(x % GP), valid = sg.len - tail_t0 - (int)(pit - whole) * ST;
                const unsigned spage = page_wait();
                if (has_new && valid <= ST && gi == (valid - 1) / GT) {
                    /* fused append: this warp holds the only granule that contains the newest slot.  It quantises the new rows
                     * exactly as the append kernel does and writes them into the shared-memory copy it is about to read and to
                     * the page in HBM (for later steps). */
                    const int tok = (sg.len - 1) & 127;
                    uint8_t *gp = cache.pool + hy3a_page_index(cache, new_block, a.layer, hl) * (size_t)cache.page_bytes;
                    uint8_t *sp = s_dyn + kFixed<CL> + a.prefix_bytes + kBarBytes<CL> + (size_t)stage * kStageBytes<DT>;
                    hy3a_geom sgeom = geom;      /* of the stage: its rows are swizzled alike */
                    sgeom.v_off = kStageV<DT>;
                    const int stok = valid - 1;
                    float4 r4 = *reinterpret_cast<const float4 *>(&s_new[0][rl_d0]);
                    float y[4] = {r4.x, r4.y, r4.z, r4.w};
                    hy3a_rowops::store_row<DT>(sp, sgeom, stok, false, y, rl_d0, lane);
                    hy3a_rowops::store_row<DT>(gp, geom, tok, false, y, rl_d0, lane);
                    r4 = *reinterpret_cast<const float4 *>(&s_new[1][rl_d0]);
                    y[0] = r4.x; y[1] = r4.y; y[2] = r4.z; y[3] = r4.w;
                    const unsigned sb = hy3a_rowops::store_row<DT>(sp, sgeom, stok, true, y, rl_d0, lane);
                    hy3a_rowops::store_row<DT>(gp, geom, tok, true, y, rl_d0, lane);
                    if (DT != 0 && lane == 0) atomicMax(cache.vs_max + a.layer * G + hl, sb);
                    __syncwarp();
                }
                if (GT * gi < valid) granule<DT, true, false>(st, sq, qf, nullptr, spage, geom, k_off, v_off, sc_off, gi, tig, valid, pscale);
                mbar_arrive(bar_base + 8 * stage);
                advance();
            }
        } else {
            for (; x < it_end * GP; advance()) {
                const int gi = (int)(x % GP), p = sg.p_begin + (int)(pit - it);
                const int valid = min(HY3A_PT, sg.len - p * HY3A_PT);
                if (GT * gi >= valid) continue; /* warp-uniform */
                const int block = cache.block_table[(size_t)sg.seq * cache.max_blocks_per_seq + p];
                const uint8_t *page = cache.pool + hy3a_page_index(cache, block, a.layer, hl) * (size_t)cache.page_bytes;
                granule<DT, false, false>(st, sq, qf, page, 0u, geom, k_off, v_off, sc_off, gi, tig, valid, pscale);
            }
        }
        it = it_end;

        /* ---- fold the consumer warps of this CTA (shared memory) */
        {
            float l = st.l;
            l += __shfl_xor_sync(0xffffffffu, l, 1);
            l += __shfl_xor_sync(0xffffffffu, l, 2);
            if (tig == 0) { s_ml[warp][g][0] = st.m; s_ml[warp][g][1] = l; }
            const float inv_ps = 1.f / pscale;
            /* the lane's 32 dims as eight 16-byte chunks: o[4q + j][b] is dim 16 (2 tig + b) + 4q + j (INT4) or
             * 64 (q >> 1) + 8 (2 tig + b) + 4 (q & 1) + j (FP16) */
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int b = 0; b < 2; b++) {
                    const int chunk = DT == 2 ? 8 * tig + 4 * b + q : 16 * (q >> 1) + 4 * tig + 2 * b + (q & 1);
                    *reinterpret_cast<float4 *>(&s_o[warp][g][4 * stage_chunk<DT>(g, chunk)]) =
                        make_float4((st.o[4 * q][b] + st.o[4 * q][b + 2]) * inv_ps, (st.o[4 * q + 1][b] + st.o[4 * q + 1][b + 2]) * inv_ps,
                                    (st.o[4 * q + 2][b] + st.o[4 * q + 2][b + 2]) * inv_ps, (st.o[4 * q + 3][b] + st.o[4 * q + 3][b + 2]) * inv_ps);
                }
        }
        consumer_sync();
        const bool red = tid < 256;                            /* the first 8 warps do the reductions */
        const int h = (tid >> 5) & 7, d4 = (tid & 31) * 4;    /* thread -> (head, 4 dims) */
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWarps; w++) M = fmaxf(M, s_ml[w][h][0]);
        float L = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            const float2 ml = *reinterpret_cast<const float2 *>(s_ml[w][h]);
            if (ml.y == 0.f) continue;
            const float f = ex2(ml.x - M);
            L += ml.y * f;
            const float4 o4 = *reinterpret_cast<const float4 *>(&s_o[w][h][4 * stage_chunk<DT>(h, lane)]);
            acc[0] += o4.x * f; acc[1] += o4.y * f; acc[2] += o4.z * f; acc[3] += o4.w * f;
        }
        if (CL) {
            if (red) cluster_send<CL ? CL : 1>(smem_u32(s_dyn) + kFixedHead, bar_base + kBarClu, cta % (CL ? CL : 1), h, lane, M, L, acc);
            break;
        }
        if (SHARD) consumer_sync();      /* s_o / s_ml are landing zones below; else they are written again behind the next segment's queries */

        /* ---- how many CTAs share this segment? */
        const int c_first = aligned ? al_first : cta_of_unit(sg.seg_u0, U, C);
        const int npieces = aligned ? al_pieces : cta_of_unit(sg.seg_u1 - 1, U, C) - c_first + 1;
        const int rec_base = aligned ? 0 : sidx;   /* record index = CTA (+ segment when CTAs may hold several pieces) */
        const size_t head_q = (size_t)(cache.kv_head_begin + hl) * 8 + h; /* global query head */
        u = sg.seg_u0 + sg.p_end;

        /* Which of the 8 heads this CTA finishes (writes out / exchanges): all of them, unless the fold of a
         * segment is spread over several of its CTAs (below). */
        int h_lo = 0, h_hi = 8;
        bool last = true;      /* this warp has its head's final record */
        float *const recs = a.scratch + ((size_t)(c_first + rec_base) * 8 + h) * kRecFloats;      /* of the segment's piece 0 */
        if (npieces > 1) {
            if (STAGED && aligned && a.spread) {
                /* ---- CTA-aligned segments (small batches): the fold is SPREAD.  Every CTA announces its record on
                 * the segment's arrival counter; the first F pieces then each fold 8/F of the heads over all pieces
                 * (one warp per head), instead of one CTA pulling every head of every piece while the others have
                 * left.  The remaining pieces leave at once.                                                      */
                const int Fmax = a.spread, F = npieces >= Fmax ? Fmax : (npieces >= 4 && Fmax >= 4 ? 4 : (npieces >= 2 && Fmax >= 2 ? 2 : 1)), hpf = 8 / F, piece = cta - c_first;
                if (red) store_record(recs + (size_t)piece * 8 * kRecFloats, lane, M, L, acc);
                consumer_sync();   /* the record is complete in CTA scope; the release publishes it */
                if (tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.counters + 8 * sidx) : "memory");
                if (piece >= F) continue;   /* CTA-uniform */
                if (tid == 0) {
                    /* bounded wait for the other pieces (they are resident: one CTA per SM at most) */
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
                            if (s_abort || (i >= (1u << 14) && t1 - t0 > 500000000ull)) break;
                        }
                    }
                    if (!ok) { s_abort = 1; if (atomicCAS(a.err, 0u, 4u) == 0u) { a.err[1] = 50u; a.err[2] = blockIdx.x; a.err[3] = seen; } }
                    s_flag = ok;
                }
                consumer_sync();
                h_lo = piece * hpf; h_hi = h_lo + hpf;
                const bool mine = red && h >= h_lo && h < h_hi;
                M = -INFINITY; L = 0.f; acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                if (s_flag && mine) {
                    const int slots = min(32, a.stages * kStageBytes<DT> / (hpf * 512));      /* the ring is idle: this CTA's pages are consumed */
                    fold_records(recs, npieces, s_dyn + kFixed<CL> + a.prefix_bytes + kBarBytes<CL> + (h - h_lo) * slots * 512, 512u, slots, lane, M, L, acc);
                }
                consumer_sync();   /* every landing zone is read (the sharded exchange lands its lines in the ring too) */
                if (tid == 0) {
                    /* the last of the F folders puts both counters back to zero for the next launch */
                    unsigned *done = a.counters + 8 * a.n_counters + sidx;
                    const unsigned old = atomicAdd(done, 1u);
                    if (old == (unsigned)(F - 1)) { a.counters[8 * sidx] = 0u; *done = 0u; }
                }
            } else {
                /* The last CTA to arrive folds, nobody waits.  The records land in the page ring where it is idle (whole CTAs to a segment:
                 * this CTA's pages are consumed), else in the head's column of s_o, which this warp alone has read. */
                const bool ring = STAGED && aligned;
                const int slots = ring ? min(32, a.stages * kStageBytes<DT> / 4096) : kWarps;
                uint8_t *const zone = ring ? s_dyn + kFixed<CL> + a.prefix_bytes + kBarBytes<CL> + h * slots * 512 : reinterpret_cast<uint8_t *>(s_o[0][h]);
                if (red) last = fold_last(recs, cta - c_first, npieces, a.counters + 8 * sidx + h, zone, ring ? 512u : (unsigned)sizeof(s_o[0]), slots, lane, M, L, acc);
                if (SHARD) consumer_sync();      /* the exchange lands its lines there too */
            }
        }
        const bool fin = red && last && h >= h_lo && h < h_hi;   /* this thread finishes its (head, 4 dims) of the segment */
        if (SHARD) {
            /* sequence sharding: this rank's records of the segment go into every other rank's gather buffer as
             * flagged lines (no fence, no separate flag: a line is valid when both of its flag words carry this
             * use's number), then the same threads collect the other ranks' lines and finish the segment */
            const int seg = row * G + hl;
            if (fin) {
                const unsigned flag = a.shard_round[seg * 8 + h] + 1u;   /* use count of this (slot, segment, head) */
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
                fa.n_ranks = a.n_dest; fa.my_rank = a.my_rank; fa.line_a = 1 + (d4 >> 1); fa.flag = flag; fa.stage = reinterpret_cast<const uint4 *>(s_dyn); fa.h = h; fa.lane = lane;
                fa.own_m = m_nat; fa.own_l = L; fa.own_acc[0] = acc[0]; fa.own_acc[1] = acc[1]; fa.own_acc[2] = acc[2]; fa.own_acc[3] = acc[3];
                if (STAGED && aligned && (size_t)a.stages * kStageBytes<DT> >= (size_t)8 * 8 * kShardLines * 16) {
                    /* CTA-aligned segments: the page ring is idle by now and holds all 8 ranks' records at once, so
                     * every rank is polled in the same round */
                    fa.stage = reinterpret_cast<const uint4 *>(s_dyn + kFixed<CL> + a.prefix_bytes + kBarBytes<CL>);
                    shard_fold<8>(fa);
                } else {
                    shard_fold<kShardBatch>(fa);
                }
                __syncwarp();                /* every lane of the head's warp has read the use count */
                if (d4 == 0) a.shard_round[seg * 8 + h] = flag;
            }
            consumer_sync();                 /* the landing zones may be reused by the next segment */
            continue;
        }
        if (!fin) continue;
        if (a.user_partials) {
            float *rec = a.user_partials + ((size_t)row * G * 8 + (size_t)hl * 8 + h) * HY3A_PARTIAL_FLOATS;
            if (d4 == 0) { rec[0] = M * kLn2; rec[1] = L; } /* m in natural-log units like the reference record */
            rec[2 + d4] = acc[0]; rec[3 + d4] = acc[1]; rec[4 + d4] = acc[2]; rec[5 + d4] = acc[3];
        } else {
            float inv = inv_sum(L);
            float4 o4 = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
            *reinterpret_cast<float4 *>(a.out + (size_t)row * a.out_stride + head_q * HY3A_D + d4) = o4;
        }
    }
    if (CL) {
        constexpr int C1 = CL ? CL : 1, HPC = 8 / C1;
        const int rank = cta % C1, seg = cta / C1, row = seg / G, hl = seg - row * G;
        const float none[4] = {0.f, 0.f, 0.f, 0.f};
        if (idle && warp < 8) cluster_send<C1>(smem_u32(s_dyn) + kFixedHead, bar_base + kBarClu, rank, warp, lane, -INFINITY, 0.f, none);
        if (warp < HPC) {
            mbar_wait(bar_base + kBarClu, 0u, &s_abort, a.err, 70u);
            float M, Ls, acc[4];
            cluster_fold<C1>(s_dyn + kFixedHead, warp, lane, M, Ls, acc);
            cluster_write(a, G, cache.kv_head_begin, row, hl * 8 + rank * HPC + warp, lane, M, Ls, acc);
        }
        /* a CTA's shared memory stays until every CTA of the cluster has sent (they have, unless a wait ran out) */
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    }
    /* sharded: rows without keys on this rank were announced at the top; the other ranks' records are folded here */
    if (SHARD)
        for (int i = cta; i < n; i += gridDim.x) {
            if (s_prefix[i + 1] != s_prefix[i]) continue;
            for (int hl = 0; hl < G; hl++) {
                const int seg = i * G + hl;
                if (tid < 256) {
                    const int h = (tid >> 5) & 7, d4 = (tid & 31) * 4;
                    shard_fold_args fa;
                    fa.rec0 = a.gathered + ((size_t)seg * 8 + h) * kShardLines; fa.rank_stride = (size_t)n * G * 8 * kShardLines; fa.err = a.err;
                    fa.out = a.out + (size_t)i * a.out_stride + ((size_t)(cache.kv_head_begin + hl) * 8 + h) * HY3A_D + d4;
                    fa.n_ranks = a.n_dest; fa.my_rank = a.my_rank; fa.line_a = 1 + (d4 >> 1); fa.flag = a.shard_round[seg * 8 + h] + 1u; fa.stage = reinterpret_cast<const uint4 *>(s_dyn); fa.h = h; fa.lane = lane;
                    fa.own_m = -INFINITY; fa.own_l = 0.f; fa.own_acc[0] = fa.own_acc[1] = fa.own_acc[2] = fa.own_acc[3] = 0.f;
                    shard_fold<kShardBatch>(fa);
                    __syncwarp();
                    if (d4 == 0) a.shard_round[seg * 8 + h] = fa.flag;
                }
                consumer_sync();
            }
        }
}

/* Merge kernel for cross-GPU partials: grid (n_rows*n_heads), block 32; lane -> 4 dims. */
__global__ void hy3a_merge_kernel(const float *partials, int n_parts, int n_rows, int n_heads, float *out, size_t out_stride) {
    int rh = blockIdx.x, lane = threadIdx.x;
    int row = rh / n_heads, h = rh % n_heads;
    float ms = -INFINITY, ss = 0.f, ov[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s = 0; s < n_parts; s++) {
        const float *p = partials + ((size_t)s * n_rows * n_heads + rh) * HY3A_PARTIAL_FLOATS;
        float pms = p[0], pss = p[1];
        if (pss == 0.f) continue;
        float nm = fmaxf(ms, pms), os = __expf(ms - nm), rs = __expf(pms - nm);
        ss = ss * os + pss * rs;
#pragma unroll
        for (int j = 0; j < 4; j++) ov[j] = ov[j] * os + p[2 + lane * 4 + j] * rs;
        ms = nm;
    }
    float inv = inv_sum(ss);
    *reinterpret_cast<float4 *>(out + (size_t)row * out_stride + (size_t)h * HY3A_D + lane * 4) = make_float4(ov[0] * inv, ov[1] * inv, ov[2] * inv, ov[3] * inv);
}

} /* namespace */

/* a launch's shared memory */
static size_t prefix_bytes(int rows) { return ((size_t)(rows + 1) * sizeof(int) + 127) & ~(size_t)127; }
static size_t ring_bytes(const hy3a_ctx *ctx) { return (size_t)ctx->decode_stages * (ctx->geom.dtype == HY3A_KV_FP16 ? kStageBytes<0> : kStageBytes<2>); }      /* not INT8's */
template <int CL>
static size_t decode_smem(size_t prefix, size_t ring) { return kFixed<CL> + prefix + kBarBytes<CL> + ring; }

template <int DT>
static const void *decode_cluster_fn(int cl) {
    return cl == 2 ? (const void *)hy3a_decode_kernel<DT, true, false, 2> : cl == 4 ? (const void *)hy3a_decode_kernel<DT, true, false, 4> : (const void *)hy3a_decode_kernel<DT, true, false, 8>;
}

cudaError_t hy3a_launch_cluster(hy3a_ctx *ctx, const void *fn, int cl, int clusters, int threads, size_t smem, void **args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cl * clusters); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = ctx->use_pdl ? 2 : 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

/* also sets the kernel's shared-memory limit on the device; 0 where such clusters cannot run */
int hy3a_cluster_cap(const void *fn, int cl, int threads, size_t smem) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64 * cl); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

void hy3a_decode_cluster_init(hy3a_ctx *ctx) {
    const size_t smem = decode_smem<2>(prefix_bytes(1), ring_bytes(ctx));      /* one CTA per SM at any batch: its registers fill more than half */
    for (int i = 1; i < 4; i++) {
        if (ctx->decode_stages < 2) ctx->cl_cap[i] = 0;
        else if (ctx->geom.dtype == HY3A_KV_INT8) ctx->cl_cap[i] = hy3a_decode_umma_cluster_cap(ctx, 1 << i);
        else ctx->cl_cap[i] = hy3a_cluster_cap(ctx->geom.dtype == HY3A_KV_FP16 ? decode_cluster_fn<0>(1 << i) : decode_cluster_fn<2>(1 << i), 1 << i, kThreads + 32, smem);
    }
}

template <int DT>
static cudaError_t launch_decode_dt(hy3a_ctx *ctx, const hy3a_cache_view &cv, const hy3a_batch_view &bv, decode_args &a) {
    const size_t prefix = prefix_bytes(ctx->batch_n);
    dim3 grid(ctx->decode_ctas);
    static bool attr_dev[64][3][3];   /* function attributes are per device: [device ordinal][cache type][variant] */
    bool (*attr_set)[3] = attr_dev[ctx->device & 63];
    a.prefix_bytes = (int)prefix;
    if (a.cluster) {
        a.stages = ctx->decode_stages;
        void *args[3] = {(void *)&cv, (void *)&bv, (void *)&a};
        return hy3a_launch_cluster(ctx, decode_cluster_fn<DT>(a.cluster), a.cluster, ctx->batch_n * ctx->cfg.kv_head_count, kThreads + 32,
                                   decode_smem<2>(prefix, ring_bytes(ctx)), args);
    }
    if (ctx->decode_stages >= 2) {
        a.stages = ctx->decode_stages;
        const size_t smem = decode_smem<0>(prefix, ring_bytes(ctx));
        const bool shard = a.n_dest > 0;
        if (!attr_set[DT][shard ? 2 : 1]) {
            cudaError_t e = shard ? cudaFuncSetAttribute(hy3a_decode_kernel<DT, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax)
                                  : cudaFuncSetAttribute(hy3a_decode_kernel<DT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
            if (e != cudaSuccess) return e;
            attr_set[DT][shard ? 2 : 1] = true;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid; cfg.blockDim = dim3(kThreads + 32); cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr; cfg.numAttrs = ctx->use_pdl ? 1 : 0;
        if (shard) return cudaLaunchKernelEx(&cfg, hy3a_decode_kernel<DT, true, true>, cv, bv, a);
        return cudaLaunchKernelEx(&cfg, hy3a_decode_kernel<DT, true>, cv, bv, a);
    } else {
        a.stages = 0;
        if (!attr_set[DT][0]) {
            cudaError_t e = cudaFuncSetAttribute(hy3a_decode_kernel<DT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
            if (e != cudaSuccess) return e;
            attr_set[DT][0] = true;
        }
        hy3a_decode_kernel<DT, false><<<grid, kThreads, decode_smem<0>(prefix, 0), ctx->stream>>>(cv, bv, a);
    }
    return cudaGetLastError();
}

/* Stages that fit in the ring for a cache type and batch capacity, at most 8; none where two whole pages do not fit (the direct variant). */
int hy3a_decode_ring_capacity(int dtype, int max_batch) {
    const long room = (long)kSmemMax - (long)decode_smem<0>(prefix_bytes(max_batch), 0);
    const int page = hy3a_make_geom(dtype).page_bytes, stage = dtype == HY3A_KV_FP16 ? kStageBytes<0> : page;
    return room < 2l * page ? 0 : (int)std::min(8l, room / stage);
}
static_assert(kRecFloats >= HY3A_PARTIAL_FLOATS && (kRecFloats * 4) % 16 == 0, "a head's record must start on a 16-byte boundary");

/* Folders per segment of the spread fold (0: the last CTA to arrive folds).  It pays off where the epilogue is the cross-GPU
 * exchange (several CTAs store to the peers instead of one); on one GPU the folders only hold their SMs longer, which delays the
 * next launch's CTAs there.  Its folders wait for the other pieces, so every CTA of the grid must be resident.  4 measured best
 * on 8 GPUs (8: 28.8, 4: 27.8, 2: 27.8, 1: 29.2 us per layer). */
static int spread_folders(const hy3a_ctx *ctx) {
    return ctx->shard_slot < 0 || ctx->decode_ctas > ctx->sm_count ? 0 : 4;
}

/* A cluster of CTAs per (row, KV head) instead of the grid, where all clusters run at once: of 2, 4 or 8, the least with which a CTA has
 * few pages (kPagesCta; a larger cluster meets later), unless the grid's even share is so much smaller that its fold is paid for
 * (kPagesFold: the difference of 2 to 3 us in pages).  Nor where a CTA's stream counts for more than the fold, a ring of 4 (INT8) instead of
 * 6 pages with it: INT8 beyond 9 pages for a CTA of 8, or beyond 8 for one of 4 on more than 64 CTAs, unless the grid's CTAs walk 16
 * rows and more to their piece; INT4 beyond 12 pages that are more than 3 above the share.  A captured launch meets other lengths when it is replayed, so there the
 * longest row that the context can hold counts.  Measured back to back, us a layer, grid / clusters of 2 / 4 / 8, 8 KV heads:
 *   INT8   300  7.8  6.4  6.6  7.5    700  8.4  6.6  6.5  7.8   2 500 10.8  9.5  7.4  8.1    8 192 11.2 25.3 15.0 10.9
 *   FP16   300  6.2  5.2  4.8  5.8    700  6.6  6.6  5.8  5.9   2 500 10.4 13.7  9.1  8.3    4 096 10.5 20.2 13.0 10.5
 *   INT4   300  8.6  7.0  6.9  7.7    700  8.7  7.4  7.1  7.8   2 500 11.3 11.1  8.1  8.5   12 000 14.3 29.5 17.6 12.5
 *   INT8, where the stream counts, grid / clusters: 1 row of 9 600 11.69 / 11.78, 3 rows of 5 000 12.91 / 13.02, 3 of 8 000 15.58 / 17.81,
 *   4 rows up to 5 000 12.37 / 13.95; 30 rows of 6 000 with 1 head clusters win by 12 %.  INT4: 1 of 14 000 13.60 / 13.83, 4 up to 8 000 14.70 / 15.96
 *   9 rows of 200 / 2 500, clusters of 2: INT8 12.8 -> 10.4 / 17.0 -> 14.9, FP16 10.5 -> 7.6 / 22.0 -> 18.9, INT4 12.4 -> 9.8 / 17.4 -> 14.0
 * The lines were drawn before the fold ran per head and one warp planned, which gave the grid 1 to 2 us and the clusters 0.1 to 0.5.  For 1 to 4
 * rows they still hold (66 shapes, grid / as the rule has it): INT8 1 000 9.0 / 7.4, 4 096 11.0 / 9.0, 9 000 12.0 / 11.8; FP16 1 000 6.7 / 5.9,
 * 3 500 9.5 / 8.5; INT4 2 500 10.1 / 7.7, 9 000 11.0 / 11.1, 12 000 12.5 / 11.6.  Of 96 shapes of 9 to 64 ragged rows, 1 to 8 heads and up to
 * 1 000 to 12 000 tokens, the rule takes what is within 3 % of the best in 74.  It takes clusters that the grid beats by 5 to 14 % in 5, all INT4 up
 * to 3 000 and 6 000 (9 rows x 4 heads 10.3 / 11.7, 32 x 1 11.2 / 12.6), and the grid where clusters win, because the grid's CTAs get more
 * than the even share that the rule compares with (INT8 and more than 32 rows have no even pieces): INT8 up to 3 000, 16 rows x 4 heads
 * 20.5 / 13.3, 32 x 2 19.4 / 13.3, 64 x 1 20.5 / 13.5, up to 6 000 24.6 / 19.7; 64 x 1 FP16 up to 3 000 18.5 / 15.3, INT4 up to 6 000 22.2 / 16.5 */
static int cluster_size(const hy3a_ctx *ctx, int most, long long total) {
    static const int kPagesCta[3] = {1, 5, 4}, kPagesFold[3] = {2, 5, 8};      /* FP16, INT8, INT4 */
    const int dt = ctx->geom.dtype, segs = ctx->batch_n * ctx->cfg.kv_head_count;
    if (most < 2 || segs > ctx->cl_cap[1]) return 0;
    /* a ring that a context of very large batches has sized to the last byte leaves no room for the landing zone */
    if (dt != HY3A_KV_INT8 && decode_smem<2>(prefix_bytes(ctx->batch_n), ring_bytes(ctx)) > (size_t)kSmemMax) return 0;
    int i = 1;
    while (i < 3 && ((most - 1) >> i) + 1 > kPagesCta[dt] && segs <= ctx->cl_cap[i + 1]) i++;
    const long long share = (total * ctx->cfg.kv_head_count + ctx->decode_ctas - 1) / ctx->decode_ctas;
    const int pages = ((most - 1) >> i) + 1;      /* of the longest row, a CTA */
    if (dt == HY3A_KV_INT8 && (i == 3 ? pages > 9 : i == 2 && pages > 8 && segs > 16 && ctx->batch_n < 16)) return 0;
    if (dt == HY3A_KV_INT4 && i > 1 && pages > 12 && pages > share + 3) return 0;
    return pages <= share + kPagesFold[dt] ? 1 << i : 0;
}
static int decode_cluster(const hy3a_ctx *ctx) {
    if ((ctx->shard_slot >= 0 && ctx->shard_world > 1) || ctx->decode_ctas < ctx->sm_count || ctx->no_clusters) return 0;      /* a world of one has nothing to exchange */
    const int cl = cluster_size(ctx, ctx->batch_pages, ctx->batch_pages_all);
    if (!cl) return 0;
    if (!hy3a_capturing(ctx)) return cl;
    return cluster_size(ctx, ctx->cfg.max_blocks_per_seq, (long long)ctx->cfg.max_blocks_per_seq * ctx->batch_n);
}

extern "C" int hy3a_decode_cluster(hy3a_ctx *ctx) {
    if (!ctx) return HY3A_EINVAL;
    if (ctx->batch_n < 1) return hy3a_fail(ctx, HY3A_ESTATE, "decode_cluster: no batch set (call hy3a_batch_set first)");
    const int cl = decode_cluster(ctx);
    return cl ? cl : 1;
}

int hy3a_launch_decode(hy3a_ctx *ctx, int layer, const float *q, size_t q_stride, float *out, size_t out_stride, float *partials,
                       const hy3a_step_inputs *step) {
    decode_args a;
    memset(&a, 0, sizeof(a));
    a.q = q; a.q_stride = q_stride; a.out = out; a.out_stride = out_stride; a.user_partials = partials;
    a.scratch = ctx->d_partials; a.counters = ctx->d_counters; a.n_counters = ctx->cfg.max_batch * ctx->cfg.kv_head_count; a.err = ctx->d_err; a.layer = layer;
    a.spread = spread_folders(ctx);
    a.wait_first = hy3a_take_fresh(ctx);
    a.early_prefetch = ctx->use_pdl && !ctx->bulk_write_pending;
    a.cluster = decode_cluster(ctx);
    if (ctx->shard_slot >= 0) {   /* set by hy3a_decode_step_sharded around this call */
        const int W = ctx->shard_world, slot = ctx->shard_slot;
        const size_t n_seg = (size_t)ctx->shard_rows * ctx->cfg.kv_head_count;
        const size_t slice = n_seg * 8 * (HY3A_PARTIAL_FLOATS / 2);    /* 16-byte lines per rank and slot */
        a.n_dest = W; a.my_rank = ctx->shard_rank;
        for (int r = 0; r < W; r++) a.dest[r] = reinterpret_cast<uint4 *>(ctx->shard_peer[r]) + ((size_t)slot * W + ctx->shard_rank) * slice;
        a.gathered = reinterpret_cast<const uint4 *>(ctx->shard_local) + (size_t)slot * W * slice;
        a.shard_round = reinterpret_cast<unsigned *>(ctx->shard_local + ctx->shard_state_off) + (size_t)slot * n_seg * 8;
    }
    if (step) {
        a.fused = 1;
        a.q_in = step->q_in; a.k_in = step->k_in; a.v_in = step->v_in;
        a.qi_stride = step->q_stride; a.ki_stride = step->k_stride; a.vi_stride = step->v_stride;
        a.q_out = step->q_out; a.q_out_stride = step->q_out_stride;
        a.norm_w = ctx->d_norm_w + (size_t)layer * 2 * HY3A_D; a.eps = ctx->cfg.rms_eps; a.rope = ctx->rope;
    }
    hy3a_cache_view cv = hy3a_view(ctx);
    hy3a_batch_view bv = hy3a_bview(ctx);
    cudaError_t e;
    switch (ctx->geom.dtype) {
        case 0: e = launch_decode_dt<0>(ctx, cv, bv, a); break;
        case 1: e = hy3a_launch_decode_umma(ctx, cv, bv, a); break;
        default: e = launch_decode_dt<2>(ctx, cv, bv, a); break;
    }
    ctx->launches++;
    ctx->bulk_write_pending = 0;   /* the kernel after this one only has this one to stay clear of */
    if (e != cudaSuccess) return hy3a_fail(ctx, HY3A_ECUDA, "decode launch: %s", cudaGetErrorString(e));
    return HY3A_OK;
}

/* ---- decode without any allocation ---------------------------------------------------------
 * Scratch for hy3a_decode_noalloc: the records and arrival counters of the cross-CTA merge live in
 * this file-scope device array instead of buffers the context allocated.  Every GPU that loads the
 * library holds these 2.4 MB until the process exits.  Layout: [kNoAllocRecords][8][132] floats of
 * records, then the counters (HY3A_COUNTERS) of the segments.                                               */
constexpr int kNoAllocRows = 64;                                   /* most (batch row, KV head) segments per call */
constexpr int kNoAllocRecords = 512 + kNoAllocRows;                /* one per CTA of the largest grid + one per segment */
constexpr size_t kNoAllocRecordBytes = (size_t)kNoAllocRecords * 8 * kRecFloats * sizeof(float);
constexpr size_t kNoAllocCounterBytes = HY3A_COUNTERS(kNoAllocRows) * sizeof(unsigned);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocRecordBytes + kNoAllocCounterBytes];
static unsigned char *g_noalloc_ptr[64];                           /* device address of the array, per device ordinal */

extern "C" int hy3a_decode_noalloc(hy3a_ctx *ctx, int layer, const float *q, size_t q_stride, float *out, size_t out_stride) {
    if (!ctx) return HY3A_EINVAL;
    if (layer < 0 || layer >= ctx->cfg.n_layers) return hy3a_fail(ctx, HY3A_EINVAL, "decode_noalloc: layer %d out of range", layer);
    if (ctx->batch_n < 1) return hy3a_fail(ctx, HY3A_ESTATE, "decode_noalloc: no batch set (call hy3a_batch_set first)");
    if (!q || !out || (((uintptr_t)q | (uintptr_t)out) & 15) || ((q_stride | out_stride) & 3))
        return hy3a_fail(ctx, HY3A_EINVAL, "decode_noalloc: q and out must be non-NULL, 16-byte aligned, strides multiples of 4");
    if (ctx->batch_n * ctx->cfg.kv_head_count > kNoAllocRows)
        return hy3a_fail(ctx, HY3A_EINVAL, "decode_noalloc: %d batch rows x %d KV heads exceed the built-in scratch (%d segments); use hy3a_decode",
                         ctx->batch_n, ctx->cfg.kv_head_count, kNoAllocRows);
    if (ctx->decode_ctas > 512) return hy3a_fail(ctx, HY3A_EINVAL, "decode_noalloc: grid of %d CTAs exceeds the built-in scratch", ctx->decode_ctas);
    if (ctx->device < 0 || ctx->device >= 64) return hy3a_fail(ctx, HY3A_EINVAL, "decode_noalloc: device ordinal %d not supported", ctx->device);
    {   /* the launch below goes to the current device: it must be the context's */
        int cur = -1;
        HY3A_CUDA(ctx, cudaGetDevice(&cur));
        if (cur != ctx->device)
            return hy3a_fail(ctx, HY3A_ESTATE, "decode_noalloc: the context lives on device %d but device %d is current (cudaSetDevice first)", ctx->device, cur);
    }
    if (!g_noalloc_ptr[ctx->device]) {
        /* one-time set-up on this device (it is current): in host code the array's name is only a handle, the
         * kernel needs the device address                                                                  */
        void *p = NULL;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) return hy3a_fail(ctx, HY3A_ECUDA, "decode_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        g_noalloc_ptr[ctx->device] = (unsigned char *)p;
    }
    unsigned char *scratch = g_noalloc_ptr[ctx->device];
    /* the arrival counters must start at zero; a call that was cut short may have left some behind */
    HY3A_CUDA(ctx, cudaMemsetAsync(scratch + kNoAllocRecordBytes, 0, kNoAllocCounterBytes, ctx->stream));
    decode_args a;
    memset(&a, 0, sizeof(a));
    a.q = q; a.q_stride = q_stride; a.out = out; a.out_stride = out_stride;
    a.scratch = reinterpret_cast<float *>(scratch);
    a.counters = reinterpret_cast<unsigned *>(scratch + kNoAllocRecordBytes);
    a.n_counters = kNoAllocRows;
    a.err = ctx->d_err; a.layer = layer;
    a.wait_first = hy3a_take_fresh(ctx);
    a.early_prefetch = 0;
    hy3a_cache_view cv = hy3a_view(ctx);
    hy3a_batch_view bv = hy3a_bview(ctx);
    cudaError_t e;
    switch (ctx->geom.dtype) {
        case 0: e = launch_decode_dt<0>(ctx, cv, bv, a); break;
        case 1: e = hy3a_launch_decode_umma(ctx, cv, bv, a); break;
        default: e = launch_decode_dt<2>(ctx, cv, bv, a); break;
    }
    ctx->launches++;
    ctx->bulk_write_pending = 0;
    if (e != cudaSuccess) return hy3a_fail(ctx, HY3A_ECUDA, "decode_noalloc launch: %s", cudaGetErrorString(e));
    return HY3A_OK;
}


int hy3a_launch_merge(hy3a_ctx *ctx, const float *partials, int n_parts, int n_rows, int n_heads, float *out, size_t out_stride) {
    hy3a_merge_kernel<<<n_rows * n_heads, 32, 0, ctx->stream>>>(partials, n_parts, n_rows, n_heads, out, out_stride);
    ctx->launches++;
    HY3A_CUDA(ctx, cudaGetLastError());
    return HY3A_OK;
}
