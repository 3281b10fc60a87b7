/*
 * prefill.cu -- causal chunk attention on 5th-generation tensor cores (tcgen05 + TMEM + TMA).
 *
 * Replaces prefill_attn_int8/int4_kernel (hy3_gpu.cu:383-447), which walks the keys serially with
 * one warp per (query head, 16-query tile) on CUDA cores.  Semantics kept: query i of the chunk has
 * global index base+i and attends keys [0, base+i]; the chunk's own K/V were appended first, so
 * queries see the cache's (quantised) K/V also for their own chunk (hy3_gpu.cu:823-832).
 *
 * Two kernels per (layer, chunk):
 *   1. hy3a_kv_to_f16_kernel<DT>: converts the sequence's pages of this layer into dense fp16 operands,
 *      dequantising INT8/INT4 (value = code * fp16 scale, hy3_gpu.cu:206-215): K as [head][token][128]
 *      (d contiguous) and V TRANSPOSED as [head][128][token] (tokens contiguous), so that both are
 *      K-major operands for the tensor cores.  The operands of a layer are kept across chunks (the
 *      context's per-layer mirrors), so a chunk only converts the pages it appended.
 *   2. hy3a_prefill_kernel: one CTA per (32 query tokens x the 8 query heads of one KV head) = two
 *      128-row Q tiles (GQA packing: the 8 heads share every K/V tile); where blocks of 16 tokens fit on the device at once, in
 *      clusters or uncut, one tile.  Warp-specialised:
 *        TMA producer: Q once, then 64-key K / V tiles into 4-stage rings (cp.async.bulk.tensor,
 *                 128-byte swizzle, mbarrier transaction counts)
 *        MMA issuers (one warp per Q tile, one elected lane): S = Q.K^T (M=128, N=64, K=16) and
 *                 O += P.V (N=128) with tcgen05.mma.cta_group::1.kind::f16, accumulators in TMEM
 *                 (per Q tile two S buffers of 64 columns and O of 128); tcgen05.commit signals mbarriers
 *        softmax warps, one thread per row: tcgen05.ld the row of S, online softmax in base 2 with a
 *                 lazily updated reference max, P as packed fp16 over the S columns (tcgen05.st; P.V
 *                 reads its A operand from tensor memory), conditional rescale of O in TMEM;
 *                 epilogue O / l -> fp32 output.
 *      Causal masking only touches the tiles that cross the diagonal.
 *
 * Every wait is bounded; a wait that runs out raises a CTA-wide abort flag, records a code in the
 * context's error word, lets all warps fall through to the end, and TMEM is always released.
 *
 * Roofline: tensor (dense fp16).  Algorithmic FLOPs = 4 * 128 * 64 * sum over queries of (pos+1).
 */
#include <cuda.h>
#include <cuda_fp16.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "ctx.h"

namespace {

constexpr int kQTok = 16;            /* query tokens per CTA (x 8 heads = 128 rows) */
constexpr int kTileBytes = 128 * 128 * 2;   /* one 128x128 fp16 operand tile = two 16 KB swizzled sub-tiles */
constexpr float kScaleLog2 = 0.08838834764831845f * 1.4426950408889634f;   /* 1/sqrt(128) * log2(e) */
constexpr float kPfThreshold = 8.f;

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
/* bounded wait, see the header comment: mbarrier.try_wait suspends the thread until the phase completes or the hint elapses,
 * so the waiter wakes within tens of ns of the arrival */
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
        if (i >= (1u << 13) && t1 - t0 > 500000000ull) break;   /* both many polls and half a second: the timer can step */
    }
    *abort_flag = 1;
    if (atomicCAS(err, 0u, 2u) == 0u) err[1] = where;
    return false;
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap *map, unsigned bar, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
/* shared-memory matrix descriptor: K-major, 128-byte swizzle; 8-row groups 1024 B apart (SBO), LBO = 1 (unused
 * for swizzled K-major), descriptor version 1 (Blackwell), layout type 2 = SWIZZLE_128B                       */
__device__ __forceinline__ unsigned long long make_desc(unsigned saddr) {
    return (unsigned long long)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
/* instruction descriptor: D = f32 (bit 4), A = B = f16 (0), both K-major, N = 128 (>>3 at bit 17), M = 128 (>>4 at bit 24) */
constexpr unsigned kIdesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
/* 32 columns of the warp's lanes; the registers are valid after tmem_ld_wait (several loads can be in flight before it) */
__device__ __forceinline__ void tmem_ld32_nowait(unsigned taddr, unsigned *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}
/* waits for all loads of the thread; the operands make every use of the registers depend on it */
__device__ __forceinline__ void tmem_ld_wait(unsigned *r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]) :: "memory");
}
__device__ __forceinline__ void tmem_st32(unsigned taddr, const unsigned (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}
/* The MMA issuers run in uniform control flow (the operands are then computed in the uniform data path the instruction
 * reads them from) and one lane, elected once per walk, issues: `lead` is 1 in that lane. */
__device__ __forceinline__ unsigned elect_one() {
    unsigned p;
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n selp.u32 %0, 1, 0, e;\n}" : "=r"(p));
    return p;
}
__device__ __forceinline__ void umma_f16_ta_lead(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned accumulate, unsigned lead) {
    asm volatile("{\n .reg .pred p, e;\n setp.ne.b32 e, %5, 0;\n setp.ne.b32 p, %4, 0;\n @e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(kIdesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ __forceinline__ void umma_commit_lead(unsigned bar, unsigned lead) {
    asm volatile("{\n .reg .pred e;\n setp.ne.b32 e, %1, 0;\n @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar), "r"(lead) : "memory");
}
__device__ __forceinline__ float fmax3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }
__device__ __forceinline__ float ex2f(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ unsigned pack_h2(float lo, float hi) { unsigned r; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo)); return r; }

/* ---- packed fp32 pairs (one instruction for two values) */
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 x, y, z, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n fma.rn.f32x2 w, x, y, z;\n mov.b64 {%0, %1}, w;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
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
__device__ __forceinline__ float2 splat(float a) { return make_float2(a, a); }
/* maximum that keeps a NaN operand (fmaxf returns the other one) */
__device__ __forceinline__ float fmax_nan(float a, float b) { float r; asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b)); return r; }
/* 2^t of a pair on the FMA pipe (the exponential unit takes 16 values per clock and SM, which the softmax of two tiles fills):
 * t = n + f, n = round(t), 2^f on [-1/2, 1/2] by the Taylor polynomial of e^(f ln 2) of degree 6 (relative error up to 1.6e-7 in
 * fp64 with these constants, 2.2e-7 in fp32 steps; the first missing term is (ln 2 / 2)^7 / 7! = 1.2e-7), times 2^n, whose bits are put together from n.  t is
 * clamped at -126 (masked keys: 2^-126 instead of 0, which is 0 in fp16 and nothing beside a denominator >= 2^-8).  A NaN (a NaN
 * score, or a row whose maximum is +inf) stays one, as in ex2.approx: the clamp keeps it, and 2^n is a factor and not added to
 * the exponent field, where it would leave a finite pattern. */
__device__ __forceinline__ float2 ex2_fma(float2 t) {
    const float magic = 12582912.f;    /* 1.5 * 2^23: adding it rounds to an integer and leaves it in the low mantissa bits */
    t.x = fmax_nan(t.x, -126.f); t.y = fmax_nan(t.y, -126.f);
    const float2 z = add2(t, splat(magic)), n = add2(z, splat(-magic)), f = fma2(n, splat(-1.f), t);
    float2 p = fma2(splat(1.5403530e-4f), f, splat(1.3333558e-3f));
    p = fma2(p, f, splat(9.6181291e-3f));
    p = fma2(p, f, splat(5.5504109e-2f));
    p = fma2(p, f, splat(2.4022651e-1f));
    p = fma2(p, f, splat(6.9314718e-1f));
    p = fma2(p, f, splat(1.f));
    return mul2(p, make_float2(__uint_as_float((__float_as_uint(z.x) << 23) + 0x3f800000u), __uint_as_float((__float_as_uint(z.y) << 23) + 0x3f800000u)));
}
__device__ __forceinline__ float row_max(const unsigned (&v)[64]) {
    float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      /* four independent chains */
#pragma unroll
    for (int i = 0; i < 64; i += 2) mx[(i >> 1) & 3] = fmax3(mx[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
    return fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
}
/* Turns on the exponential unit: tile A and tile B compute their exponentials alternately.  Left alone the two tiles fall into
 * step -- both wait, load and reduce at the same time and then share the unit at half speed (1 250 clocks for 64 columns of both,
 * in a period of 1 985 clocks per step); with turns one tile's exponentials run under the other's waits: 1 560-1 620 clocks. */
__device__ __forceinline__ void turn_wait(int x) { asm volatile("bar.sync %0, 256;" ::"r"(1 + x) : "memory"); }
__device__ __forceinline__ void turn_pass(int x) { asm volatile("bar.arrive %0, 256;" ::"r"(2 - x) : "memory"); }
__device__ __forceinline__ float ex2v(float x) { float r; asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
/* P = 2^(s * scale - m) of a row's 64 scores as packed fp16 pairs; returns the (pairwise) sum of the unrounded values (the fp16
 * rounding of P is a zero-mean 2^-12 relative error per term, far below the tolerance).  One pair in eight goes through the FMA
 * pipe: 512 tokens behind 4 096 take 73.0 us with none, 70.8 with one, 73.0 with two (the FMA form costs issue slots that the
 * waiting tile's maximum wants); 2 048 fresh tokens 82.1 / 81.6 / 82.3. */
template <bool CUT, bool TURNS>
__device__ __forceinline__ float2 softmax_exp(const unsigned (&v)[64], float m, unsigned (&pk)[32], int x, bool pass) {
    /* m == -inf: every key of the row so far is masked; the arguments are then -inf, not NaN, and all P are 0 */
    const float2 sc = splat(kScaleLog2), nm = splat(CUT && m == -INFINITY ? 0.f : -m);
    float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, t[32];
#pragma unroll
    for (int i = 0; i < 32; i++) t[i] = fma2(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sc, nm);
    if (TURNS) turn_wait(x);
#pragma unroll
    for (int i = 0; i < 32; i++) {
        if ((i & 7) == 7) t[i] = ex2_fma(t[i]);
        else { t[i].x = ex2v(t[i].x); t[i].y = ex2v(t[i].y); }
    }
    if (TURNS && pass) turn_pass(x);
#pragma unroll
    for (int i = 0; i < 32; i++) {
        pk[i] = pack_h2(t[i].x, t[i].y);
        ls[i & 1] = add2(ls[i & 1], t[i]);
    }
    return add2(ls[0], ls[1]);
}

/* ---- pass 1: pages -> dense fp16 K [head][tok][128] and V^T [head][128][tok] ------------------- */
template <int DT>
__global__ void __launch_bounds__(256) hy3a_kv_to_f16_kernel(hy3a_cache_view cache, int layer, int seq, int pg0, int ntok, int tok_stride, __half *ws_k, __half *ws_vt) {
    const hy3a_geom g = hy3a_make_geom(DT);
    const int pg = pg0 + blockIdx.x, hl = blockIdx.y, tid = threadIdx.x;
    /* programmatic dependent launch: the appended rows must be complete; the attention kernel may set itself up */
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int block = cache.block_table[(size_t)seq * cache.max_blocks_per_seq + pg];
    const uint8_t *page = cache.pool + hy3a_page_index(cache, block, layer, hl) * (size_t)cache.page_bytes;
    const __half *ks = reinterpret_cast<const __half *>(page + g.ks_off), *vs = reinterpret_cast<const __half *>(page + g.vs_off);
    /* one block converts 32 tokens of the page (blockIdx.z): short dependent chains and 4x the blocks, because a chunk only
     * brings a handful of new pages and the attention kernel waits for this one */
    const int tq = blockIdx.z * 32;
    /* K: 32 tokens x 16 groups of 8 dims */
#pragma unroll
    for (int idx = tid; idx < 32 * 16; idx += 256) {
        const int tok = tq + (idx >> 4), d = (idx & 15) * 8, t = pg * 128 + tok;
        uint4 o = make_uint4(0, 0, 0, 0);
        if (t < ntok) {
            if (DT == 0) {
                o = *reinterpret_cast<const uint4 *>(page + hy3a_k_dim_off<0>(tok, d));
            } else {
                const float s = __half2float(ks[tok]);
                float f[8];
                if (DT == 1) {
                    const uint2 w = *reinterpret_cast<const uint2 *>(page + hy3a_k_dim_off<1>(tok, d));
                    const unsigned ww[2] = {w.x, w.y};
#pragma unroll
                    for (int i = 0; i < 8; i++) f[i] = (float)(signed char)((ww[i >> 2] >> (8 * (i & 3))) & 0xFF) * s;
                } else {
                    const unsigned w = *reinterpret_cast<const unsigned *>(page + hy3a_k_dim_off<2>(tok, d));
#pragma unroll
                    for (int i = 0; i < 8; i++) { int n = (w >> (4 * i)) & 0xF; f[i] = (float)(n > 7 ? n - 16 : n) * s; }
                }
                __half2 h0 = __floats2half2_rn(f[0], f[1]), h1 = __floats2half2_rn(f[2], f[3]), h2 = __floats2half2_rn(f[4], f[5]), h3 = __floats2half2_rn(f[6], f[7]);
                o = make_uint4(*reinterpret_cast<unsigned *>(&h0), *reinterpret_cast<unsigned *>(&h1), *reinterpret_cast<unsigned *>(&h2), *reinterpret_cast<unsigned *>(&h3));
            }
        }
        *reinterpret_cast<uint4 *>(ws_k + ((size_t)hl * tok_stride + t) * HY3A_D + d) = o;
    }
    /* V^T: thread = (dim, 16 of the block's tokens); 8 consecutive tokens per 16-byte store */
    const int d = tid & 127, th = tid >> 7;
#pragma unroll
    for (int t8 = 0; t8 < 2; t8++) {
        __half hv[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int tok = tq + th * 16 + t8 * 8 + i, t = pg * 128 + tok;
            float v = 0.f;
            if (t < ntok) {
                if (DT == 0) {
                    v = __half2float(*reinterpret_cast<const __half *>(page + g.v_off + hy3a_v16_dim_off(tok, d)));
                } else if (DT == 1) {
                    v = (float)(signed char)page[g.v_off + hy3a_vt_off(d, tok)] * __half2float(vs[tok]);
                } else {
                    const int b = page[g.v_off + hy3a_v_unit_off<2>(tok, d & ~3) + ((d & 3) >> 1)];
                    v = (float)(((b >> ((d & 1) * 4)) & 0xF) - 8) * __half2float(vs[tok]);
                }
            }
            hv[i] = __float2half_rn(v);
        }
        *reinterpret_cast<uint4 *>(ws_vt + ((size_t)hl * HY3A_D + d) * tok_stride + pg * 128 + tq + th * 16 + t8 * 8) = *reinterpret_cast<uint4 *>(hv);
    }
}

struct prefill_args {
    float *out;
    size_t out_stride;
    int base, nq, kv_head_begin, kv_heads, entries, group;   /* entries per head (blocks, or pieces of cut blocks), dealt to the heads in groups */
    unsigned *err;
    float *rec;             /* records of cut blocks: [slot][8 warps][kRecWarp] */
    unsigned *cnt;          /* arrivals: [slot][8 warps], left at zero */
};
/* record of one softmax warp: O as [32 column quads][32 rows] float4 (a warp stores 512 contiguous bytes), then {m, l} per row */
constexpr int kRecWarp = 32 * 128 + 64;
static_assert(8 * kRecWarp * 4 == HY3A_PF_REC_BYTES, "record size");

/* ---- pass 2: the attention kernel -------------------------------------------------------------------------------------
 * One CTA = 32 query tokens x the 8 query heads of one KV head = two 128-row Q tiles A and B that share every K/V tile
 * (GQA packing); P lives in tensor memory.  A K/V tile is 64 keys, so that each Q tile has TWO S buffers (2 x 64 TMEM columns) beside its O (128
 * columns): 2 x 256 = 512 columns.  S_x(j+2) is issued right behind P_x(j).V_j into the buffer P_x(j) lives in, i.e. the
 * scores of a step are computed while the softmax of the step before runs, and the loop
 *      S ready -> softmax -> P -> P.V -> next S
 * falls apart into a softmax chain (one thread per row, 64 columns
 * per step, no exchange between threads) and an MMA chain that only meet at the P and S barriers.  The softmax warps
 * wait for P.V only when a row's reference maximum moved (lazy rescale of O) and at the end.
 * Warps 0-3 / 4-7: softmax of tile A / B; warp 8: TMA producer (4-stage rings of 16 KB K and V tiles); warps 9 / 10:
 * MMA issuers of tile A / B, each in uniform control flow with one lane elected once (one thread issues an MMA every
 * ~26 ns at best, which a single issuer for both tiles would be bound by).                                       */
constexpr int kQTok2 = HY3A_PF_QTOK;           /* query tokens per CTA = two tiles of kQTok */
constexpr int kKeys3 = HY3A_PF_KEYS;
/* Neighbouring CTAs (the two SMs of a TPC, a GPC) should walk the same head: they ask L2 for the same K/V lines at the same time.  So
 * a grid that is resident at once goes head by head, and a larger one in groups of 8 blocks per head, the groups in descending
 * order of length, because the longest blocks must not start last: 2 048 fresh tokens 94.5 us in ascending order, 81.6 in this.
 * The size of the group matters little (operands from HBM, heads alternating every 1 / 2 / 4 / 8 / 16 blocks): 953 tokens behind
 * 2 048 take 82.0 / 82.1 / 81.8 / 80.8 / 82.7 us, 2 048 fresh ones 80.5 / 80.7 / 81.1 / 81.6 / 83.3; 512 behind 4 096, resident at
 * once, 70.8 head by head and 72.3 alternating. */
constexpr int kGroup = 8;
constexpr int kK3Bytes = kKeys3 * 128 * 2;      /* one K tile = two sub-tiles [64 keys][64 dims]; one V^T tile = [128 dims][64 keys] */
constexpr int kSt3 = 4;                         /* ring stages */
constexpr int kPf3Threads = 352;
constexpr int kOff3Q = 0, kOff3K = kOff3Q + 2 * kTileBytes, kOff3V = kOff3K + kSt3 * kK3Bytes, kOff3Bar = kOff3V + kSt3 * kK3Bytes;
constexpr int kPf3Smem = kOff3Bar + 512 + 1024;
/* K0F, K0E [2]: the first two K tiles (loaded / consumed); DF, DE [4 stages]: step j's data = V_j and K_(j+2) (loaded /
 * consumed); SF, P [tile][buffer]; O [tile][last but one, last]: each completes once */
enum { B3_Q = 0, B3_K0F = 1, B3_K0E = 3, B3_DF = 5, B3_DE = 9, B3_SF = 13, B3_P = 17, B3_O = 21 };
constexpr unsigned kIdescN64 = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_f16_n64_lead(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned accumulate, unsigned lead) {
    asm volatile("{\n .reg .pred p, e;\n setp.ne.b32 e, %5, 0;\n setp.ne.b32 p, %4, 0;\n @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(kIdescN64), "r"(accumulate), "r"(lead) : "memory");
}
/* where a CTA's piece lies; an uncut block is one piece from step 0 */
struct pf_where { int hl, qblk, j0, ntiles, piece, np, rec0; };
/* CTA -> (entry, head) */
__device__ __forceinline__ void entry_of(const prefill_args &a, int &ent, int &hl) {
    const int per = a.group * a.kv_heads, grp = blockIdx.x / per, in = blockIdx.x - grp * per, gsz = min(a.group, a.entries - grp * a.group);
    hl = in / gsz;
    ent = grp * a.group + in - hl * gsz;
}
/* blocks whole / cut, records through memory / cut over the CTAs of a cluster */
enum { PF_WHOLE = 0, PF_CUT = 1, PF_CLUSTER = 2 };
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_addr(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster16(unsigned addr, float a, float b, float c, float d) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void st_cluster8(unsigned addr, float a, float b) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
/* TILES: query tiles of a CTA.  One where blocks of 16 tokens fit at once as well (hy3a_launch_prefill; never where blocks are cut): a block then
 * has half the softmax and half the exchange of a cluster, and none for a second tile without tokens; warps 4-7 and 10 have nothing to do.  us a layer with its
 * append, two tiles / one: 45 tokens behind 1 001 19.7 / 15.2, 64 behind 8 192 43.6 / 34.2, 16 behind 500 13.9 / 12.7; uncut,
 * 30 behind 300 16.7 / 12.8, 256 fresh ones 15.4 / 13.0. */
template <int MODE, int CL, int TILES = 2>
__device__ __forceinline__ void prefill_body(const CUtensorMap &tm_q, const CUtensorMap &tm_k, const CUtensorMap &tm_v, const prefill_args &a, const pf_where &w) {
    extern __shared__ uint8_t s_raw[];
    uint8_t *sm = s_raw + ((1024u - (smem_u32(s_raw) & 1023u)) & 1023u);
    const unsigned sbase = smem_u32(sm);
    const unsigned bar0 = sbase + kOff3Bar;
    volatile unsigned *s_tmem = reinterpret_cast<volatile unsigned *>(sm + kOff3Bar + 256);
    volatile int *s_abort = reinterpret_cast<volatile int *>(sm + kOff3Bar + 260);
#define BAR(i) (bar0 + 8u * (unsigned)(i))

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr bool CUT = MODE != PF_WHOLE;
    const int hl = w.hl, qblk = w.qblk, ntiles = w.ntiles, j0 = CUT ? w.j0 : 0, np = MODE == PF_CUT ? w.np : 1, piece = w.piece, rec0 = w.rec0;
    constexpr int kRows = 128 * TILES;
    const int q0 = qblk * kQTok * TILES;

    if (tid == 0) {
        *s_abort = 0;
        mbar_init(BAR(B3_Q), 1);
        for (int i = 0; i < 2; i++) { mbar_init(BAR(B3_K0F + i), 1); mbar_init(BAR(B3_K0E + i), TILES); }
        for (int i = 0; i < kSt3; i++) { mbar_init(BAR(B3_DF + i), 1); mbar_init(BAR(B3_DE + i), TILES); }   /* K0E, DE: one commit per issuer */
        for (int i = 0; i < 4; i++) { mbar_init(BAR(B3_SF + i), 1); mbar_init(BAR(B3_P + i), 4); }   /* P: one arrival per softmax warp of the tile */
        for (int i = 0; i < 4; i++) mbar_init(BAR(B3_O + i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8 && lane < 3) {   /* the descriptors' first use is then no miss behind the wait for the preceding kernel */
        const CUtensorMap *m = lane == 0 ? &tm_q : (lane == 1 ? &tm_k : &tm_v);
        asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
    }
    if (warp == 0) {   /* one warp allocates all 512 TMEM columns (1 CTA per SM) */
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kOff3Bar + 256), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = *s_tmem;
    /* tile x: S buffers at columns 128x and 128x + 64 (P over the first 32 columns of its S), O at columns 256 + 128x */

    if (warp == 8) {
        /* ===================== TMA producer ===================== */
        if (lane == 0) {
            /* programmatic dependent launch: everything above ran beside the tail of the conversion kernel; the
             * operands are complete from here on (all global reads of this CTA follow this thread's copies) */
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            mbar_expect_tx(BAR(B3_Q), TILES * kTileBytes);
            for (int x = 0; x < TILES; x++) {
                tma_load_3d(sbase + kOff3Q + x * kTileBytes, &tm_q, BAR(B3_Q), 0, (a.kv_head_begin + hl) * 8, q0 + x * kQTok);
                tma_load_3d(sbase + kOff3Q + x * kTileBytes + 16384, &tm_q, BAR(B3_Q), 64, (a.kv_head_begin + hl) * 8, q0 + x * kQTok);
            }
            /* the first two K tiles, then per step j one transaction: V_j and K_(j+2) (S_(j+2) is issued behind P_j.V_j,
             * so the issuers need both at the same time and wait for them once) */
            for (int j = 0; j < 2 && j < ntiles; j++) {
                mbar_expect_tx(BAR(B3_K0F + j), kK3Bytes);
                tma_load_3d(sbase + kOff3K + j * kK3Bytes, &tm_k, BAR(B3_K0F + j), 0, (j0 + j) * kKeys3, hl);
                tma_load_3d(sbase + kOff3K + j * kK3Bytes + 8192, &tm_k, BAR(B3_K0F + j), 64, (j0 + j) * kKeys3, hl);
            }
            for (int j = 0; j < ntiles; j++) {
                const int st = j & (kSt3 - 1), j2 = j + 2, st2 = j2 & (kSt3 - 1); const unsigned ph = (unsigned)(j / kSt3) & 1u;
                /* V slot st held V_(j-4), K slot st2 held K_(j-2): both were released by step j-4 -- except K_0 and K_1, which
                 * the issuers release on barriers of their own */
                if (!mbar_wait_blocking(BAR(B3_DE + st), ph ^ 1u, s_abort, a.err, 10u)) break;
                if ((j == 2 || j == 3) && j2 < ntiles && !mbar_wait_blocking(BAR(B3_K0E + j - 2), 0u, s_abort, a.err, 11u)) break;
                mbar_expect_tx(BAR(B3_DF + st), j2 < ntiles ? 2 * kK3Bytes : kK3Bytes);
                tma_load_3d(sbase + kOff3V + st * kK3Bytes, &tm_v, BAR(B3_DF + st), (j0 + j) * kKeys3, 0, hl);
                if (j2 < ntiles) {
                    tma_load_3d(sbase + kOff3K + st2 * kK3Bytes, &tm_k, BAR(B3_DF + st), 0, (j0 + j2) * kKeys3, hl);
                    tma_load_3d(sbase + kOff3K + st2 * kK3Bytes + 8192, &tm_k, BAR(B3_DF + st), 64, (j0 + j2) * kKeys3, hl);
                }
            }
        }
    } else if (warp >= 9) {
        if (warp < 9 + TILES) {
        /* ===================== MMA issuer of tile x (whole warp, one elected lane issues) =====================
         * order: S_x(0) S_x(1) | PV_x(0) S_x(2) | PV_x(1) S_x(3) | ...   tcgen05.commit covers what this thread issued, so
         * a K or V stage is released by one commit of each issuer */
        const int x = warp - 9;
        /* one election for the whole walk: `lead` is 1 in the issuing lane (an elect.sync in front of every MMA and commit
         * costs 1.7 % of the kernel) */
        const unsigned lead = elect_one();
        bool ok = mbar_wait_blocking(BAR(B3_Q), 0u, s_abort, a.err, 20u);
        const unsigned long long dQ = make_desc(sbase + kOff3Q + x * kTileBytes);
        const unsigned long long dK0 = make_desc(sbase + kOff3K), dV0 = make_desc(sbase + kOff3V);
        const unsigned tm_sx = tmem + 128u * x, tm_ox = tmem + 256u + 128u * x;
        auto issue_qk = [&](int j) {      /* S_x(j) = Q_x . K_j^T into buffer j & 1: 8 k-steps of 16 over d = 128 */
            const unsigned long long k = dK0 + (unsigned long long)((j & (kSt3 - 1)) * (kK3Bytes >> 4));
            const unsigned d = tm_sx + 64u * (j & 1);
#pragma unroll
            for (int kk = 0; kk < 8; kk++)      /* the second half of d lies one sub-tile further on: 16 KB for Q, 8 KB for K */
                umma_f16_n64_lead(d, dQ + (unsigned long long)((kk >> 2) * 1024 + (kk & 3) * 2), k + (unsigned long long)((kk >> 2) * 512 + (kk & 3) * 2), kk > 0, lead);
            umma_commit_lead(BAR(B3_SF + 2 * x + (j & 1)), lead);
        };
        /* tile B starts when the first softmax of tile A is through: half a period out of phase, the MMAs of one tile
         * run while the other tile's issuer is between two steps and its softmax warps have the SM's exponential
         * unit to themselves (nothing pulls the two loops apart by itself when they start together) */
        if (ok && x == 1 && (MODE != PF_CLUSTER || ntiles > 0)) ok = mbar_wait_blocking(BAR(B3_P + 0), 0u, s_abort, a.err, 22u);
        for (int j = 0; j < 2 && j < ntiles && ok; j++) {
            ok = __all_sync(0xffffffffu, mbar_wait_blocking(BAR(B3_K0F + j), 0u, s_abort, a.err, 21u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            issue_qk(j);
            umma_commit_lead(BAR(B3_K0E + j), lead);
        }
        for (int j = 0; j < ntiles && ok; j++) {
            const int st = j & (kSt3 - 1), j2 = j + 2; const unsigned ph = (unsigned)(j / kSt3) & 1u;
            ok = mbar_wait_blocking(BAR(B3_DF + st), ph, s_abort, a.err, 23u);                                               /* V_j and K_(j+2) */
            if (ok) ok = mbar_wait_blocking(BAR(B3_P + 2 * x + (j & 1)), (unsigned)(j >> 1) & 1u, s_abort, a.err, 24u);   /* P_x(j) in tensor memory, O_x rescaled */
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            /* O_x += P_x(j) . V_j : 4 k-steps of 16 keys; A = 8 columns of packed fp16 pairs per step */
            {
                const unsigned long long v = dV0 + (unsigned long long)(st * (kK3Bytes >> 4));
                const unsigned pa = tm_sx + 64u * (j & 1);
                const unsigned acc0 = j > 0 ? 1u : 0u;
#pragma unroll
                for (int kk = 0; kk < 4; kk++) umma_f16_ta_lead(tm_ox, pa + 8u * kk, v + (unsigned long long)(kk * 2), kk > 0 ? 1u : acc0, lead);
            }
            /* completion of P.V is only asked for directly at the end (last rescale, epilogue); before that the softmax
             * warps learn it from S_x(j+2), which this thread issues behind it */
            if (j + 2 >= ntiles) umma_commit_lead(BAR(B3_O + 2 * x + (j + 1 == ntiles ? 1 : 0)), lead);
            if (j2 < ntiles) issue_qk(j2);
            umma_commit_lead(BAR(B3_DE + st), lead);
        }
        }
    } else if (warp < 4 * TILES) {
        /* ===================== softmax warps: tile x = warp / 4; thread = one row of Q tile x ===================== */
        const int x = warp >> 2, t_local = (tid & 127) >> 3;
        const int tq0 = q0 + x * kQTok;                          /* first query token of this tile */
        const int qpos = a.base + tq0 + t_local;                 /* global index of this row's query */
        const unsigned lane_base = (unsigned)((warp & 3) * 32) << 16; /* this warp's quarter of the TMEM lanes */
        const unsigned tm_o = tmem + 256u + 128u * x + lane_base;
        float m = -INFINITY;
        float2 l2 = make_float2(0.f, 0.f);
        bool ok = true;
        if (TILES == 2 && x == 1 && (MODE != PF_CLUSTER || ntiles > 0)) turn_pass(1);      /* tile A has the first turn (a piece of a cluster may have no steps) */
        for (int j = 0; j < ntiles; j++) {       /* to the end also after a wait ran out: the turns have to match */
            const unsigned tm_s = tmem + 128u * x + 64u * (j & 1) + lane_base;
            ok = __all_sync(0xffffffffu, mbar_wait_blocking(BAR(B3_SF + 2 * x + (j & 1)), (unsigned)(j >> 1) & 1u, s_abort, a.err, 30u));   /* keep the warp together */
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int k0 = (j0 + j) * kKeys3;
            const bool masked = (k0 + kKeys3 - 1 > a.base + tq0);   /* the tile crosses the diagonal of some row */
            unsigned v[64];
            tmem_ld32_nowait(tm_s, v);
            tmem_ld32_nowait(tm_s + 32u, v + 32);
            tmem_ld_wait(v);
            tmem_ld_wait(v + 32);
            if (masked) {      /* only the tiles on the diagonal pay for the causal test */
#pragma unroll
                for (int i = 0; i < 64; i++) if (k0 + i > qpos) v[i] = 0xff800000u;
            }
            /* the maximum is taken over the raw scores (the scale is positive) and the scale is folded into the exponent's
             * argument.  A tile that is masked for the whole row (its keys all lie behind the row's query; only in the last
             * tiles of the CTA) has mx = -inf: nothing moves and all its P are 0 */
            const float mx = row_max(v) * kScaleLog2;
            const bool grow = mx > m + kPfThreshold;              /* true while m == -inf, unless all keys so far are masked (last piece of a cut block) */
            if (__any_sync(0xffffffffu, grow)) {
                /* tcgen05.ld / .st are warp-collective: the whole warp rescales its 32 rows as soon as one of them moved its
                 * reference (the others multiply by exactly 1).  O_x is only ours when P_x(j-1).V_(j-1) has completed:
                 * S_x(j+1) was issued behind P_x(j-1).V, and a commit covers everything its thread issued before */
                const float m_new = grow ? mx : m, alpha = grow ? ex2f(m - m_new) : 1.f;     /* 0 on the first tile (m = -inf) */
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, j + 1 < ntiles ? mbar_wait_blocking(BAR(B3_SF + 2 * x + ((j + 1) & 1)), (unsigned)((j + 1) >> 1) & 1u, s_abort, a.err, 31u)
                                                               : mbar_wait_blocking(BAR(B3_O + 2 * x), 0u, s_abort, a.err, 31u));
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (ok) {
#pragma unroll 1
                        for (int c = 0; c < 4; c++) {
                            unsigned o[32];
                            tmem_ld32_nowait(tm_o + 32u * c, o);
                            tmem_ld_wait(o);
#pragma unroll
                            for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st32(tm_o + 32u * c, o);
                        }
                    }
                }
                l2.x *= alpha; l2.y *= alpha;
                m = m_new;
            }
            unsigned pk[32];
            const float2 ls = softmax_exp<CUT, TILES == 2>(v, m, pk, x, x == 0 || j + 1 < ntiles);
            l2 = add2(l2, ls);
            /* P over the first 32 columns of this S buffer (column c = keys 2c, 2c+1) */
            tmem_st32(tm_s, pk);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(B3_P + 2 * x + (j & 1)));
        }
        const float l = l2.x + l2.y;
        /* epilogue: O / l.  The issuer commits P.V of the last two tiles on barriers of their own, which therefore complete
         * exactly once (a parity wait on a barrier that runs through many phases can only tell the last completed phase
         * from the one before it, and a waiter here could be two behind).  The last commit covers all earlier MMAs. */
        if (ok && ntiles > 0) ok = mbar_wait_blocking(BAR(B3_O + 2 * x + 1), 0u, s_abort, a.err, 32u);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        ok = __all_sync(0xffffffffu, ok);                     /* warp-uniform: tcgen05.ld is warp-collective */
        if (MODE == PF_CLUSTER) {
            /* The CL pieces of a block meet in shared memory: CTA r of the cluster finishes columns [128 r / CL, 128 (r + 1) / CL) of
             * all rows.  Every piece sends the others their columns of its O and every row's {m, l}; the zones lie over the Q
             * tiles and the K ring, which are free in all CTAs once all have arrived behind their last P.V.  Bound by the bytes
             * between the SMs (98 KB out of and into each CTA of 4): 45 tokens behind 1 001 in two tiles a CTA take 14.3 us a launch,
             * 21.0 with records through memory, and 19.0 with chunks of a row side by side (a store then crosses as 32 pieces of 16 bytes). */
            constexpr int W4 = 32 / CL;                          /* float4 chunks of a row that a CTA finishes */
            constexpr int kZone = W4 * kRows * 16;               /* one source's zone: [W4 chunks][rows] */
            constexpr int kOffMl = CL * kZone, kOffWt = kOffMl + CL * kRows * 8;
            static_assert(kOffWt + CL * kRows * 4 <= kOff3Bar, "the zones overlap the barriers");
            const int me = w.piece, row = tid;
            /* chunk c of all rows is contiguous, so that a warp's store crosses as 512 consecutive bytes; rows are permuted within
             * groups of 8 by the chunk, so that 8 lanes which read a row's chunks (CL = 8: two rows') hit all banks */
            auto zone_off = [](int r, int c) { return c * (kRows * 16) + ((r & ~7) | ((r ^ (CL == 8 ? 2 * c : c)) & 7)) * 16; };
            const bool live = tq0 + (warp & 3) * 4 < a.nq;       /* the warp has query tokens: else nothing to send or finish */
            cluster_arrive();
            cluster_wait();
#pragma unroll 1
            for (int c = 0; c < 4 && live; c++) {
                unsigned v[32];
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = 0u;          /* a piece without steps has no O */
                if (ntiles > 0 && ok) {
                    tmem_ld32_nowait(tm_o + 32u * c, v);
                    tmem_ld_wait(v);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int c4 = 8 * c + i;                    /* chunk of the whole row */
                    st_cluster16(cluster_addr(sbase + me * kZone + zone_off(row, c4 % W4), c4 / W4),
                                 __uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
                }
            }
#pragma unroll
            for (int r = 0; r < CL; r++) if (live) st_cluster8(cluster_addr(sbase + kOffMl + (me * kRows + row) * 8, r), m, l);
            cluster_arrive();
            cluster_wait();
            /* weights of the pieces for this thread's row (a piece of masked keys has m = -inf: weight 0; key 0 is never masked) */
            if (live) {
                float2 ml[CL];
#pragma unroll
                for (int r = 0; r < CL; r++) ml[r] = *reinterpret_cast<const float2 *>(sm + kOffMl + (r * kRows + row) * 8);
                float M = ml[0].x, L = 0.f;
#pragma unroll
                for (int r = 1; r < CL; r++) M = fmaxf(M, ml[r].x);
#pragma unroll
                for (int r = 0; r < CL; r++) { ml[r].x = ex2f(ml[r].x - M); L += ml[r].y * ml[r].x; }
                const float inv = L > 0.f ? 1.f / L : 0.f;
#pragma unroll
                for (int r = 0; r < CL; r++) *reinterpret_cast<float *>(sm + kOffWt + (r * kRows + row) * 4) = ml[r].x * inv;
            }
            __syncwarp();                                        /* a warp folds its own 32 rows */
            const int c = lane % W4;
            float *o0 = a.out + (size_t)((a.kv_head_begin + hl) * 8) * HY3A_D + (me * W4 + c) * 4;
#pragma unroll
            for (int i = 0; i < W4 && live; i++) {
                const int r = warp * 32 + i * (32 / W4) + lane / W4, t = q0 + (r >> 3);
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int p = 0; p < CL; p++) {
                    const float4 v = *reinterpret_cast<const float4 *>(sm + p * kZone + zone_off(r, c));
                    const float f = *reinterpret_cast<const float *>(sm + kOffWt + (p * kRows + r) * 4);
                    acc.x = fmaf(v.x, f, acc.x); acc.y = fmaf(v.y, f, acc.y); acc.z = fmaf(v.z, f, acc.z); acc.w = fmaf(v.w, f, acc.w);
                }
                if (t < a.nq) *reinterpret_cast<float4 *>(o0 + (size_t)t * a.out_stride + (r & 7) * HY3A_D) = acc;
            }
        } else if (np == 1 && ok) {
            /* A thread holds a row, so storing from the registers touches 32 rows per instruction; the warp's 32 rows go through
             * shared memory instead, 64 columns at a time (its quarter of Q_x, which P.V's last commit says is read; 16-byte
             * chunk c of row r at c ^ (r & 7): conflict-free both ways), and leave as two rows of 256 contiguous bytes per
             * instruction (one step of 32 tokens 8.4 -> 6.4 us a launch, 512 fresh tokens 16.4 -> 14.3 us). */
            const float inv = l > 0.f ? 1.f / l : 0.f;
            uint8_t *stage = sm + kOff3Q + x * kTileBytes + (warp & 3) * 8192;
            const int t0 = tq0 + (warp & 3) * 4, nrow = min(32, (a.nq - t0) * 8);          /* rows of valid query tokens (none: <= 0) */
            float *o0 = a.out + (size_t)t0 * a.out_stride + (size_t)((a.kv_head_begin + hl) * 8) * HY3A_D + (lane & 15) * 4;
#pragma unroll 1
            for (int c = 0; c < 2; c++) {
                unsigned v[64];
                tmem_ld32_nowait(tm_o + 64u * c, v);
                tmem_ld32_nowait(tm_o + 64u * c + 32u, v + 32);
                tmem_ld_wait(v);
                tmem_ld_wait(v + 32);
#pragma unroll
                for (int i = 0; i < 16; i++)
                    *reinterpret_cast<float4 *>(stage + lane * 256 + ((i ^ (lane & 7)) << 4)) =
                        make_float4(__uint_as_float(v[4 * i]) * inv, __uint_as_float(v[4 * i + 1]) * inv, __uint_as_float(v[4 * i + 2]) * inv, __uint_as_float(v[4 * i + 3]) * inv);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int r2 = 2 * i + (lane >> 4);
                    if (r2 < nrow) *reinterpret_cast<float4 *>(o0 + (size_t)(r2 >> 3) * a.out_stride + (r2 & 7) * HY3A_D + 64 * c) =
                        *reinterpret_cast<const float4 *>(stage + r2 * 256 + (((lane & 15) ^ (r2 & 7)) << 4));
                }
                __syncwarp();
            }
        } else if (np > 1 && tq0 + (warp & 3) * 4 < a.nq) {   /* a warp without query tokens leaves no record */
            /* a piece of a cut block: every softmax warp leaves the record of its 32 rows, and the last of the np warps with
             * these rows to arrive folds the records in the order of the pieces (the result does not depend on who is last) */
            const size_t slot0 = (size_t)rec0 * a.kv_heads + hl;          /* record of piece p: slot0 + p * kv_heads */
            const size_t rec_step = (size_t)a.kv_heads * 8 * kRecWarp;
            float *rec = a.rec + (slot0 * 8 + warp) * kRecWarp;
            if (ok) {
                float4 *dst = reinterpret_cast<float4 *>(rec + piece * rec_step);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    unsigned v[32];
                    tmem_ld32_nowait(tm_o + 32u * c, v);
                    tmem_ld_wait(v);
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        __stcg(dst + (8 * c + i) * 32 + lane, make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3])));
                }
                __stcg(reinterpret_cast<float2 *>(dst + 1024) + lane, make_float2(m, l));
            }
            __threadfence();
            __syncwarp();
            unsigned old = 0;
            if (lane == 0) old = atomicAdd(a.cnt + slot0 * 8 + warp, 1u);
            old = __shfl_sync(0xffffffffu, old, 0);
            if (old == (unsigned)np - 1u) {
                __threadfence();
                if (lane == 0) a.cnt[slot0 * 8 + warp] = 0u;              /* ready for the next launch */
                /* the loads of four records are in flight at once (indices past the end read the last record again) */
                auto ml_of = [&](int p) { return __ldcg(reinterpret_cast<const float2 *>(rec + min(p, np - 1) * rec_step + 4096) + lane); };
                float M = -INFINITY, L = 0.f;
                for (int p = 0; p < np; p += 4) {
                    float2 ml[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) ml[i] = ml_of(p + i);
                    /* finite from the first record on: key 0 is never masked */
                    const float m_new = fmaxf(fmaxf(fmaxf(M, ml[0].x), ml[1].x), fmaxf(ml[2].x, ml[3].x));
                    L *= ex2f(M - m_new);
                    M = m_new;
#pragma unroll
                    for (int i = 0; i < 4; i++) if (p + i < np) L += ml[i].y * ex2f(ml[i].x - M);     /* a record of masked keys has weight 0 */
                }
                const float inv = L > 0.f ? 1.f / L : 0.f;
                const bool row_valid = tq0 + t_local < a.nq;
                float *orow = a.out + (size_t)(tq0 + t_local) * a.out_stride + (size_t)((a.kv_head_begin + hl) * 8 + (tid & 7)) * HY3A_D;
#pragma unroll 1
                for (int c = 0; c < 4; c++) {
                    float4 acc[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
                    for (int p = 0; p < np; p += 2) {       /* two records in flight: a trip to L2 is most of a round */
                        const bool two = p + 1 < np;
                        const float *r0 = rec + p * rec_step, *r1 = two ? r0 + rec_step : r0;
                        float4 v0[8], v1[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            v0[i] = __ldcg(reinterpret_cast<const float4 *>(r0) + (8 * c + i) * 32 + lane);
                            v1[i] = __ldcg(reinterpret_cast<const float4 *>(r1) + (8 * c + i) * 32 + lane);
                        }
                        const float f0 = ex2f(ml_of(p).x - M) * inv, f1 = two ? ex2f(ml_of(p + 1).x - M) * inv : 0.f;
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            acc[i].x = fmaf(v1[i].x, f1, fmaf(v0[i].x, f0, acc[i].x)); acc[i].y = fmaf(v1[i].y, f1, fmaf(v0[i].y, f0, acc[i].y));
                            acc[i].z = fmaf(v1[i].z, f1, fmaf(v0[i].z, f0, acc[i].z)); acc[i].w = fmaf(v1[i].w, f1, fmaf(v0[i].w, f0, acc[i].w));
                        }
                    }
                    if (row_valid)
#pragma unroll
                    for (int i = 0; i < 8; i++) *reinterpret_cast<float4 *>(orow + 32 * c + 4 * i) = acc[i];
                }
            }
        }
    }
    if (MODE == PF_CLUSTER && warp >= 4 * TILES) {       /* the other roles arrive for the two meetings of the epilogue */
        __syncwarp();
        cluster_arrive(); cluster_wait();
        cluster_arrive(); cluster_wait();
    }
    /* ---- common exit: everybody arrives here, also after a wait ran out; release TMEM */
    if (*s_abort && warp == 8 && lane == 0) {
        /* copies already issued must land before the shared memory goes away */
        for (int st = 0; st < kSt3; st++)
            for (unsigned ph = 0; ph < 2; ph++)
                for (unsigned spin = 0; spin < (1u << 12) && !mbar_test(BAR(B3_DF + st), ph); spin++) __nanosleep(64);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
#undef BAR
}
/* blocks uncut (full grids; of one tile where these do not fill the SMs) */
template <int TILES>
__global__ void __launch_bounds__(kPf3Threads, 1)
hy3a_prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ prefill_args a) {
    pf_where w = {0, 0, 0, 0, 0, 1, 0};
    int ent;
    entry_of(a, ent, w.hl);
    w.qblk = a.entries - 1 - ent;
    w.ntiles = (min(a.base + (w.qblk + 1) * kQTok * TILES, a.base + a.nq) + kKeys3 - 1) / kKeys3;      /* keys behind these do not matter for this CTA */
    prefill_body<PF_WHOLE, 1, TILES>(tm_q, tm_k, tm_v, a, w);
}
/* blocks cut along the keys (grids that would leave SMs idle); a separate kernel, because the offsets and the -inf test of its
 * inner loop cost the other one 5 % */
__global__ void __launch_bounds__(kPf3Threads, 1)
hy3a_prefill_cut_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ prefill_args a,
                        const __grid_constant__ hy3a_pf_table tab) {
    int ent, hl;
    entry_of(a, ent, hl);
    const hy3a_pf_piece pc = tab.e[ent];
    const pf_where w = {hl, pc.qblk, pc.j0, pc.n, pc.piece, pc.np, pc.rec};
    prefill_body<PF_CUT, 1>(tm_q, tm_k, tm_v, a, w);
}
/* blocks cut into CL pieces, one per CTA of a cluster */
template <int CL, int TILES>
__global__ void __launch_bounds__(kPf3Threads, 1)
hy3a_prefill_cluster_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ prefill_args a) {
    pf_where w = {0, 0, 0, 0, 0, 1, 0};
    const int blk = blockIdx.x / CL, ent = blk / a.kv_heads;      /* longest blocks first */
    w.piece = blockIdx.x - blk * CL;                              /* = rank in the cluster */
    w.hl = blk - ent * a.kv_heads;
    w.qblk = a.entries - 1 - ent;
    const int nt = (min(a.base + (w.qblk + 1) * kQTok * TILES, a.base + a.nq) + kKeys3 - 1) / kKeys3;
    w.j0 = w.piece * nt / CL;
    w.ntiles = (w.piece + 1) * nt / CL - w.j0;
    prefill_body<PF_CLUSTER, CL, TILES>(tm_q, tm_k, tm_v, a, w);
}


} /* namespace */

template <int TILES>
static const void *pf_cluster_fn(int cl) {
    return cl == 2 ? (const void *)hy3a_prefill_cluster_kernel<2, TILES> : cl == 4 ? (const void *)hy3a_prefill_cluster_kernel<4, TILES> : (const void *)hy3a_prefill_cluster_kernel<8, TILES>;
}

typedef CUresult (*hy3a_encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                         const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                         CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static hy3a_encode_tiled_fn get_encode_tiled(void) {
    static hy3a_encode_tiled_fn fn = NULL;
    if (!fn) {
        void *p = NULL;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            fn = (hy3a_encode_tiled_fn)p;
    }
    return fn;
}

/* 3-D fp16 tensor map with a 128-byte swizzle; dims/box innermost first, strides in bytes for dims 1 and 2 */
static int make_map(hy3a_ctx *ctx, CUtensorMap *map, void *base, const cuuint64_t dims[3], const cuuint64_t strides[2], const cuuint32_t box[3]) {
    hy3a_encode_tiled_fn enc = get_encode_tiled();
    if (!enc) return hy3a_fail(ctx, HY3A_ECUDA, "prefill: cuTensorMapEncodeTiled is not available from the driver");
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return hy3a_fail(ctx, HY3A_ECUDA, "prefill: cuTensorMapEncodeTiled failed (%d)", (int)r);
    return HY3A_OK;
}

/* Attributes of the attention kernels on the context's device (they are per device), and how many clusters of 2^i CTAs fit on it at
 * once (148 SMs of a B200: 74 of 2, 33 of 4, 15 of 8). */
static int prefill_device(hy3a_ctx *ctx, const int **cap) {
    static bool done_dev[64];
    static int cap_dev[64][4];
    const int dev = ctx->device & 63;
    if (!done_dev[dev]) {
        HY3A_CUDA(ctx, cudaFuncSetAttribute(hy3a_prefill_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPf3Smem));
        HY3A_CUDA(ctx, cudaFuncSetAttribute(hy3a_prefill_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPf3Smem));
        HY3A_CUDA(ctx, cudaFuncSetAttribute(hy3a_prefill_cut_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPf3Smem));
        for (int i = 1; i < 4; i++) {
            const void *f = pf_cluster_fn<2>(1 << i);
            HY3A_CUDA(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kPf3Smem));
            HY3A_CUDA(ctx, cudaFuncSetAttribute(pf_cluster_fn<1>(1 << i), cudaFuncAttributeMaxDynamicSharedMemorySize, kPf3Smem));
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = 1 << i; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(64 << i); cfg.blockDim = dim3(kPf3Threads); cfg.dynamicSmemBytes = kPf3Smem; cfg.attrs = at; cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }   /* no clusters of this size */
            cap_dev[dev][i] = n;
        }
        done_dev[dev] = true;
    }
    *cap = cap_dev[dev];
    return HY3A_OK;
}

/* the cut depends on the chunk's sizes alone; the layers of a chunk share it */
static void plan_chunk(hy3a_ctx *ctx, const int *cap, int base_slot, int nq) {
    if (ctx->pf_plan_base == base_slot && ctx->pf_plan_nq == nq) return;
    float end = 0.f;
    hy3a_pf_plan(base_slot, nq, ctx->cfg.kv_head_count, ctx->sm_count, ctx->d_pf_rec ? HY3A_PF_MAX_SLOTS : 0, &ctx->pf_plan, &end);
    ctx->pf_plan_cluster = ctx->no_clusters ? 1 : hy3a_pf_cluster(base_slot, nq, ctx->cfg.kv_head_count, cap, end, ctx->pf_plan);
    ctx->pf_plan_base = base_slot; ctx->pf_plan_nq = nq;
}

extern "C" int hy3a_prefill_cluster(hy3a_ctx *ctx, int base_slot, int nq) {
    if (!ctx) return HY3A_EINVAL;
    if (base_slot < 0 || nq < 1) return hy3a_fail(ctx, HY3A_EINVAL, "prefill_cluster: base_slot %d, nq %d", base_slot, nq);
    hy3a_device_guard guard(ctx->device);      /* a query: any device may be current */
    const int *cap = NULL;
    int rc = prefill_device(ctx, &cap);
    if (rc) return rc;
    plan_chunk(ctx, cap, base_slot, nq);
    return ctx->pf_plan_cluster;
}

int hy3a_launch_prefill(hy3a_ctx *ctx, int layer, int seq, int base_slot, int nq, const void *q16, float *out, size_t out_stride) {
    const int kvh = ctx->cfg.kv_head_count;
    const int ntok = base_slot + nq;
    const int pages = (ntok + HY3A_PT - 1) / HY3A_PT;
    int tok_stride = pages * HY3A_PT, pg0 = 0;
    void *ws_k = NULL, *ws_v = NULL;
    /* 1st choice: this layer's operand mirror -- only the pages written since the last chunk are converted */
    if (ctx->pf_mbudget) {
        if (ctx->pf_mseq != seq) { for (int l = 0; l < ctx->cfg.n_layers; l++) ctx->pf_mntok[l] = 0; ctx->pf_mseq = seq; }
        const int want = (tok_stride + 1023) / 1024 * 1024;
        if (want > ctx->pf_mcap[layer]) {
            const int seq_cap = (ctx->cfg.max_blocks_per_seq * HY3A_PT + 1023) / 1024 * 1024;
            int cap = 2 * ctx->pf_mcap[layer];
            if (cap > seq_cap) cap = seq_cap;
            if (cap < want) cap = want;
            const size_t old_b = 2 * (size_t)kvh * ctx->pf_mcap[layer] * HY3A_D * sizeof(__half), new_b = 2 * (size_t)kvh * cap * HY3A_D * sizeof(__half);
            if (ctx->pf_mbytes - old_b + new_b <= ctx->pf_mbudget) {
                HY3A_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
                cudaFree(ctx->pf_mk[layer]); cudaFree(ctx->pf_mv[layer]);
                ctx->pf_mk[layer] = ctx->pf_mv[layer] = NULL; ctx->pf_mcap[layer] = 0; ctx->pf_mntok[layer] = 0; ctx->pf_mbytes -= old_b;
                /* zeroed once: columns past a sequence's end are read by the last tile (and masked), so they must never
                 * hold a NaN or Inf pattern; afterwards only finite values are written */
                if (cudaMalloc(&ctx->pf_mk[layer], new_b / 2) == cudaSuccess && cudaMalloc(&ctx->pf_mv[layer], new_b / 2) == cudaSuccess &&
                    cudaMemsetAsync(ctx->pf_mk[layer], 0, new_b / 2, ctx->stream) == cudaSuccess && cudaMemsetAsync(ctx->pf_mv[layer], 0, new_b / 2, ctx->stream) == cudaSuccess) {
                    ctx->pf_mcap[layer] = cap; ctx->pf_mbytes += new_b;
                } else {
                    cudaGetLastError();
                    cudaFree(ctx->pf_mk[layer]); ctx->pf_mk[layer] = ctx->pf_mv[layer] = NULL;   /* fall through to the shared workspace */
                }
            }
        }
        if (want <= ctx->pf_mcap[layer]) {
            ws_k = ctx->pf_mk[layer]; ws_v = ctx->pf_mv[layer];
            tok_stride = ctx->pf_mcap[layer];
            /* a partly filled page is converted again; nothing is, when the append kernel wrote the rows through */
            pg0 = ctx->pf_mntok[layer] >= ntok ? pages : ctx->pf_mntok[layer] / HY3A_PT;
            if (ctx->pf_mntok[layer] < ntok) ctx->pf_mntok[layer] = ntok;
        }
    }
    /* 2nd choice: one workspace shared by all layers, rebuilt from the pages on every call (grow-only, in steps of
     * 1024 tokens) */
    if (!ws_k) {
        const size_t need = (size_t)kvh * (((size_t)tok_stride + 1023) / 1024 * 1024) * HY3A_D * sizeof(__half);
        if (need > ctx->pf_bytes) {
            HY3A_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            cudaFree(ctx->d_pf_k); cudaFree(ctx->d_pf_v);
            ctx->d_pf_k = ctx->d_pf_v = NULL; ctx->pf_bytes = 0;
            if (cudaMalloc(&ctx->d_pf_k, need) != cudaSuccess || cudaMalloc(&ctx->d_pf_v, need) != cudaSuccess) {
                cudaFree(ctx->d_pf_k); ctx->d_pf_k = NULL;
                return hy3a_fail(ctx, HY3A_ENOMEM, "prefill: cannot allocate 2 x %zu bytes of fp16 workspace", need);
            }
            ctx->pf_bytes = need;
        }
        ws_k = ctx->d_pf_k; ws_v = ctx->d_pf_v;
    }
    hy3a_cache_view cv = hy3a_view(ctx);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    if (pages > pg0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(pages - pg0, kvh, 4); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = 0; cfg.stream = ctx->stream;
        cfg.attrs = attr; cfg.numAttrs = ctx->use_pdl ? 1 : 0;
        __half *wk = (__half *)ws_k, *wv = (__half *)ws_v;
        cudaError_t e;
        switch (ctx->geom.dtype) {
            case 0: e = cudaLaunchKernelEx(&cfg, hy3a_kv_to_f16_kernel<0>, cv, layer, seq, pg0, ntok, tok_stride, wk, wv); break;
            case 1: e = cudaLaunchKernelEx(&cfg, hy3a_kv_to_f16_kernel<1>, cv, layer, seq, pg0, ntok, tok_stride, wk, wv); break;
            default: e = cudaLaunchKernelEx(&cfg, hy3a_kv_to_f16_kernel<2>, cv, layer, seq, pg0, ntok, tok_stride, wk, wv); break;
        }
        ctx->launches++;
        HY3A_CUDA(ctx, e);
    }

    const int keys = kKeys3;
    CUtensorMap tq, tk, tv;
    {
        const cuuint64_t dq[3] = {HY3A_D, HY3A_N_HEAD, (cuuint64_t)nq}, sq[2] = {HY3A_D * 2, HY3A_N_HEAD * HY3A_D * 2};
        const cuuint32_t bq[3] = {64, 8, kQTok};
        int rc = make_map(ctx, &tq, const_cast<void *>(q16), dq, sq, bq);
        if (rc) return rc;
        const cuuint64_t dk[3] = {HY3A_D, (cuuint64_t)tok_stride, (cuuint64_t)kvh}, sk[2] = {HY3A_D * 2, (cuuint64_t)tok_stride * HY3A_D * 2};
        const cuuint32_t bk[3] = {64, (cuuint32_t)keys, 1};
        rc = make_map(ctx, &tk, ws_k, dk, sk, bk);
        if (rc) return rc;
        const cuuint64_t dv[3] = {(cuuint64_t)tok_stride, HY3A_D, (cuuint64_t)kvh}, sv[2] = {(cuuint64_t)tok_stride * 2, (cuuint64_t)tok_stride * HY3A_D * 2};
        const cuuint32_t bv[3] = {64, HY3A_D, 1};
        rc = make_map(ctx, &tv, ws_v, dv, sv, bv);
        if (rc) return rc;
    }
    const int *cl_cap = NULL;
    {
        int rc = prefill_device(ctx, &cl_cap);
        if (rc) return rc;
    }
    prefill_args a = {};
    a.out = out; a.out_stride = out_stride; a.base = base_slot; a.nq = nq; a.kv_head_begin = ctx->cfg.kv_head_begin; a.err = ctx->d_err;
    a.kv_heads = kvh; a.rec = ctx->d_pf_rec; a.cnt = ctx->d_pf_cnt;
    {
        plan_chunk(ctx, cl_cap, base_slot, nq);
        const int cl = ctx->pf_plan_cluster, blocks = (nq + kQTok2 - 1) / kQTok2;
        /* blocks of one tile where they fit at once too: as many SMs again share the softmax, and the exchange of clusters */
        const int blocks1 = (nq + kQTok - 1) / kQTok;
        cudaLaunchConfig_t cfg = {};
        cfg.stream = ctx->stream; cfg.blockDim = dim3(kPf3Threads); cfg.dynamicSmemBytes = kPf3Smem;
        cudaLaunchAttribute at[2];
        at[0] = attr[0];
        cfg.attrs = at; cfg.numAttrs = ctx->use_pdl ? 1 : 0;
        if (cl > 1) {
            const bool one = blocks1 * kvh <= cl_cap[cl == 2 ? 1 : cl == 4 ? 2 : 3];
            a.entries = one ? blocks1 : blocks;
            cudaLaunchAttribute &ca = at[cfg.numAttrs++];
            ca.id = cudaLaunchAttributeClusterDimension; ca.val.clusterDim.x = cl; ca.val.clusterDim.y = ca.val.clusterDim.z = 1;
            cfg.gridDim = dim3(a.entries * kvh * cl);
            void *args[4] = {&tq, &tk, &tv, &a};
            HY3A_CUDA(ctx, cudaLaunchKernelExC(&cfg, one ? pf_cluster_fn<1>(cl) : pf_cluster_fn<2>(cl), args));
        } else {
            const bool one = !ctx->pf_plan.count && blocks1 * kvh <= ctx->sm_count;
            const int entries = ctx->pf_plan.count ? ctx->pf_plan.count : one ? blocks1 : blocks;
            a.entries = entries; a.group = entries * kvh <= ctx->sm_count ? entries : kGroup;
            cfg.gridDim = dim3(entries * kvh);
            if (ctx->pf_plan.count) HY3A_CUDA(ctx, cudaLaunchKernelEx(&cfg, hy3a_prefill_cut_kernel, tq, tk, tv, a, ctx->pf_plan));
            else HY3A_CUDA(ctx, cudaLaunchKernelEx(&cfg, one ? hy3a_prefill_kernel<1> : hy3a_prefill_kernel<2>, tq, tk, tv, a));
        }
    }
    ctx->launches++;
    ctx->bulk_write_pending = 1;
    HY3A_CUDA(ctx, cudaGetLastError());
    return HY3A_OK;
}
