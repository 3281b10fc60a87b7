/*
 * prefill_plan.h -- how the chunked prefill is cut into CTAs (host code, no CUDA).
 *
 * A block is 32 query tokens of one KV head; it walks ceil(keys / 64) steps of 64 keys.  A chunk has
 * ceil(nq / 32) x heads blocks whose lengths grow with the query index, and one CTA occupies an SM, so blocks alone can leave
 * most SMs idle: 45 tokens are 16 blocks, 128 are 32.  A block may therefore be cut along the keys into pieces of M steps
 * (the last takes the rest); every piece of a cut block leaves a {m, l, O} record and the last to arrive folds them.  M is
 * chosen per chunk by list scheduling in units of steps, longest pieces first.  Or the CTAs of a cluster share a block
 * (hy3a_pf_cluster, below).
 */
#ifndef HY3A_PREFILL_PLAN_H
#define HY3A_PREFILL_PLAN_H

#include <stdint.h>
#include <string.h>

#include <algorithm>

#define HY3A_PF_MAX_PIECES 256   /* table entries (pieces of one head); longer chunks run uncut */
#define HY3A_PF_MAX_SLOTS 512    /* piece records in the scratch */
#define HY3A_PF_REC_BYTES (8 * (32 * 128 + 64) * 4)   /* 8 warps x 32 rows x {O[128], m, l} fp32 */
#define HY3A_PF_QTOK 32
#define HY3A_PF_KEYS 64

struct hy3a_pf_piece {
    uint16_t qblk;               /* query block: tokens 32 qblk .. */
    uint16_t j0, n;              /* steps [j0, j0 + n) of 64 keys */
    uint16_t rec;                /* index of the block's first record per head (cut blocks) */
    uint8_t piece, np;           /* this piece, pieces of the block */
    uint16_t pad;
};
struct hy3a_pf_table {
    int count;                   /* 0: uncut blocks in descending order, no table needed */
    hy3a_pf_piece e[HY3A_PF_MAX_PIECES];
};

/* The plan and the choice of clusters compare blocks of 32 tokens, two query tiles a CTA.  The launch takes blocks of 16, one tile a CTA, where
 * these fit at once as well (hy3a_launch_prefill); what that saves (blocks cut into records never take it) is not in these costs.
 * Costs in steps of both query tiles (0.79 us in a CTA by itself, 0.9 with 128 CTAs): start and end of a CTA, writing a record,
 * folding one record.  To derive them again: a one-step launch takes 6.5 us; 32 tokens behind 4 064 (8 CTAs uncut, 56.9 us) in 2 /
 * 4 / 8 / 16 pieces a block take 42.5 / 32.1 / 28.1 / 33.6 us, i.e. 10.7 / 13.0 / 15.3 / 24 us beside the steps and the 6.5, where
 * 5 + 1.5 pieces say 6.3 / 8.7 / 13.4 / 22.9.  The model is 2 to 4 us low for few pieces, which the 0.88 below allows for. */
constexpr float kPfCostCta = 8.0f, kPfCostRecord = 5.0f, kPfCostFold = 1.5f;

static inline int hy3a_pf_steps(int base, int nq, int qblk) {
    const int end = std::min(base + (qblk + 1) * HY3A_PF_QTOK, base + nq);
    return (end + HY3A_PF_KEYS - 1) / HY3A_PF_KEYS;
}

/* when the last CTA of the table ends, in steps (list scheduling on a heap of SM groups that divide the heads evenly); gives
 * up as soon as the end is known to be no earlier than `limit` */
static inline float hy3a_pf_makespan(const hy3a_pf_table *t, int heads, int sms, float limit, float extra = 0.f) {
    int unit = heads;
    while (unit > 1 && (sms % unit || heads % unit)) unit--;
    const int ng = std::min(sms / unit, 256), reps = heads / unit;
    float load[256];
    for (int i = 0; i < ng; i++) load[i] = 0.f;
    float end = 0.f;
    for (int c = 0; c < t->count; c++) {
        const hy3a_pf_piece &e = t->e[c];
        const float cost = kPfCostCta + extra + e.n + (e.np > 1 ? kPfCostRecord : 0.f), fold = e.np > 1 ? kPfCostFold * e.np : 0.f;
        for (int r = 0; r < reps; r++) {
            const float v = load[0] + cost;       /* the least loaded group is at the root */
            if (v + fold > end) { end = v + fold; if (end >= limit) return end; }
            int i = 0;
            for (int k = 1; k < ng; k = 2 * i + 1) {
                if (k + 1 < ng && load[k + 1] < load[k]) k++;
                if (load[k] >= v) break;
                load[i] = load[k]; i = k;
            }
            load[i] = v;
        }
    }
    return end;
}

/* pieces of at most M steps in descending order of length; false: does not fit the table or the records, or the work alone
 * fills the SMs up to `limit` */
static inline bool hy3a_pf_cut(int base, int nq, int heads, int sms, int M, int max_slots, float limit, hy3a_pf_table *t) {
    const int nqb = (nq + HY3A_PF_QTOK - 1) / HY3A_PF_QTOK;
    int rec = 0, count = 0;
    float work = 0.f;
    for (int q = nqb - 1; q >= 0; q--) {
        const int nt = hy3a_pf_steps(base, nq, q), np = (nt + M - 1) / M;
        if (np > 255 || count + np > HY3A_PF_MAX_PIECES || (np > 1 && (rec + np) * heads > max_slots)) return false;
        work += nt + np * (kPfCostCta + (np > 1 ? kPfCostRecord : 0.f));
        int j0 = 0;
        for (int p = 0; p < np; p++) {
            hy3a_pf_piece &e = t->e[count++];
            e.qblk = (uint16_t)q; e.j0 = (uint16_t)j0; e.n = (uint16_t)std::min(M, nt - j0);
            e.rec = (uint16_t)(np > 1 ? rec : 0); e.piece = (uint8_t)p; e.np = (uint8_t)np; e.pad = 0;
            j0 += e.n;
        }
        if (np > 1) rec += np;
    }
    if (work * heads >= limit * sms) return false;
    t->count = count;
    std::sort(t->e, t->e + count, [](const hy3a_pf_piece &a, const hy3a_pf_piece &b) { return a.n != b.n ? a.n > b.n : (a.qblk != b.qblk ? a.qblk > b.qblk : a.piece < b.piece); });
    return true;
}

/* the plan of a chunk; max_slots = 0: no records, i.e. uncut blocks */
static inline void hy3a_pf_plan(int base, int nq, int heads, int sms, int max_slots, hy3a_pf_table *out, float *end = nullptr) {
    out->count = 0;
    const int nqb = (nq + HY3A_PF_QTOK - 1) / HY3A_PF_QTOK, longest = hy3a_pf_steps(base, nq, nqb - 1);
    if (nqb > HY3A_PF_MAX_PIECES || longest > 65535) return;
    long long total = 0;
    for (int q = 0; q < nqb; q++) total += hy3a_pf_steps(base, nq, q);
    const float share = (float)(total * heads) / sms;                 /* steps per SM */
    int cand[16], nc = 0;
    cand[nc++] = longest;                                             /* uncut */
    if (max_slots > 0 && longest > 1) {
        /* pieces a little above the even share (or an integral part of it), whose rests fill the remaining SMs; equal pieces */
        static const float f[8] = {1.06f, 1.12f, 1.0f, 0.56f, 0.52f, 0.36f, 0.27f, 1.2f};
        for (int i = 0; i < 8; i++) { const int M = (int)(share * f[i] + 0.5f * kPfCostCta); if (M >= 2 && M < longest) cand[nc++] = M; }
        for (int k = 2; k <= 6; k++) { const int M = (longest + k - 1) / k; if (M >= 2) cand[nc++] = M; }
    }
    hy3a_pf_table t;
    float best = 3e38f;
    for (int i = 0; i < nc; i++) {
        /* the kernel for cut blocks is 5 % slower a step, and rests that share an SM with others cost more than this model says */
        const float limit = best * (i == 0 ? 1.f : (out->count == 0 ? 0.88f : 0.98f));
        if (!hy3a_pf_cut(base, nq, heads, sms, cand[i], max_slots, limit, &t)) continue;
        const float m = hy3a_pf_makespan(&t, heads, sms, limit);
        if (m < limit) {
            best = m;
            if (end) *end = m;
            if (i) memcpy(out, &t, sizeof(int) + sizeof(hy3a_pf_piece) * (size_t)t.count);      /* uncut: no table */
        }
    }
}

/* CTAs per block (1: what the plan above says, whose end in steps is `end`, with blocks cut into records or not).  The blocks of a short chunk may run as clusters of 2,
 * 4 or 8 CTAs that share a block's keys evenly and meet in shared memory instead of through records; cap[i]: clusters of 2^i CTAs
 * that fit at once.  The meeting costs kPfCostMeet[i] steps when all 32 query tokens of a block are in use, and down to
 * kPfCostMeet[0] with the softmax warps that hold some (4 tokens each).  Measured with two tiles a CTA throughout, us a launch, 8 heads,
 * whole / with records / clusters of 2 / 4 / 8:
 *    45 behind  1 001   21.0  21.0  16.2  14.3  24.9      32 behind  4 064   56.9  28.6  36.2  23.9  20.6
 *     2 behind  1 001   18.2  18.2  13.0   9.3   7.6     128 behind  2 000   35.5  27.1  23.9  19.8  48.7
 *   200 behind  1 000   22.9  23.0  18.1  30.2  60.7     128 behind 16 000  230.6  72.9 110.1  67.8 119.5
 *    30 behind    300   11.1  11.1  10.8  11.1  13.9      64 behind  8 192  113.4  39.6  64.2  39.1  53.1
 *   600 behind  4 000  116.1 116.0 107.5 130.7      600 behind 16 000  435.7 324.7 350.1 336.2
 * and with one tile where the launch takes it (uncut up to 18 blocks of 16 a head, clusters of 2 / 4 / 8 up to 9 / 4 / 1):
 *    45 behind  1 001   15.1  15.2  11.8  10.6  25.3      32 behind  4 064   44.5  28.8  25.9  16.8  20.7
 *     2 behind  1 001   13.7  13.8  10.0   7.3   6.1     128 behind  2 000   26.2  27.6  17.7  20.4  48.1
 *   200 behind  1 000   17.0  17.1  18.3  30.2  60.0     128 behind 16 000  164.1  76.7  87.6  69.7 120.4
 *    30 behind    300    8.3   8.3   8.0   7.8  13.9      64 behind  8 192   86.2  40.4  47.8  29.7  53.4
 *     8 behind 16 000  158.8  38.0  84.0  45.0  26.7
 * The choice below was fitted to the first table.  Of 51 shapes measured so, it is more than 3 % behind the best in 11: 8 behind 16 000
 * 37.8, 32 behind 4 064 20.7, 128 behind 2 000 19.9, 200 behind 1 000 18.3, the others by 3 to 10 %.
 * Clusters of 4 and 8 only where all fit at once.  Records stay the better way for few tokens behind a very long history (more than
 * 8 pieces per block) and for a little more than one block per SM. */
constexpr float kPfCostMeet[4] = {0.8f, 3.5f, 5.5f, 10.f};
static inline int hy3a_pf_cluster(int base, int nq, int heads, const int cap[4], float end, const hy3a_pf_table &plan) {
    const int nqb = (nq + HY3A_PF_QTOK - 1) / HY3A_PF_QTOK, longest = hy3a_pf_steps(base, nq, nqb - 1);
    if (nqb > HY3A_PF_MAX_PIECES || end <= 0.f || longest > 65535) return 1;
    int best = 1;
    const float used = std::min(8, (nq + 3) / 4) * 0.125f;
    int np = 0;
    for (int c = 0; c < plan.count; c++) np = std::max(np, (int)plan.e[c].np);
    hy3a_pf_table t;
    t.count = nqb;
    for (int i = 1; i < 4; i++) {
        const int cl = 1 << i;
        const bool at_once = nqb * heads <= cap[i];
        if (cap[i] < 1 || (cl > 2 && !at_once)) continue;
        for (int c = 0; c < nqb; c++) {
            t.e[c].n = (uint16_t)((hy3a_pf_steps(base, nq, nqb - 1 - c) + cl - 1) / cl);
            t.e[c].np = 1;
        }
        /* the model of the records is up to 4 us low, and 0.7 of their fold goes with the tokens in use; that of several rounds of
         * clusters on every SM is a few percent low */
        float limit = end;
        /* a step of at most 4 tokens takes 0.2 longer (2 behind 16 000: 39.5 with records, 44.4 in clusters of 8; 8 tokens 37.8 and 38.1) */
        const float slow = nq <= 4 && np > 1 ? 0.2f * longest * (1.f / cl - 1.f / np) : 0.f;
        if (best == 1) limit = !at_once ? 0.97f * end : np > 1 ? end + 1.f + 3.6f * used - 0.7f * kPfCostFold * np * (1.f - used) - slow : end;
        const float m = hy3a_pf_makespan(&t, heads, cap[i], limit, kPfCostMeet[0] + (kPfCostMeet[i] - kPfCostMeet[0]) * used);
        if (m < limit) { best = cl; end = m; }
    }
    return best;
}

#endif
