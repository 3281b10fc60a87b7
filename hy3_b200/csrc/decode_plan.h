/*
 * decode_plan.h -- rules of the decode kernels' split into CTAs that the kernels and the host's description of them
 * (hy3a_decode_schedule_kv) share.  A unit is one page of one (row, KV head) segment.
 */
#ifndef HY3A_DECODE_PLAN_H
#define HY3A_DECODE_PLAN_H

#ifdef __CUDACC__
#define HY3A_HD __host__ __device__ __forceinline__
#else
#define HY3A_HD static inline
#endif

/* INT8 kernel, single-row grid: the last kLate pieces of the last segment take kLateCut pages less each (they start late) */
constexpr unsigned HY3A_LATE = 4, HY3A_LATE_CUT = 2;
/* A second segment in a CTA (queries, fold, record) costs more than this many pages.  The line was drawn when it cost about 6 us, before the
 * fold ran per head; 14 ragged batches since, us a layer with 0 / 5 / 12 pages, FP16, INT4: 14 rows up to 1 412 tokens x 8 heads
 * 17.2 / 12.0 / 12.0, 18.6 / 10.8 / 10.8; 30 up to 1 510 x 4 22.9 / 15.6 / 15.6, 30.8 / 13.7 / 13.6; 20 up to 9 594 x 4 43.2 / 43.4 / 34.8,
 * 38.2 / 38.2 / 20.3; 25 up to 1 020 x 4, INT4, 12.3 / 12.3 / 12.6; the others within 1 %.  So more than 5 would pay now for long rows. */
constexpr unsigned HY3A_STRADDLE_PAGES = 5;

/* Most pieces of a segment of p pages: every piece is a record to fetch and fold behind the last page, every page time of its CTA.  It
 * matters where few KV heads have many CTAs each.  The line was drawn when every record was a dependent step of the fold (0.11 us; a page 0.57);
 * the folding warp takes the first 32 in one step now, and a segment that keeps to 32 still gains most.  us a layer with 36 + p / 32 / without
 * a line / with this one, INT8, FP16, INT4:
 *   1 head, 20 000 tokens  11.3 / 23.3 / 10.3  11.5 / 21.0 / 11.1  11.6 / 22.6 / 10.3     1 head, 200 000  25.6 / 30.9 / 25.2  30.8 / 35.9 / 30.8  22.0 / 27.4 / 22.2
 *   2 heads, 60 000        17.1 / 22.2 / 17.6  21.1 / 24.3 / 22.0  15.3 / 19.6 / 15.8     4 heads, 20 000  16.6 / 16.6 / 11.5  16.8 / 16.8 / 13.1  14.8 / 14.8 / 11.0
 *   1 head, 60 000         14.5 / 24.7 / 15.9  17.7 / 26.0 / 18.3  14.6 / 23.1 / 15.3 */
HY3A_HD unsigned hy3a_most_pieces(unsigned p) { return 24u + p / 32u; }

/* Even pieces (FP16 / INT4 kernel): 2 to 32 rows with fewer than four CTAs per segment; four round well enough */
HY3A_HD bool hy3a_even_applies(int n, int G, unsigned grid) {
    return n >= 2 && n <= 32 && (unsigned)(n * G) < grid && (unsigned)(n * G) * 4u > grid;
}
/* Most pages that the bisection has to look at: with n rows, pieces of ceil(P / (cap - n + 1)) pages always fit, because
 * sum ceil(p / L) <= ceil(P / L) + n - 1; nor is more than the longest row of use.  n <= cap. */
HY3A_HD unsigned hy3a_piece_bound(unsigned P, unsigned cap, unsigned n, unsigned longest) {
    const unsigned d = cap - n + 1u, b = (P + d - 1u) / d;
    return b < longest ? b : longest;
}
/* The least L in [lo, hi] for which pieces(L) <= cap, by bisection; hi fits.  Exact, in at most log2(hi - lo) + 1 rounds: a search
 * stopped after 8 ends up to 17 % above the least with one very long row among short ones, and the rule below then refuses the
 * split (100 000 tokens and 9 x 128, 4 KV heads: INT4 82.0 us a layer that way, 27.5 with the least; FP16 63.1 and 44.0; 8 rows
 * of 2 718 to 7 075 tokens 21.1 and 20.8). */
template <class Pieces>
HY3A_HD unsigned hy3a_least_piece(unsigned lo, unsigned hi, unsigned cap, Pieces pieces) {
    while (lo < hi) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        if (pieces(mid) <= cap) hi = mid; else lo = mid + 1u;
    }
    return hi;
}
/* whether pieces of at most L of the P pages per head are kept, or units are dealt in equal contiguous ranges instead */
HY3A_HD bool hy3a_even_accepted(unsigned L, unsigned P, int G, unsigned grid) {
    const unsigned long long sum = (unsigned long long)P * (unsigned)G + grid - 1ull;
    const unsigned long long even = sum >> 32 ? sum / grid : (unsigned)sum / grid;      /* a 64-bit division costs hundreds of cycles */
    return L * 4ull <= even * 5ull + 4ull || L <= even + HY3A_STRADDLE_PAGES;
}

#endif
