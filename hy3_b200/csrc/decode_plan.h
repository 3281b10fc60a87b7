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
/* a second segment in a CTA (queries, fold, record: about 6 us) costs more than this many pages */
constexpr unsigned HY3A_STRADDLE_PAGES = 5;

/* Most pieces of a segment of p pages: every piece is a record to fetch and fold (0.11 us behind the last page), every page 0.57 us of
 * its CTA, so beyond some sqrt(5 p) more pieces cost more than they save; this line stays near it from 100 to 3 000 pages.  It
 * matters where few KV heads have many CTAs each.  us a layer without / with it, INT8, FP16, INT4:
 *   1 head, 20 000 tokens  23.2 -> 10.7  28.1 -> 14.1  30.7 -> 13.1     1 head, 200 000  29.4 -> 26.3  45.2 -> 39.6  39.2 -> 27.3
 *   2 heads, 60 000        19.9 -> 15.8  27.0 -> 25.5  24.6 -> 18.0     4 heads, 20 000  14.6 -> 11.4  19.7 -> 16.7  18.5 -> 13.4 */
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
