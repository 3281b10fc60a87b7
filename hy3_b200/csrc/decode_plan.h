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

/* Even pieces (FP16 / INT4 kernel): 2 to 32 rows with fewer than four CTAs per segment; four round well enough */
HY3A_HD bool hy3a_even_applies(int n, int G, unsigned grid) {
    return n >= 2 && n <= 32 && (unsigned)(n * G) < grid && (unsigned)(n * G) * 4u > grid;
}
/* The least L in [lo, hi] for which pieces(L) <= cap, by bisection; hi fits. */
template <class Pieces>
HY3A_HD unsigned hy3a_least_piece(unsigned lo, unsigned hi, unsigned cap, Pieces pieces) {
    for (int i = 0; i < 8 && lo < hi; i++) {
        const unsigned mid = (lo + hi) >> 1;
        if (pieces(mid) <= cap) hi = mid; else lo = mid + 1u;
    }
    return hi;
}
/* whether pieces of at most L of the P pages per head are kept, or units are dealt in equal contiguous ranges instead */
HY3A_HD bool hy3a_even_accepted(unsigned L, unsigned P, int G, unsigned grid) {
    const unsigned long long even = ((unsigned long long)P * (unsigned)G + grid - 1ull) / grid;
    return L * 4ull <= even * 5ull + 4ull || L <= even + HY3A_STRADDLE_PAGES;
}

#endif
