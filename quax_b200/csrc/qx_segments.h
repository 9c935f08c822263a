// qx_segments.h -- how a class's quartets are ordered by their primitives and cut into
// launch segments (host arithmetic only; a class may hold more than 2^31 quartets, so
// every count and position is 64 bits).
#pragma once
#include <algorithm>

namespace qx {

// Powers of two a count is compared with: 2^0 .. 2^24, the primitives of a quartet of four
// shells of 64.
constexpr int SEG_POW = 25;

// Order key of a primitive count: every count of its own up to 64, above in steps of 1/64,
// none of which spans a power of two -- 1,217 keys at most, 449 up to 4,096 primitives, so
// that the counts of every class and host thread stay small (the orders of ten atoms: 1.1 ms;
// with a key per count and a thread per 16,384 quartets 2.1).
inline int seg_key(long long n) {
    const long long m = std::min(n, 1LL << 24) - 1;
    if (m < 64) return (int)m;
    const int e = 63 - __builtin_clzll((unsigned long long)m);
    return 64 + (e - 6) * 64 + (int)((m >> (e - 6)) & 63);
}

// From the histogram over keys 0 .. nkey - 1 (summed over threads already): the quartets
// with more than 2^k primitives.
inline void seg_prefix(const long long* hist, int nkey, long long* prefix) {
    int b = nkey;
    long long s = 0;
    for (int k = SEG_POW - 1; k >= 0; --k) {
        const int from = k < 24 ? seg_key((1LL << k) + 1) : nkey;
        for (; b > from; --b) s += hist[b - 1];
        prefix[k] = s;
    }
}

constexpr int SL_SEGS = 6;  // 1 to 32 lanes

// Segments of a straight-line class: segment k holds the quartets [first[k], first[k + 1])
// of the processing order, 2^lg[k] lanes each, so that a lane walks at most `share`
// primitives -- what each of the GPU's resident threads (148 SMs, about 768) gets of the
// class, at least 64, or 16 where there is not one primitive per thread and only latency
// counts.  Smaller shares cost more in the transfer, which one lane of a group runs, than
// they save in the tail, which other classes fill (ten atoms unique 4.21 ms at 16, 3.94 at
// 64, 4.12 at 256; 12 atoms J/K 13.8, 13.2, 13.2; H2O 30 us at 16, 48 at 64).  prefix is
// null without a processing order; then all quartets take the lanes of the largest one
// (equal counts) or `lg` (>= 0: lanes by the class's average).  Returns the segments.
inline int sl_segments(long long nq, long long prims, long long max_prims, const long long* prefix, int lg,
                       long long* first, int* lgs) {
    first[0] = 0;
    if (!prefix && lg >= 0) {
        first[1] = nq;
        lgs[0] = lg;
        return 1;
    }
    const long long threads = 148LL * 768;
    const long long share = prims < threads ? 16LL : std::max(64LL, prims / threads);
    int low = 4;
    while (low < SEG_POW - 1 && (2LL << low) <= share) ++low;
    int top = 0;  // lanes of the largest quartets
    while (top < SL_SEGS - 1 && (max_prims - 1) >> (low + top)) ++top;
    if (!prefix) {
        first[1] = nq;
        lgs[0] = top;
        return 1;
    }
    for (int k = 0; k <= top; ++k) {  // largest quartets, and most lanes, first
        lgs[k] = top - k;
        first[k + 1] = k == top ? nq : prefix[low + top - k - 1];
    }
    return top + 1;
}

// Segments of a tile launch: segment j holds the quartets [first[j], ...) of the
// processing order with 2^j blocks each, from block start[j] on; the largest quartets have
// the highest j and come first.  A block takes at most `share` primitives, rounded down to
// a power of two; at most `cap` parts.  Without a prefix all quartets count as the
// largest.  Returns the number of segments; `blocks` their sum.
inline int tile_segments(long long nq, long long share, long long max_prims, const long long* prefix, int cap,
                         long long* first, long long* start, long long* blocks) {
    int low = 0;
    while (low < SEG_POW - 1 && (2LL << low) <= share) ++low;
    int nseg = 1;
    while (nseg < SEG_POW && (1LL << nseg) <= cap && (max_prims - 1) >> (low + nseg - 1)) ++nseg;
    long long from = 0;
    *blocks = 0;
    for (int j = nseg - 1; j >= 0; --j) {
        first[j] = from;
        start[j] = *blocks;
        long long to = nq;
        if (j > 0 && prefix) to = low + j - 1 < SEG_POW ? prefix[low + j - 1] : 0;
        to = std::max(from, to);
        *blocks += (to - from) << j;
        from = to;
    }
    return nseg;
}

}  // namespace qx
