// Host build of the launch-segment arithmetic (test infrastructure).
#include "qx_segments.h"

using namespace qx;

extern "C" int seg_pow(void) { return SEG_POW; }
extern "C" int seg_key_of(long long n) { return seg_key(n); }
extern "C" void seg_prefix_of(const long long* hist, int nkey, long long* prefix) { seg_prefix(hist, nkey, prefix); }
extern "C" int sl_segs(long long nq, long long prims, long long max_prims, const long long* prefix, int lg,
                       long long* first, int* lgs) {
    return sl_segments(nq, prims, max_prims, prefix, lg, first, lgs);
}
extern "C" int tile_segs(long long nq, long long share, long long max_prims, const long long* prefix, int cap,
                         long long* first, long long* start, long long* blocks) {
    return tile_segments(nq, share, max_prims, prefix, cap, first, start, blocks);
}
