// Host build of the primitive-pair selection (test infrastructure): the two exponents of
// every primitive pair of the shell pair (1, 0), s1 >= s2, that build_pairs keeps.
#include "qx_setup.h"

using namespace qx;

extern "C" int kept_pairs(const double* coords, const int* l, const int* nprim, const double* exps,
                          const double* coefs, double tol, double* out) {
    const int atom[2] = {0, 1};
    ShellTables t;
    std::string err;
    if (normalize_shells("kept_pairs", 2, 2, l, nprim, atom, exps, coefs, 3, t, err)) return -1;
    std::vector<PrimPair> prims;
    std::vector<PairInfo> pairs;
    std::vector<int> cls;
    build_pairs(t, coords, tol, prims, pairs, cls);
    const PairInfo& p = pairs[1];  // (1, 0), behind (0, 0)
    for (int k = 0; k < p.nprim; ++k) {
        const PrimPair& q = prims[p.prim_off + k];
        const bool first = p.s1 == 0;  // alpha belongs to the shell of higher angular momentum
        out[2 * k] = first ? q.alpha : q.zeta - q.alpha;      // shell 0
        out[2 * k + 1] = first ? q.zeta - q.alpha : q.alpha;  // shell 1
    }
    return p.nprim;
}
