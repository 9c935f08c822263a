// qx_jk.cuh -- J and K of one quartet's block of integrals.
#pragma once
#include "qx_kernels.cuh"

namespace qx {

// Adds a quartet's block to J and K: the up-to-8 images of each integral regroup into
// six block contractions with D (J_AB over the ket, J_CD over the bra, and the four
// exchange blocks), so each touched entry takes one atomic per quartet instead of one per
// integral and image.  G(o) is integral o = ((a NB + b) NC + c) ND + d; thread tid of nth.
template <int NA, int NB, int NC, int ND, class Block>
__device__ __forceinline__ void jk_block(double* __restrict__ J, double* __restrict__ K, const double* __restrict__ D,
                                         long long n, const PairInfo& P, const PairInfo& Q, bool s12, bool s34,
                                         bool sPQ, int tid, int nth, Block&& G) {
    const long long bA = P.bf1, bB = P.bf2, bC = Q.bf1, bD = Q.bf2;
    auto at = [&](int ia, int ib, int ic, int id) { return G(((ia * NB + ib) * NC + ic) * ND + id); };
    auto Dv = [&](long long r, long long c) { return __ldg(D + r * n + c); };
    constexpr int nJA = NA * NB, nJC = NC * ND, nK1 = NA * NC, nK2 = NB * NC, nK3 = NA * ND, nK4 = NB * ND;
    for (int e = tid; e < nJA + nJC + nK1 + nK2 + nK3 + nK4; e += nth) {
        int r = e;
        double x = 0.0;
        if (r < nJA) {  // J_ij += (1 + s34) sum_kl G D_kl, and J_ji with s12
            const int ia = r / NB, ib = r % NB;
            for (int ic = 0; ic < NC; ++ic)
                for (int id = 0; id < ND; ++id) x = fma(at(ia, ib, ic, id), Dv(bC + ic, bD + id), x);
            x *= 1.0 + s34;
            atomicAdd(J + (bA + ia) * n + bB + ib, x);
            if (s12) atomicAdd(J + (bB + ib) * n + bA + ia, x);
            continue;
        }
        r -= nJA;
        if (r < nJC) {  // with sPQ: J_kl += (1 + s12) sum_ij G D_ij, and J_lk with s34
            if (!sPQ) continue;
            const int ic = r / ND, id = r % ND;
            for (int ia = 0; ia < NA; ++ia)
                for (int ib = 0; ib < NB; ++ib) x = fma(at(ia, ib, ic, id), Dv(bA + ia, bB + ib), x);
            x *= 1.0 + s12;
            atomicAdd(J + (bC + ic) * n + bD + id, x);
            if (s34) atomicAdd(J + (bD + id) * n + bC + ic, x);
            continue;
        }
        r -= nJC;
        if (r < nK1) {  // K_ik += sum_jl G D_jl (and K_ki with sPQ)
            const int ia = r / NC, ic = r % NC;
            for (int ib = 0; ib < NB; ++ib)
                for (int id = 0; id < ND; ++id) x = fma(at(ia, ib, ic, id), Dv(bB + ib, bD + id), x);
            atomicAdd(K + (bA + ia) * n + bC + ic, x);
            if (sPQ) atomicAdd(K + (bC + ic) * n + bA + ia, x);
            continue;
        }
        r -= nK1;
        if (r < nK2) {  // with s12: K_jk += sum_il G D_il (and K_kj with sPQ)
            if (!s12) continue;
            const int ib = r / NC, ic = r % NC;
            for (int ia = 0; ia < NA; ++ia)
                for (int id = 0; id < ND; ++id) x = fma(at(ia, ib, ic, id), Dv(bA + ia, bD + id), x);
            atomicAdd(K + (bB + ib) * n + bC + ic, x);
            if (sPQ) atomicAdd(K + (bC + ic) * n + bB + ib, x);
            continue;
        }
        r -= nK2;
        if (r < nK3) {  // with s34: K_il += sum_jk G D_jk (and K_li with sPQ)
            if (!s34) continue;
            const int ia = r / ND, id = r % ND;
            for (int ib = 0; ib < NB; ++ib)
                for (int ic = 0; ic < NC; ++ic) x = fma(at(ia, ib, ic, id), Dv(bB + ib, bC + ic), x);
            atomicAdd(K + (bA + ia) * n + bD + id, x);
            if (sPQ) atomicAdd(K + (bD + id) * n + bA + ia, x);
            continue;
        }
        r -= nK3;
        if (!(s12 && s34)) continue;  // with both: K_jl += sum_ik G D_ik (and K_lj with sPQ)
        const int ib = r / ND, id = r % ND;
        for (int ia = 0; ia < NA; ++ia)
            for (int ic = 0; ic < NC; ++ic) x = fma(at(ia, ib, ic, id), Dv(bA + ia, bC + ic), x);
        atomicAdd(K + (bB + ib) * n + bD + id, x);
        if (sPQ) atomicAdd(K + (bD + id) * n + bB + ib, x);
    }
}

}  // namespace qx
