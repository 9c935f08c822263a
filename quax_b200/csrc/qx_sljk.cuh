// qx_sljk.cuh -- direct J/K of the straight-line classes (2^log2g lanes per quartet).
//
// The quartet's block regroups into the six contractions of qx_jk.cuh inside the lane
// that owns it: every integral, as the transfer forms it, is folded into the sums over
// its quartet's J and K entries, which then take one atomic per entry and image instead
// of one per integral and image -- 24 instead of 48 for (ps|ss), 114 instead of 864 for
// (dp|ps).  Those atomics bound the straight-line classes; now their recurrences do, and
// summing the entries that neighbouring lanes share (J_AB, K_AC) over the warp first
// changed nothing.  12 atoms (n = 160): J/K 18.4 -> 15.1 ms.
#pragma once
#include "qx_kernels.cuh"

namespace qx {

template <int NA, int NB, int NC, int ND>
struct SlJkSums {
    const double *dAB, *dCD, *dAC, *dAD, *dBC, *dBD;  // D blocks, row stride n
    long long n;
    double jAB[NA * NB], jCD[NC * ND], kAC[NA * NC], kAD[NA * ND], kBC[NB * NC], kBD[NB * ND];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < NA * NB; ++i) jAB[i] = 0.0;
#pragma unroll
        for (int i = 0; i < NC * ND; ++i) jCD[i] = 0.0;
#pragma unroll
        for (int i = 0; i < NA * NC; ++i) kAC[i] = 0.0;
#pragma unroll
        for (int i = 0; i < NA * ND; ++i) kAD[i] = 0.0;
#pragma unroll
        for (int i = 0; i < NB * NC; ++i) kBC[i] = 0.0;
#pragma unroll
        for (int i = 0; i < NB * ND; ++i) kBD[i] = 0.0;
    }
    // integral k = ((a NB + b) NC + c) ND + d; k is a literal at every call
    __device__ __forceinline__ void operator()(int k, double v) {
        const int d = k % ND, c = (k / ND) % NC, b = (k / (ND * NC)) % NB, a = k / (ND * NC * NB);
        jAB[a * NB + b] = fma(v, __ldg(dCD + c * n + d), jAB[a * NB + b]);
        jCD[c * ND + d] = fma(v, __ldg(dAB + a * n + b), jCD[c * ND + d]);
        kAC[a * NC + c] = fma(v, __ldg(dBD + b * n + d), kAC[a * NC + c]);
        kAD[a * ND + d] = fma(v, __ldg(dBC + b * n + c), kAD[a * ND + d]);
        kBC[b * NC + c] = fma(v, __ldg(dAD + a * n + d), kBC[b * NC + c]);
        kBD[b * ND + d] = fma(v, __ldg(dAC + a * n + c), kBD[b * ND + d]);
    }
};

// M_ij += x (and M_ji with `both`) over an NI x NJ block.
template <int NI, int NJ>
__device__ __forceinline__ void sl_jk_add(double* __restrict__ M, long long n, long long i0, long long j0, bool both,
                                          double f, const double* x) {
#pragma unroll
    for (int i = 0; i < NI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const double v = f * x[i * NJ + j];
            atomicAdd(M + (i0 + i) * n + j0 + j, v);
            if (both) atomicAdd(M + (j0 + j) * n + i0 + i, v);
        }
}

template <class C, int LA, int LB, int LC, int LD, class Acc>
__device__ __noinline__ void finish_jk(const EriArgs& a, const PairInfo& P, const PairInfo& Q, int2 pq, Acc acc) {
    constexpr int NA = ncart_h(LA), NB = ncart_h(LB), NC = ncart_h(LC), ND = ncart_h(LD);
    const bool s12 = P.s1 != P.s2, s34 = Q.s1 != Q.s2, sPQ = pq.x != pq.y;
    const long long n = a.n, A = P.bf1, B = P.bf2, Cc = Q.bf1, Dd = Q.bf2;
    const double* D = a.dens;
    SlJkSums<NA, NB, NC, ND> st;
    st.dAB = D + A * n + B;
    st.dCD = D + Cc * n + Dd;
    st.dAC = D + A * n + Cc;
    st.dAD = D + A * n + Dd;
    st.dBC = D + B * n + Cc;
    st.dBD = D + B * n + Dd;
    st.n = n;
    st.clear();
    C::hrr(acc, st, P.ABx, P.ABy, P.ABz, Q.ABx, Q.ABy, Q.ABz);
    sl_jk_add<NA, NB>(a.out, n, A, B, s12, 1.0 + s34, st.jAB);
    if (sPQ) sl_jk_add<NC, ND>(a.out, n, Cc, Dd, s34, 1.0 + s12, st.jCD);
    sl_jk_add<NA, NC>(a.out2, n, A, Cc, sPQ, 1.0, st.kAC);
    if (s12) sl_jk_add<NB, NC>(a.out2, n, B, Cc, sPQ, 1.0, st.kBC);
    if (s34) sl_jk_add<NA, ND>(a.out2, n, A, Dd, sPQ, 1.0, st.kAD);
    if (s12 && s34) sl_jk_add<NB, ND>(a.out2, n, B, Dd, sPQ, 1.0, st.kBD);
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(AccPolicy<EriCls<LA, LB, LC, LD>::NACC>::bs) k_sljk(EriArgs a) {
    using C = EriCls<LA, LB, LC, LD>;
    using Pol = AccPolicy<C::NACC>;
    const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long qi = gt >> a.log2g;
    const int sub = (int)(gt & ((1 << a.log2g) - 1));
    bool active = qi < a.nq;
    if (active) qi = list_index(a, qi);
    // every lane stays to the end: the group reduction shuffles over the full warp
    const int2 pq = active ? a.quartets[qi] : make_int2(0, 0);
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    if (active && jk_screened(a, pq, P, Q)) active = false;  // group-uniform
    auto go = [&](auto& acc) {
        contract_quartet<C>(a, P, Q, acc, sub, active);
        if (active && sub == 0) finish_jk<C, LA, LB, LC, LD>(a, P, Q, pq, acc);
    };
    if constexpr (Pol::kind == ACC_REG) {
        RegAcc<C::NACC> acc;
        go(acc);
    } else if constexpr (Pol::kind == ACC_SMEM) {
        extern __shared__ double smem_acc[];
        StridedAcc acc{smem_acc + threadIdx.x, Pol::bs};
        go(acc);
    } else {
        StridedAcc acc{a.scratch + gt, (long long)gridDim.x * blockDim.x};
        go(acc);
    }
}

template <int LA, int LB, int LC, int LD>
void launch_sljk(const EriArgs& a, cudaStream_t s) {
    using Pol = AccPolicy<EriCls<LA, LB, LC, LD>::NACC>;
    const long long nb = ((a.nq << a.log2g) + Pol::bs - 1) / Pol::bs;
    if (nb == 0) return;
    auto k = k_sljk<LA, LB, LC, LD>;
    if (Pol::smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Pol::smem);
    k<<<(unsigned)nb, Pol::bs, Pol::smem, s>>>(a);
}

}  // namespace qx
