// qx_sl.cuh -- the straight-line class kernels over a handle's quartet lists: 2^lg lanes
// per quartet, lg by the quartet's primitives.
//
// A lane that walks a quartet of 4,096 primitives takes a hundred times as long as its
// average neighbour, and with one lane count per launch such quartets were its tail: ten
// atoms, (ds|ps): FP64 pipe 52% busy while blocks ran, 20% over the launch.  The
// processing order has the largest quartets first, so a launch is cut into segments of
// equal lane count that keep a lane's share of primitives below a bound (SlArgs).
//
// J/K: the quartet's block regroups into the six contractions of qx_jk.cuh inside the lane
// that owns it: every integral, as the transfer forms it, is folded into the sums over
// its quartet's J and K entries, which then take one atomic per entry and image instead
// of one per integral and image -- 24 instead of 48 for (ps|ss), 114 instead of 864 for
// (dp|ps).  Summing the entries that neighbouring lanes share (J_AB, K_AC) over the warp
// first changed nothing: the recurrences bound these kernels, not the atomics.
// Ten atoms unique 4.18 -> 3.94 ms, dense (8 atoms) 2.05 -> 1.98 ms, J/K of 12 atoms
// 18.4 ms integral by integral -> 15.4 by blocks -> 13.2 by segments.
#pragma once
#include "qx_kernels.cuh"
#include "qx_segments.h"

namespace qx {

// Segment k holds the quartets [first[k], first[k + 1]) of the processing order, 2^lg[k]
// lanes each, from block start[k] on.
struct SlArgs {
    EriArgs e;
    int nseg = 1;
    long long start[SL_SEGS] = {};
    long long first[SL_SEGS + 1] = {};
    int lg[SL_SEGS] = {};
};

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

template <int LA, int LB, int LC, int LD, int MODE>
__global__ void __launch_bounds__(AccPolicy<EriCls<LA, LB, LC, LD>::NACC>::bs) k_sl(SlArgs sa) {
    using C = EriCls<LA, LB, LC, LD>;
    using Pol = AccPolicy<C::NACC>;
    static_assert(Pol::kind != ACC_GLOBAL, "straight-line classes keep their accumulators on the SM");
    int seg = sa.nseg - 1;  // block-uniform
    while (seg > 0 && (long long)blockIdx.x < sa.start[seg]) --seg;
    EriArgs a = sa.e;
    a.log2g = sa.lg[seg];
    const long long gt = ((long long)blockIdx.x - sa.start[seg]) * Pol::bs + threadIdx.x;
    long long qi = sa.first[seg] + (gt >> a.log2g);
    const int sub = (int)(gt & ((1 << a.log2g) - 1));
    bool active = qi < sa.first[seg + 1];
    if (active) qi = list_index(a, qi);
    // every lane stays to the end: the group reduction shuffles over the full warp
    const int2 pq = active ? a.quartets[qi] : make_int2(0, 0);
    const PairInfo P = a.pairs[pq.x];
    const PairInfo Q = a.pairs[pq.y];
    if (MODE == MODE_JK && active && jk_screened(a, pq, P, Q)) active = false;  // group-uniform
    auto go = [&](auto& acc) {
        contract_quartet<C>(a, P, Q, acc, sub, active);
        if (!active || sub) return;
        if constexpr (MODE == MODE_JK) finish_jk<C, LA, LB, LC, LD>(a, P, Q, pq, acc);
        else finish_quartet<C, LA, LB, LC, LD, MODE>(a, P, Q, pq, qi, acc);
    };
    if constexpr (Pol::kind == ACC_REG) {
        RegAcc<C::NACC> acc;
        go(acc);
    } else {
        extern __shared__ double smem_acc[];
        StridedAcc acc{smem_acc + threadIdx.x, Pol::bs};
        go(acc);
    }
}

template <int LA, int LB, int LC, int LD, int MODE>
void launch_sl_mode(SlArgs& sa, cudaStream_t s) {
    using Pol = AccPolicy<EriCls<LA, LB, LC, LD>::NACC>;
    long long blocks = 0;
    for (int k = 0; k < sa.nseg; ++k) {
        sa.start[k] = blocks;
        blocks += (((sa.first[k + 1] - sa.first[k]) << sa.lg[k]) + Pol::bs - 1) / Pol::bs;
    }
    if (blocks == 0) return;
    auto k = k_sl<LA, LB, LC, LD, MODE>;
    if (Pol::smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, Pol::smem);
    k<<<(unsigned)blocks, Pol::bs, Pol::smem, s>>>(sa);
}

template <int LA, int LB, int LC, int LD>
void launch_sl(SlArgs& sa, int mode, cudaStream_t s) {
    if (mode == MODE_DENSE) return launch_sl_mode<LA, LB, LC, LD, MODE_DENSE>(sa, s);
    if (mode == MODE_UNIQUE) return launch_sl_mode<LA, LB, LC, LD, MODE_UNIQUE>(sa, s);
    if (mode == MODE_JK) return launch_sl_mode<LA, LB, LC, LD, MODE_JK>(sa, s);
    if constexpr (LA == LC && LB == LD) launch_sl_mode<LA, LB, LC, LD, MODE_SCHWARZ>(sa, s);
}

}  // namespace qx
