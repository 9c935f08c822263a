// qx_plain.cuh -- Rys quadrature of plain integrals, every class up to (ff|ff), in the
// block organisation of qx_tile.cuh.
//
// Method.  (ab|cd) of a primitive quartet is sum_r w_r Ix Iy Iz over the Rys nodes, the
// 1-D factors by the recurrences of qx_rys.cuh and the transfer I(a,b+1) = I(a+1,b) +
// AB I(a,b) of each side in one dimension and per root.  Rounding errors of the 1-D
// recurrence enter I(a+k) of all k alike and pass the transfer with their own size;
// applied once to the contracted (e0|f0) sums -- 1.5 to 2.7 times fewer operations in the
// sums, and what the Obara-Saika programs do -- the transfer multiplies the independent
// rounding of every sum by up to (|AB| / |PB|)^b: (33|22) and (33|33) came out 3 to 4 times
// further from an 80-bit evaluation (median over quartets), single quartets up to 70 times.
//
// Organisation.  A block owns (quartet, part of its primitives).  Per batch of PB
// primitives: nodes and weights (one thread per function), the 1-D tables with the bra
// transferred (one thread per primitive, root and direction), the ket transfer in place
// (one thread per table column), then the sums: a lane owns one (c, d) and one of NP
// primitives of the batch, a warp one chunk of the (a, b) -- a set of a_x values, compile
// time, so that the chunk's sums live in registers and one load of a column serves them.
//
// Parts of a quartet meet in the outputs.  J and K take atomics, as always.  A dense,
// unique or Schwarz value is written once, by one thread: the parts form a cluster and add their
// blocks over distributed shared memory in the order of the parts, so that the images of
// an integral are equal to the bit and repeated calls give the same tensor.
//
// What bounds it: FP64 latency in the sums and the barriers around the tables.  Six atoms
// with f shells, J/K 3.5 ms; table kernels 14.0 (they read three four-index entries per
// component and root from shared memory, and walked all primitives of a quartet on one
// team), transfer after the contraction 2.9.  Unique integrals of four such atoms 4.8 ms,
// transfer after the contraction and atomics 3.9.
#pragma once
#include <cooperative_groups.h>

#include "qx_jk.cuh"
#include "qx_tile.cuh"

namespace qx {

template <int LA, int LB, int LC, int LD>
struct PlainCls {
    static constexpr int la = LA, lb = LB, lc = LC, ld = LD;
    static constexpr bool DER = false;  // tl_nodes
    static constexpr int SCP = 0;
    static constexpr int NA = ncart_h(LA), NB = ncart_h(LB), NC = ncart_h(LC), ND = ncart_h(LD);
    static constexpr int NAB = NA * NB, NCD = NC * ND, NCOMP = NAB * NCD;
    static constexpr int NR = (LA + LB + LC + LD) / 2 + 1;
    static constexpr int NI = LA + LB + 1, NK = LC + LD + 1;
    // a unit (primitive, root, direction): columns c (LD + 1) + d of BRA entries a (LB + 1)
    // + b, padded to 2 mod 4 doubles so that columns start on different 16-byte units
    static constexpr int BRA = (LA + 1) * (LB + 1), KET = (LC + 1) * (LD + 1);
    static constexpr int BP = (BRA + 1) / 4 * 4 + 2;
    static_assert(BP >= BRA && BP % 4 == 2, "column padding");
    static constexpr int UNIT = KET * BP, PER_PRIM = 3 * NR * UNIT;
    // chunks of the (a, b) by a_x: a thread's sums next to its columns must fit its registers
    static constexpr int BUDGET = 56;
    QX_HD static constexpr int per_ax(int x) { return (LA - x + 1) * NB; }
    static constexpr int NCH = (NAB + BUDGET - 1) / BUDGET;
    struct Chunks {
        int mask[4];
        int most;
    };
    QX_HD static constexpr Chunks chunks() {
        Chunks c{};
        int load[4] = {0, 0, 0, 0};
        for (int x = 0; x <= LA; ++x) {  // largest first onto the least loaded
            int b = 0;
            for (int k = 1; k < NCH; ++k)
                if (load[k] < load[b]) b = k;
            c.mask[b] |= 1 << x;
            load[b] += per_ax(x);
        }
        for (int k = 0; k < NCH; ++k)
            if (load[k] > c.most) c.most = load[k];
        return c;
    }
    QX_HD static constexpr int MASK(int k) { return chunks().mask[k]; }
    static constexpr int NSLOT = chunks().most;
    // lanes: NF, NCHB and NP as TileRole reads them
    static constexpr int NF = NCD, NCHB = NCH, WMIN = (NF + 31) / 32;
    static_assert(NCH * WMIN <= TILE_MAXW && NCH <= LA + 1, "the block holds every chunk");
    static constexpr int WPC = tl_wpc(NF, WMIN, NCHB);
    static constexpr int W = WPC * NCHB, NT = 32 * W;
    static constexpr int NP = 32 * WPC / NF;
    static constexpr int PB = tl_pb(NP, NR, NT, PER_PRIM);
    // shared memory, in doubles: nodes and weights, maxima, then a region that holds the
    // batch's tables or, after the primitives, the block of integrals with RSUB more of
    // them for the sum over the NP primitives
    static constexpr int UW = 2 * NR * PB;
    static constexpr int HEAD = (UW + TILE_MAXW + 1) / 2 * 2;
    static constexpr int TABS = PB * PER_PRIM, BLOCKS = NCOMP * (NP > 1 ? 2 : 1);
    static constexpr int REGION = TABS > BLOCKS ? TABS : BLOCKS;
    static constexpr int RSUB = (REGION - NCOMP) / NCOMP < 1 ? 1 : (REGION - NCOMP) / NCOMP;
    static constexpr int SMEM = 8 * (HEAD + REGION);
    static_assert(SMEM <= 227 * 1024, "tables exceed shared memory");
};

// ------------------------------------------------------------------ phases -----
// 2-D tables of the batch with the bra transferred: unit = (primitive * NR + root) * 3 +
// direction, row k (ket quanta) at k * BP.
template <class C>
QX_HD inline void pl_tables(const TileQuartet& w, const PrimPair* bra, const PrimPair* ket, int t0, int nb,
                            const double* uw, double* tab, int tid, int nth) {
    const int nk = w.Q.nprim;
    for (int i = tid; i < nb * C::NR * 3; i += nth) {
        const int p = i / (3 * C::NR), rest = i - p * 3 * C::NR, r = rest / 3, x = rest - 3 * r;
        const int t = t0 + p, ib = t / nk, ik = t - ib * nk;
        const PrimPair &a = bra[ib], &c = ket[ik];
        const double rs = 1.0 / (a.zeta + c.zeta);
        const double u = uw[p * 2 * C::NR + r];
        const double qe = u * c.zeta * rs, pe = u * a.zeta * rs;
        const double B00 = 0.5 * u * rs, B10 = a.oo2z * (1.0 - qe), B01 = c.oo2z * (1.0 - pe);
        const double PA = x == 0 ? a.PAx : (x == 1 ? a.PAy : a.PAz), QC = x == 0 ? c.PAx : (x == 1 ? c.PAy : c.PAz);
        const double PQ = x == 0 ? a.Px - c.Px : (x == 1 ? a.Py - c.Py : a.Pz - c.Pz);
        const double AB = x == 0 ? w.P.ABx : (x == 1 ? w.P.ABy : w.P.ABz);
        const double C00 = PA - qe * PQ, D00 = QC + pe * PQ;
        double* o = tab + (size_t)i * C::UNIT;
        double cur[C::NI], prev[C::NI];
        cur[0] = x == 2 ? uw[p * 2 * C::NR + C::NR + r] : 1.0;
        if constexpr (C::NI > 1) cur[1] = C00 * cur[0];
#pragma unroll
        for (int j = 2; j < C::NI; ++j) cur[j] = fma(C00, cur[j - 1], (j - 1) * B10 * cur[j - 2]);
#pragma unroll
        for (int j = 0; j < C::NI; ++j) prev[j] = 0.0;
#pragma unroll
        for (int k = 0; k < C::NK; ++k) {
            if (k > 0) {
                const double kb = (k - 1) * B01;
                double nxt[C::NI];
#pragma unroll
                for (int j = 0; j < C::NI; ++j) {
                    double v = D00 * cur[j];
                    if (k > 1) v = fma(kb, prev[j], v);
                    if (j > 0) v = fma(j * B00, cur[j - 1], v);
                    nxt[j] = v;
                }
#pragma unroll
                for (int j = 0; j < C::NI; ++j) {
                    prev[j] = cur[j];
                    cur[j] = nxt[j];
                }
            }
            double lev[C::NI];
#pragma unroll
            for (int j = 0; j < C::NI; ++j) lev[j] = cur[j];
#pragma unroll
            for (int b = 0; b <= C::lb; ++b) {
#pragma unroll
                for (int j = 0; j <= C::la; ++j) o[k * C::BP + j * (C::lb + 1) + b] = lev[j];
#pragma unroll
                for (int j = 0; j + 1 + b < C::NI; ++j) lev[j] = fma(AB, lev[j], lev[j + 1]);
            }
        }
    }
}

// Ket transfer: item = (unit, bra entry); its NK rows become the KET columns' entries, in
// place (a thread reads its rows before it writes).
template <class C>
QX_HD inline void pl_ket(const TileQuartet& w, int nb, double* tab, int tid, int nth) {
    for (int i = tid; i < nb * C::NR * 3 * C::BRA; i += nth) {
        const int u = i / C::BRA, x = u % 3;
        const double CD = x == 0 ? w.Q.ABx : (x == 1 ? w.Q.ABy : w.Q.ABz);
        double* o = tab + (size_t)u * C::UNIT + (i - u * C::BRA);
        double lev[C::NK];
#pragma unroll
        for (int k = 0; k < C::NK; ++k) lev[k] = o[k * C::BP];
#pragma unroll
        for (int d = 0; d <= C::ld; ++d) {
#pragma unroll
            for (int k = 0; k <= C::lc; ++k) o[(k * (C::ld + 1) + d) * C::BP] = lev[k];
#pragma unroll
            for (int k = 0; k + 1 + d < C::NK; ++k) lev[k] = fma(CD, lev[k], lev[k + 1]);
        }
    }
}

// Entries [lo, hi) of a column, 16 bytes at a time.
template <int LO, int HI, int N>
QX_HD inline void pl_col(const double* p, double (&v)[N]) {
#ifdef __CUDA_ARCH__
#pragma unroll
    for (int i = LO / 2 * 2; i < HI; i += 2) {
        const double2 t = *reinterpret_cast<const double2*>(p + i);
        v[i] = t.x;
        if (i + 1 < N) v[i + 1 < N ? i + 1 : i] = t.y;
    }
#else
    for (int i = LO; i < HI; ++i) v[i] = p[i];
#endif
}

// Cartesian quanta of component k of a shell.
QX_HD inline void pl_cart(int l, int k, int& x, int& y, int& z) {
    int m = 0;
    while ((m + 1) * (m + 2) / 2 <= k) ++m;
    z = k - m * (m + 1) / 2;
    y = m - z;
    x = l - m;
}

// Columns of (c, d)'s quanta in the three directions.
template <class C>
struct PlainLane {
    int x, y, z;
    QX_HD explicit PlainLane(int cd) {
        const int c = cd / C::ND, d = cd - c * C::ND;
        int cx, cy, cz, dx, dy, dz;
        pl_cart(C::lc, c, cx, cy, cz);
        pl_cart(C::ld, d, dx, dy, dz);
        x = (cx * (C::ld + 1) + dx) * C::BP;
        y = (cy * (C::ld + 1) + dy) * C::BP;
        z = (cz * (C::ld + 1) + dz) * C::BP;
    }
};

// Runs fn(slot, ab, ix, iy, iz) over a chunk's (a, b): column entries of the three
// directions (compile-time after unrolling).
template <class C, int M, class F>
QX_HD inline void pl_each(F&& fn) {
    constexpr int LA = C::la, LB = C::lb;
    int s = 0;
#pragma unroll
    for (int ax = 0; ax <= LA; ++ax) {
        if (!((M >> ax) & 1)) continue;
#pragma unroll
        for (int ay = 0; ay <= LA - ax; ++ay) {
            const int az = LA - ax - ay, ka = LA - ax;
#pragma unroll
            for (int bx = 0; bx <= LB; ++bx) {
#pragma unroll
                for (int by = 0; by <= LB - bx; ++by) {
                    const int bz = LB - bx - by, kb = LB - bx;
                    fn(s, (ka * (ka + 1) / 2 + az) * C::NB + kb * (kb + 1) / 2 + bz, ax * (LB + 1) + bx,
                       ay * (LB + 1) + by, az * (LB + 1) + bz);
                    ++s;
                }
            }
        }
    }
}

// One primitive of a thread's (c, d) and chunk: tab points at its NR * 3 units.
template <class C, int M>
QX_HD inline void pl_prim(const double* tab, const PlainLane<C>& l, double (&U)[C::NSLOT]) {
    // the a_x the chunk starts at bounds its a_y and a_z, and the columns' entries it reads
    constexpr int X0 = (M & 1) ? 0 : (M & 2) ? 1 : (M & 4) ? 2 : 3;
    constexpr int X1 = (M & 8) ? 3 : (M & 4) ? 2 : (M & 2) ? 1 : 0;
    constexpr int B = C::lb + 1, TOP = (C::la - X0 + 1) * B;
#pragma unroll 1
    for (int r = 0; r < C::NR; ++r) {
        const double* t = tab + r * 3 * C::UNIT;
        double X[C::BRA], Y[C::BRA], Z[C::BRA];
        pl_col<X0 * B, (X1 + 1) * B>(t + l.x, X);
        pl_col<0, TOP>(t + C::UNIT + l.y, Y);
        pl_col<0, TOP>(t + 2 * C::UNIT + l.z, Z);
        pl_each<C, M>([&](int s, int, int ix, int iy, int iz) { U[s] = fma(X[ix] * Y[iy], Z[iz], U[s]); });
    }
}

template <class C, int K>
QX_HD inline void pl_prim_chunk(int chunk, const double* tab, const PlainLane<C>& l, double (&U)[C::NSLOT]) {
    if constexpr (K + 1 < C::NCH) {
        if (chunk != K) {
            pl_prim_chunk<C, K + 1>(chunk, tab, l, U);
            return;
        }
    }
    pl_prim<C, C::MASK(K)>(tab, l, U);
}

// A thread's sums to the block of integrals.
template <class C, int K>
QX_HD inline void pl_store(int chunk, double* out, int cd, const double (&U)[C::NSLOT]) {
    if constexpr (K + 1 < C::NCH) {
        if (chunk != K) {
            pl_store<C, K + 1>(chunk, out, cd, U);
            return;
        }
    }
    pl_each<C, C::MASK(K)>([&](int s, int ab, int, int, int) { out[ab * C::NCD + cd] = U[s]; });
}

#ifndef TILE_HOST
// ------------------------------------------------------------------ device -----
template <class C>
struct PlainBounds {
    static constexpr int VALUES = C::NSLOT + 3 * C::BRA + 2;
    static constexpr int REGS0 = 2 * VALUES + 48;
    static constexpr int REGS = REGS0 > 255 ? 255 : (REGS0 < 64 ? 64 : REGS0);
    static constexpr int BY_REGS = 65536 / (C::NT * REGS), BY_SMEM = 227 * 1024 / (C::SMEM + 1024);
    static constexpr int B0 = BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM;
    static constexpr int MINB = B0 < 1 ? 1 : (B0 > 16 ? 16 : B0);
};

template <class C>
__global__ void __launch_bounds__(C::NT, PlainBounds<C>::MINB) k_plain(TileArgs ta, int mode) {
    constexpr int NT = C::NT;
    extern __shared__ __align__(16) double tile_sm[];
    __shared__ TileQuartet w;
    const int tid = threadIdx.x;
    double* uw = tile_sm;
    double* red = uw + C::UW;
    double* tab = tile_sm + C::HEAD;
    double* out = tab;  // after the primitives
    const EriArgs& a = ta.e;
    const TileBlock at = tile_block(ta);
    const long long n = a.n, qi = list_index(a, at.quartet);
    const int2 pq = a.quartets[qi];
    const int ntot = a.pairs[pq.x].nprim * a.pairs[pq.y].nprim;
    const int part = at.part, stride = at.parts * C::PB;
    // else the parts of a quartet are one cluster: all of them stay
    const bool joint = at.parts > 1 && mode != MODE_JK;
    if (!joint && part * C::PB >= ntot) return;  // whole block
    tile_pairs<NT>(a, pq, w, tid);
    __syncthreads();
    if (mode == MODE_JK && jk_screened(a, pq, w.P, w.Q)) return;  // block-uniform
    const TileRole<C> role(tid, 0);
    const PlainLane<C> lane(role.f);
    double U[C::NSLOT];
#pragma unroll
    for (int s = 0; s < C::NSLOT; ++s) U[s] = 0.0;
    const PrimPair* bra = a.prims + w.P.prim_off;
    const PrimPair* ket = a.prims + w.Q.prim_off;
    for (int t0 = part * C::PB; t0 < ntot; t0 += stride) {
        const int nb = min(C::PB, ntot - t0);
        tl_nodes<C>(ta.rys, w, bra, ket, t0, nb, uw, nullptr, tid, NT);
        __syncthreads();  // the previous batch's sums are done, too
        pl_tables<C>(w, bra, ket, t0, nb, uw, tab, tid, NT);
        __syncthreads();
        if constexpr (C::ld > 0) {
            pl_ket<C>(w, nb, tab, tid, NT);
            __syncthreads();
        }
        if (role.on)
            for (int p = role.sub; p < nb; p += C::NP)
                pl_prim_chunk<C, 0>(role.chunk, tab + (size_t)p * C::PER_PRIM, lane, U);
    }
    __syncthreads();
    if (role.on && role.sub == 0) pl_store<C, 0>(role.chunk, out, role.f, U);
    if constexpr (C::NP > 1) {  // the primitives side by side, in order
        double* side = out + C::NCOMP;
        for (int s0 = 1; s0 < C::NP; s0 += C::RSUB) {
            const int ns = min(C::RSUB, C::NP - s0);
            if (role.on && role.sub >= s0 && role.sub < s0 + ns)
                pl_store<C, 0>(role.chunk, side + (role.sub - s0) * C::NCOMP, role.f, U);
            __syncthreads();
            for (int i = tid; i < C::NCOMP; i += NT) {
                double v = out[i];
                for (int k = 0; k < ns; ++k) v += side[k * C::NCOMP + i];
                out[i] = v;
            }
            __syncthreads();
        }
    } else {
        __syncthreads();
    }
    const bool s12 = w.P.s1 != w.P.s2, s34 = w.Q.s1 != w.Q.s2, sPQ = pq.x != pq.y;
    if (mode == MODE_JK) {
        jk_block<C::NA, C::NB, C::NC, C::ND>(a.out, a.out2, a.dens, n, w.P, w.Q, s12, s34, sPQ, tid, NT,
                                             [&](int o) { return out[o]; });
        return;
    }
    namespace cg = cooperative_groups;
    if (joint) cg::this_cluster().sync();  // every part's block stands
    auto value = [&](int o) {
        if (!joint) return out[o];
        double v = 0.0;
        for (int k = 0; k < at.parts; ++k) v += *cg::this_cluster().map_shared_rank(out + o, k);
        return v;
    };
    if (mode == MODE_SCHWARZ) {
        if (part == 0) {  // block-uniform
            double mx = 0.0;
            if constexpr (C::NAB == C::NCD)
                for (int o = tid; o < C::NAB; o += NT) mx = fmax(mx, fabs(value(o * C::NCD + o)));
            for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
            if ((tid & 31) == 0) red[tid >> 5] = mx;
            __syncthreads();
            if (tid == 0) {
                for (int k = 1; k < C::W; ++k) mx = fmax(mx, red[k]);
                a.out[pq.x] = mx;
            }
        }
    } else {
        for (int o = part * NT + tid; o < C::NCOMP; o += at.parts * NT) {
            const double v = value(o);
            if (mode == MODE_UNIQUE) {
                a.out[a.base + (long long)o * a.nq + qi] = v;
                continue;
            }
            const int ab = o / C::NCD, cd = o - ab * C::NCD;
            const long long i = w.P.bf1 + ab / C::NB, j = w.P.bf2 + ab % C::NB, k = w.Q.bf1 + cd / C::ND,
                            l = w.Q.bf2 + cd % C::ND;
            dense_images(a.out, n, i, j, k, l, s12, s34, sPQ, v);
        }
    }
    if (joint) cg::this_cluster().sync();  // and is read before it goes
}

// Blocks of a class, by shares of primitives as in launch_tile.  All but J/K launch each
// segment by itself, for its cluster size, and at most the portable 8 parts.
template <class C>
void launch_plain(TileArgs& ta, int mode, long long nq, long long prims, long long max_prims, const long long* prefix,
                  cudaStream_t s) {
    if (nq <= 0) return;
    auto k = k_plain<C>;
    if (C::SMEM > 40 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    const long long share = std::max<long long>(2 * C::PB, prims / (148LL * PlainBounds<C>::MINB * 8) + 1);
    const int cap = mode == MODE_JK ? 1 << 24 : 8;
    long long blocks;
    ta.nseg = tile_segments(nq, share, max_prims, prefix, cap, ta.first, ta.start, &blocks);
    ta.lg0 = 0;
    if (mode == MODE_JK || ta.nseg == 1) {
        for (ta.block0 = 0; ta.block0 < blocks; ta.block0 += TILE_GRID)
            k<<<(unsigned)std::min(TILE_GRID, blocks - ta.block0), C::NT, C::SMEM, s>>>(ta, mode);
        return;
    }
    TileArgs one = ta;
    one.nseg = 1;
    for (int j = ta.nseg - 1; j >= 0; --j) {
        const long long nb = (j > 0 ? ta.start[j - 1] : blocks) - ta.start[j];
        one.lg0 = j;
        one.first[0] = ta.first[j];
        one.start[0] = 0;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 1u << j;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        for (one.block0 = 0; one.block0 < nb; one.block0 += TILE_GRID) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3((unsigned)std::min(TILE_GRID, nb - one.block0));
            cfg.blockDim = dim3(C::NT);
            cfg.dynamicSmemBytes = C::SMEM;
            cfg.stream = s;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            cudaLaunchKernelEx(&cfg, k, one, mode);
        }
    }
}
#endif  // TILE_HOST

}  // namespace qx
