// qx_tile.cuh -- the adjoint gradient by Rys quadrature with the transfer after the
// contraction, every class up to (ff|ff); and the pieces it shares with the plain
// integrals (qx_plain.cuh).
//
// Method.  A primitive [e0|f0] with all quanta on the first centre of each side is
// sum_r w_r Ix(ex,fx) Iy(ey,fy) Iz(ez,fz) over the Rys nodes (Dupuis, Rys & King, J. Chem.
// Phys. 65, 111 (1976)); the 1-D factors follow the two-term recurrences of qx_rys.cuh.
// The transfer (ab| = sum_k C(b,k) AB^{b-k} (a+k,0| (Head-Gordon & Pople, J. Chem. Phys.
// 89, 5777 (1988), in closed form) does not depend on the primitives.
//
// The gradient never forms derivative integrals.  With G[e,f] = the transfer's transpose
// applied to Gamma, and U[e,f] the (e0|f0) values, E = sum G[e,f] U[e,f].  Per primitive
// and root a thread sums G over two directions, gx[ex] = sum G Iy Iz, and one direction's
// short sums give E0 = sum G V, LA = sum G e V(e-1) and LC = sum G f V(f-1).  Moving the
// bra as a whole changes only P - Q; differentiating the recurrences,
//   t = sum_r (-2 rho u PQ E0 - u q/(p+q) LA + u p/(p+q) LC)_r  (p, q: the two zetas),
// and the derivatives of the Gaussians at fixed P - Q are polynomials again:
//   dE/dA = sum_prim (a/p) t - (b/p) (LA + 2 a AB E0) + X_AB,   dE/dB = t - dE/dA
//   dE/dC = sum_prim -(c/q) t - (d/q) (LC + 2 c CD E0) + X_CD,  dE/dD = -t - dE/dC
// with X_AB = sum (dG/dAB) U.  No term is raised, so no tight exponent multiplies a
// difference of moments, as 2 b (V(e+1) + AB V(e)) would for a tight b: on eight random
// molecules with s to f shells the gradient lies 1e-15 to 9e-14 of its largest entry from
// an 80-bit evaluation, the programs it replaces 4e-15 to 2e-11.  (The transfer after the
// contraction does cost the (33|xx) classes digits, up to 1e-12 of the class's own
// contribution, where the others lost more.)
//
// Organisation.  A block owns (quartet, part of its primitives).  Per batch of PB
// primitives: the nodes and weights (one thread per function), the 2-D tables in shared
// memory (one thread per primitive, root and direction), then the sums: a lane owns one
// f and one of NP primitives of the batch, a warp one chunk of the e's -- a set of ex
// values, compile time, so that a chunk's values live in registers and one load of a
// column serves them all.  Parts of a quartet add into the gradient with atomics.
//
// TK_PLAIN: the same transfer forwards, in host code only; its phases serve the host check
// of the tables (the plain kernels transfer each 1-D factor instead, for accuracy).
//
// What bounds it: the FP64 pipe in the sums (about 2/3 of the instructions of the large
// classes); the kernels it replaces kept the (a,b,c,d) tables of every root and read 21 of
// their entries per component and root, which bound them on shared memory, and walked all
// primitives of a quartet on one team.
#pragma once
#include <algorithm>

#include "qx_rys.cuh"
#include "qx_segments.h"

namespace qx {

// ------------------------------------------------------------------ one side ---
QX_HD constexpr int tl_hoff(int l) { return l * (l + 1) * (l + 2) / 6; }

// The side (l1 l2|: its (e0| values e = l1 .. l1 + l2 and the terms of its transfer.
// A combo is (b, k <= b) with the coefficient prod_x C(b_x, k_x) AB_x^{b_x - k_x}; a
// term is (a, combo), reading e = a + k.
template <int L1, int L2>
struct TileSide {
    static constexpr int LO = L1, HI = L1 + L2;
    static constexpr int NE = tl_hoff(HI + 1) - tl_hoff(LO);
    static constexpr int N1 = ncart_h(L1), N2 = ncart_h(L2), NP = N1 * N2;
    QX_HD static constexpr int ncombo() {
        int n = 0;
        for (int x = L2; x >= 0; --x)
            for (int y = L2 - x; y >= 0; --y) n += (x + 1) * (y + 1) * (L2 - x - y + 1);
        return n;
    }
    static constexpr int NCOMBO = ncombo(), NTERM = N1 * NCOMBO;
    struct Tab {
        unsigned char fe[NTERM];       // e of term ia * NCOMBO + c
        unsigned short inv[NTERM];     // terms sorted by e
        unsigned short ioff[NE + 1];   // e's range in inv
        unsigned char cb[NCOMBO];      // combo -> b
        unsigned char cx[NCOMBO], cy[NCOMBO], cz[NCOMBO];  // b_x | k_x << 2
        unsigned char c0[N2 + 1];      // b's combos
        unsigned char ex[NE], ey[NE], ez[NE];
    };
    QX_HD static constexpr Tab make() {
        Tab t{};
        int n = 0;
        for (int l = LO; l <= HI; ++l)
            for (int x = l; x >= 0; --x)
                for (int y = l - x; y >= 0; --y, ++n) {
                    t.ex[n] = (unsigned char)x;
                    t.ey[n] = (unsigned char)y;
                    t.ez[n] = (unsigned char)(l - x - y);
                }
        int c = 0, b = 0;
        for (int x = L2; x >= 0; --x)
            for (int y = L2 - x; y >= 0; --y, ++b) {
                const int z = L2 - x - y;
                t.c0[b] = (unsigned char)c;
                for (int i = 0; i <= x; ++i)
                    for (int j = 0; j <= y; ++j)
                        for (int k = 0; k <= z; ++k, ++c) {
                            t.cb[c] = (unsigned char)b;
                            t.cx[c] = (unsigned char)(x | i << 2);
                            t.cy[c] = (unsigned char)(y | j << 2);
                            t.cz[c] = (unsigned char)(z | k << 2);
                        }
            }
        t.c0[N2] = (unsigned char)c;
        int a = 0;
        for (int x = L1; x >= 0; --x)
            for (int y = L1 - x; y >= 0; --y, ++a)
                for (int q = 0; q < NCOMBO; ++q) {
                    const int ex = x + (t.cx[q] >> 2), ey = y + (t.cy[q] >> 2), ez = L1 - x - y + (t.cz[q] >> 2);
                    const int l = ex + ey + ez, k = ey + ez;
                    t.fe[a * NCOMBO + q] = (unsigned char)(tl_hoff(l) - tl_hoff(LO) + k * (k + 1) / 2 + ez);
                }
        int m = 0;
        for (int e = 0; e < NE; ++e) {
            t.ioff[e] = (unsigned short)m;
            for (int q = 0; q < NTERM; ++q)
                if (t.fe[q] == e) t.inv[m++] = (unsigned short)q;
        }
        t.ioff[NE] = (unsigned short)m;
        return t;
    }
};
#ifdef __CUDA_ARCH__
template <int L1, int L2>
__device__ const typename TileSide<L1, L2>::Tab g_tile_tab = TileSide<L1, L2>::make();
#else
template <int L1, int L2>
const typename TileSide<L1, L2>::Tab g_tile_tab = TileSide<L1, L2>::make();
#endif

enum { TK_PLAIN = 0, TK_GRAD = 1 };

// ------------------------------------------------------------------ one class --
constexpr int TILE_SMEM_TARGET = 72 * 1024;  // tables of a batch (bytes)
constexpr int TILE_MAXW = 8;                 // warps per block
constexpr long long TILE_GRID = 1LL << 30;   // blocks per launch

// Warps per chunk: the fewest that hold all nf lanes, more while their lanes fill better
// and while no more than 16 primitives are summed side by side (a quartet has a few dozen).
QX_HD constexpr int tl_wpc(int nf, int wmin, int nchb) {
    int best = wmin;
    double bu = 0.0;
    for (int w = wmin; w * nchb <= TILE_MAXW; ++w) {
        if (w > wmin && 32 * w / nf > 16) break;
        const double u = (double)(32 * w / nf * nf) / (32 * w) + (w * nchb <= 4 ? 0.04 * w * nchb : 0.0);
        if (u > bu + 0.08) {
            bu = u;
            best = w;
        }
    }
    return best;
}
// Primitives per batch: a multiple of np whose units fill the block's threads best.
QX_HD constexpr int tl_pb(int np, int nr, int nt, int per_prim) {
    const int cap = TILE_SMEM_TARGET / 8 / per_prim;
    int best = np;
    double bu = 0.0;
    for (int p = np; p <= cap && p <= 128; p += np) {
        const int u = 3 * nr * p, rounds = (u + nt - 1) / nt;
        const double f = (double)u / (rounds * nt) - 0.02 * rounds;
        if (f > bu + 0.02) {
            bu = f;
            best = p;
        }
    }
    return best;
}

template <int LA, int LB, int LC, int LD, int KIND>
struct TileCls {
    using Bra = TileSide<LA, LB>;
    using Ket = TileSide<LC, LD>;
    static constexpr int kind = KIND;
    static constexpr int la = LA, lb = LB, lc = LC, ld = LD;
    static constexpr bool DER = KIND != TK_PLAIN;
    static constexpr int NE = Bra::NE, NF = Ket::NE, NFP = NF | 1;
    static constexpr int NAB = Bra::NP, NCD = Ket::NP, NCDP = NCD | 1, NCOMP = NAB * NCD;
    static constexpr int NR = (LA + LB + LC + LD + KIND) / 2 + 1;
    static_assert(NR <= QX_RYS_NMAX, "Rys table too short for this class");
    static constexpr int NI = LA + LB + 1, NK = LC + LD + 1;
    // columns start on different 16-byte units: padded to 2 mod 4 doubles
    static constexpr int NIP = NI <= 2 ? 2 : (NI <= 6 ? 6 : 10);
    static constexpr int UNIT = NK * NIP;
    // chunks of the e's by ex: the values a thread keeps (plain: U; gradient: G and U)
    // next to the columns must fit its registers
    static constexpr int BUDGET = KIND == TK_PLAIN ? 80 : 27;
    QX_HD static constexpr int per_ex(int x) {
        int n = 0;
        for (int y = 0; x + y <= LA + LB; ++y)
            for (int z = 0; x + y + z <= LA + LB; ++z)
                if (x + y + z >= LA) ++n;
        return n;
    }
    // chunks per block: all, or (the largest classes) as many as the block's warps hold;
    // the other chunks are blocks of their own (everything after the sums is linear in U)
    static constexpr int WMIN = (NF + 31) / 32;
    static constexpr int NCH0 = (NE + BUDGET - 1) / BUDGET > LA + LB + 1 ? LA + LB + 1 : (NE + BUDGET - 1) / BUDGET;
    static constexpr int NCHB0 = NCH0 * WMIN <= TILE_MAXW ? NCH0 : TILE_MAXW / WMIN;
    static constexpr int NPASS = (NCH0 + NCHB0 - 1) / NCHB0;
    static constexpr int NCHB = (NCH0 + NPASS - 1) / NPASS;
    static constexpr int NCH = NPASS * NCHB;
    static_assert(NCH <= LA + LB + 1, "more chunks than ex values");
    struct Chunks {
        int mask[8];
        int most;
    };
    QX_HD static constexpr Chunks chunks() {
        Chunks c{};
        int load[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int x = 0; x <= LA + LB; ++x) {  // per_ex falls with x: largest first onto the least loaded
            int b = 0;
            for (int k = 1; k < NCH; ++k)
                if (load[k] < load[b]) b = k;
            c.mask[b] |= 1 << x;
            load[b] += per_ex(x);
        }
        for (int k = 0; k < NCH; ++k)
            if (load[k] > c.most) c.most = load[k];
        return c;
    }
    QX_HD static constexpr int MASK(int k) { return chunks().mask[k]; }
    static constexpr int NSLOT = chunks().most;
    static constexpr int WPC = tl_wpc(NF, WMIN, NCHB);
    static constexpr int W = WPC * NCHB, NT = 32 * W;
    static constexpr int NP = 32 * WPC / NF;  // primitives of a batch summed side by side
    static constexpr int PER_PRIM = 3 * NR * UNIT;  // table entries of one primitive
    static constexpr int PB = tl_pb(NP, NR, NT, PER_PRIM);
    // shared memory, in doubles: the persistent part, then a region that holds the
    // batch's tables, or (before and after the primitives) the transfer's arrays
    static constexpr int CO = (Bra::NCOMBO + Ket::NCOMBO) * (DER ? 4 : 1);
    static constexpr int NDEN = DER ? Bra::NP + Ket::NP + (Bra::N1 + Bra::N2) * (Ket::N1 + Ket::N2) : 0;
    // the scalars and nodes of two batches: the sums read theirs while the next are made
    static constexpr int SCP = 11;  // per primitive
    static constexpr int NSC = DER ? 2 * SCP * PB : 0;
    static constexpr int UWB = 2 * NR * PB;  // nodes and weights
    static constexpr int UW = DER ? 2 * UWB : UWB;
    static constexpr int HEAD = (CO + NDEN + NSC + UW + 9 * TILE_MAXW + 1) / 2 * 2;
    static constexpr int YSZ = NE * NFP;
    static constexpr int OUTSZ = KIND == TK_PLAIN ? NCOMP : 0;  // J/K: the block itself, over U
    static constexpr int Y = ((YSZ > OUTSZ ? YSZ : OUTSZ) + 1) / 2 * 2;
    static constexpr int XA = NAB * NFP, XB = DER ? NE * NCDP : 0;
    static constexpr int X = XA > XB ? XA : XB;
    static constexpr int TABS = PB * PER_PRIM;
    static_assert(NP == 1 || NPASS == 1, "sums over side-by-side primitives expect every chunk in the block");
    static constexpr int RED = NP > 1 ? YSZ + NE * NFP : 0;  // sums over the NP primitives
    static constexpr int REG0 = TABS > Y + X ? TABS : Y + X;
    static constexpr int REGION = REG0 > RED ? REG0 : RED;
    static constexpr int SMEM = 8 * (HEAD + REGION);
    static_assert(SMEM <= 227 * 1024, "tile program exceeds shared memory");
    static constexpr int RSUB = (REGION - YSZ) / (NE * NFP) < 1 ? 1 : (REGION - YSZ) / (NE * NFP);
};

struct TileArgs {
    EriArgs e;
    const double* rys = nullptr;
    // segments of the launch (tile_segments), 2^(lg0 + k) blocks that share a quartet's
    // primitives in segment k; block0: a launch's first block, where they do not fit one grid
    int nseg = 1, lg0 = 0;
    long long block0 = 0;
    long long start[SEG_POW] = {};
    long long first[SEG_POW] = {};
    const double* D = nullptr;
    double cj = 0.0, ck = 0.0;
    double* grad = nullptr;  // 3N, atomic adds
};

// ------------------------------------------------------------------ phases -----
struct TileQuartet {
    PairInfo P, Q;
};

QX_HD inline double tl_pow(double x, int n) { return n == 0 ? 1.0 : (n == 1 ? x : (n == 2 ? x * x : x * x * x)); }

// Transfer coefficients of one side: co[c], and with DER co[(1 + x) * NCOMBO + c] = its
// derivative with respect to AB_x.
template <class Side, bool DER>
QX_HD inline void tl_coefs(const typename Side::Tab& t, const double* AB, double* co, int tid, int nth) {
    constexpr int binom[4][4] = {{1, 0, 0, 0}, {1, 1, 0, 0}, {1, 2, 1, 0}, {1, 3, 3, 1}};
    for (int c = tid; c < Side::NCOMBO; c += nth) {
        const int q[3] = {t.cx[c], t.cy[c], t.cz[c]};
        double f[3], g[3];  // factor and its derivative per direction
        for (int x = 0; x < 3; ++x) {
            const int b = q[x] & 3, k = q[x] >> 2, m = b - k;
            const double n = binom[b][k];
            f[x] = n * tl_pow(AB[x], m);
            g[x] = m > 0 ? n * m * tl_pow(AB[x], m - 1) : 0.0;
        }
        co[c] = f[0] * f[1] * f[2];
        if (DER) {
            co[Side::NCOMBO + c] = g[0] * f[1] * f[2];
            co[2 * Side::NCOMBO + c] = f[0] * g[1] * f[2];
            co[3 * Side::NCOMBO + c] = f[0] * f[1] * g[2];
        }
    }
}

// Density blocks of a quartet: AB, CD, AC, AD, BC, BD.
template <class C>
QX_HD inline void tl_density(const double* D, long long n, const PairInfo& P, const PairInfo& Q, double* den, int tid,
                             int nth) {
    constexpr int NA = C::Bra::N1, NB = C::Bra::N2, NC = C::Ket::N1, ND = C::Ket::N2;
    for (int i = tid; i < C::NDEN; i += nth) {
        int r = i;
        long long p, q;
        if (r < NA * NB) {
            p = P.bf1 + r / NB;
            q = P.bf2 + r % NB;
        } else if ((r -= NA * NB) < NC * ND) {
            p = Q.bf1 + r / ND;
            q = Q.bf2 + r % ND;
        } else if ((r -= NC * ND) < NA * NC) {
            p = P.bf1 + r / NC;
            q = Q.bf1 + r % NC;
        } else if ((r -= NA * NC) < NA * ND) {
            p = P.bf1 + r / ND;
            q = Q.bf2 + r % ND;
        } else if ((r -= NA * ND) < NB * NC) {
            p = P.bf2 + r / NC;
            q = Q.bf1 + r % NC;
        } else {
            r -= NB * NC;
            p = P.bf2 + r / ND;
            q = Q.bf2 + r % ND;
        }
        den[i] = D[p * n + q];
    }
}

// Gamma of one component, summed over the integral's distinct images.
template <class C>
struct TileGamma {
    const double* den;
    double fj, fd, fx;  // Coulomb, direct and crossed exchange factors
    QX_HD double operator()(int ab, int cd) const {
        constexpr int NA = C::Bra::N1, NB = C::Bra::N2, NC = C::Ket::N1, ND = C::Ket::N2;
        constexpr int oAC = NA * NB + NC * ND, oAD = oAC + NA * NC, oBC = oAD + NA * ND, oBD = oBC + NB * NC;
        const int a = ab / NB, b = ab - a * NB, c = cd / ND, d = cd - c * ND;
        return fj * den[ab] * den[NA * NB + cd] + fd * den[oAC + a * NC + c] * den[oBD + b * ND + d] +
               fx * den[oAD + a * ND + d] * den[oBC + b * NC + c];
    }
};
template <class C>
QX_HD inline TileGamma<C> tl_gamma(const double* den, const PairInfo& P, const PairInfo& Q, bool sPQ, double cj,
                                   double ck) {
    const bool s12 = P.s1 != P.s2, s34 = Q.s1 != Q.s2;
    return {den, cj * (1.0 + sPQ) * (1.0 + s12) * (1.0 + s34), ck * (1.0 + sPQ) * (1.0 + (double)(s12 && s34)),
            ck * (1.0 + sPQ) * ((double)s12 + (double)s34)};
}

// H[ab][f] = sum over (cd -> f) of coefficient times Gamma[ab][cd].
template <class C>
QX_HD inline void tl_gam_ket(const typename C::Ket::Tab& t, const double* co, const TileGamma<C>& G,
                             double* H, int tid, int nth) {
    for (int i = tid; i < C::NAB * C::NF; i += nth) {
        const int ab = i / C::NF, f = i - ab * C::NF;
        double s = 0.0;
        for (int q = t.ioff[f]; q < t.ioff[f + 1]; ++q) {
            const int term = t.inv[q], ic = term / C::Ket::NCOMBO, c = term - ic * C::Ket::NCOMBO;
            s = fma(G(ab, ic * C::Ket::N2 + t.cb[c]), co[c], s);
        }
        H[ab * C::NFP + f] = s;
    }
}

// G[e][f] = sum over (ab -> e) of coefficient times H[ab][f].
template <class C>
QX_HD inline void tl_gam_bra(const typename C::Bra::Tab& t, const double* co, const double* H,
                             double* G, int tid, int nth) {
    for (int i = tid; i < C::NE * C::NF; i += nth) {
        const int e = i / C::NF, f = i - e * C::NF;
        double s = 0.0;
        for (int q = t.ioff[e]; q < t.ioff[e + 1]; ++q) {
            const int term = t.inv[q], ia = term / C::Bra::NCOMBO, c = term - ia * C::Bra::NCOMBO;
            s = fma(co[c], H[(ia * C::Bra::N2 + t.cb[c]) * C::NFP + f], s);
        }
        G[e * C::NFP + f] = s;
    }
}

// H2[e][cd] = sum over (ab -> e) of coefficient times Gamma[ab][cd].
template <class C>
QX_HD inline void tl_gam_bra2(const typename C::Bra::Tab& t, const double* co, const TileGamma<C>& G,
                              double* H2, int tid, int nth) {
    for (int i = tid; i < C::NE * C::NCD; i += nth) {
        const int e = i / C::NCD, cd = i - e * C::NCD;
        double s = 0.0;
        for (int q = t.ioff[e]; q < t.ioff[e + 1]; ++q) {
            const int term = t.inv[q], ia = term / C::Bra::NCOMBO, c = term - ia * C::Bra::NCOMBO;
            s = fma(G(ia * C::Bra::N2 + t.cb[c], cd), co[c], s);
        }
        H2[e * C::NCDP + cd] = s;
    }
}

// X_AB: dot products of U with H over f for every bra term, times the coefficient's
// derivatives; X_CD: U with H2 over e for every ket term.
template <class C>
QX_HD inline void tl_x_bra(const typename C::Bra::Tab& t, const double* co, const double* U,
                           const double* H, double* g, int tid, int nth) {
    for (int i = tid; i < C::Bra::NTERM; i += nth) {
        const int ia = i / C::Bra::NCOMBO, c = i - ia * C::Bra::NCOMBO;
        const double *u = U + t.fe[i] * C::NFP, *h = H + (ia * C::Bra::N2 + t.cb[c]) * C::NFP;
        double s = 0.0;
        for (int f = 0; f < C::NF; ++f) s = fma(u[f], h[f], s);
        for (int x = 0; x < 3; ++x) {
            const double v = fma(co[(1 + x) * C::Bra::NCOMBO + c], s, 0.0);
            g[x] += v;
            g[3 + x] -= v;
        }
    }
}
template <class C>
QX_HD inline void tl_x_ket(const typename C::Ket::Tab& t, const double* co, const double* U,
                           const double* H2, double* g, int tid, int nth) {
    for (int i = tid; i < C::Ket::NTERM; i += nth) {
        const int ic = i / C::Ket::NCOMBO, c = i - ic * C::Ket::NCOMBO;
        const double *u = U + t.fe[i], *h = H2 + ic * C::Ket::N2 + t.cb[c];
        double s = 0.0;
        for (int e = 0; e < C::NE; ++e) s = fma(u[e * C::NFP], h[e * C::NCDP], s);
        for (int x = 0; x < 3; ++x) g[6 + x] += fma(co[(1 + x) * C::Ket::NCOMBO + c], s, 0.0);
    }
}

// Forward transfer (TK_PLAIN): H[ab][f] from U, and one component from H.
template <class C>
QX_HD inline void tl_fwd_bra(const typename C::Bra::Tab& t, const double* co, const double* U, double* H, int tid,
                             int nth) {
    for (int i = tid; i < C::NAB * C::NF; i += nth) {
        const int ab = i / C::NF, f = i - ab * C::NF, ia = ab / C::Bra::N2, ib = ab - ia * C::Bra::N2;
        double s = 0.0;
        for (int c = t.c0[ib]; c < t.c0[ib + 1]; ++c)
            s = fma(co[c], U[t.fe[ia * C::Bra::NCOMBO + c] * C::NFP + f], s);
        H[ab * C::NFP + f] = s;
    }
}
template <class C>
QX_HD inline double tl_fwd_ket(const typename C::Ket::Tab& t, const double* co, const double* H, int ab, int cd) {
    const int ic = cd / C::Ket::N2, id = cd - ic * C::Ket::N2;
    double s = 0.0;
    for (int c = t.c0[id]; c < t.c0[id + 1]; ++c)
        s = fma(co[c], H[ab * C::NFP + t.fe[ic * C::Ket::NCOMBO + c]], s);
    return s;
}

// Nodes and weights of the batch: item = primitive * 2 NR + function; a weight carries the
// prefactor.
template <class C>
QX_HD inline void tl_nodes(const double* rys, const TileQuartet& w, const PrimPair* bra,
                           const PrimPair* ket, int t0, int nb, double* uw, double* sc, int tid, int nth) {
    constexpr int NF2 = 2 * C::NR;
    const int nk = w.Q.nprim;
    for (int i = tid; i < nb * NF2; i += nth) {
        const int p = i / NF2, fn = i - p * NF2, t = t0 + p, ib = t / nk, ik = t - ib * nk;
        const PrimPair &a = bra[ib], &c = ket[ik];
        const double PQ[3] = {a.Px - c.Px, a.Py - c.Py, a.Pz - c.Pz};
        const double rs = 1.0 / (a.zeta + c.zeta), rho = a.zeta * c.zeta * rs;
        const double T = rho * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
        const double v = rys_fn<C::NR>(rys, fn, T);
        uw[i] = fn < C::NR ? v : v * (a.K * c.K * sqrt(rs));
        if (C::DER && fn == 0) {
            double* q = sc + C::SCP * p;
            q[0] = a.alpha / a.zeta;
            q[1] = (a.zeta - a.alpha) / a.zeta;
            q[2] = 2.0 * a.alpha;
            q[3] = c.alpha / c.zeta;
            q[4] = (c.zeta - c.alpha) / c.zeta;
            q[5] = 2.0 * c.alpha;
            q[6] = c.zeta * rs;
            q[7] = a.zeta * rs;
            for (int x = 0; x < 3; ++x) q[8 + x] = -2.0 * rho * PQ[x];
        }
    }
}

// 2-D tables of the batch: unit = (primitive * NR + root) * 3 + direction, column k at
// k * NIP.
template <class C>
QX_HD inline void tl_tables(const TileQuartet& w, const PrimPair* bra, const PrimPair* ket, int t0,
                            int nb, const double* uw, double* tab, int tid, int nth) {
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
        const double C00 = PA - qe * PQ, D00 = QC + pe * PQ;
        double* o = tab + (size_t)i * C::UNIT;
        double cur[C::NI], prev[C::NI];
        cur[0] = x == 2 ? uw[p * 2 * C::NR + C::NR + r] : 1.0;
        if constexpr (C::NI > 1) cur[1] = C00 * cur[0];
#pragma unroll
        for (int j = 2; j < C::NI; ++j) cur[j] = fma(C00, cur[j - 1], (j - 1) * B10 * cur[j - 2]);
#pragma unroll
        for (int j = 0; j < C::NI; ++j) {
            o[j] = cur[j];
            prev[j] = 0.0;
        }
#pragma unroll
        for (int k = 1; k < C::NK; ++k) {
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
                o[k * C::NIP + j] = cur[j];
            }
        }
    }
}

// ------------------------------------------------------------------ the sums ---
// Registers of one thread.
template <class C>
struct TileThread {
    double U[C::NSLOT];
    double G[C::DER ? C::NSLOT : 1];
    double g[9];
};

// Runs fn(slot, e, ex, ey, ez) over a chunk's e's (compile-time after unrolling).
template <class C, int M, class F>
QX_HD inline void tl_each(F&& fn) {
    constexpr int HI = C::Bra::HI, LO = C::Bra::LO;
    int s = 0;
#pragma unroll
    for (int ex = 0; ex <= HI; ++ex) {
        if (!((M >> ex) & 1)) continue;
#pragma unroll
        for (int ey = 0; ey <= HI; ++ey) {
#pragma unroll
            for (int ez = 0; ez <= HI; ++ez) {
                const int l = ex + ey + ez;
                if (l < LO || l > HI) continue;
                const int k = ey + ez;
                fn(s, tl_hoff(l) - tl_hoff(LO) + k * (k + 1) / 2 + ez, ex, ey, ez);
                ++s;
            }
        }
    }
}

// Column loads (16 bytes at a time).
template <int N>
QX_HD inline void tl_col(const double* p, double (&v)[N]) {
#ifdef __CUDA_ARCH__
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const double2 t = *reinterpret_cast<const double2*>(p + i);
        v[i] = t.x;
        if (i + 1 < N) v[i + 1 < N ? i + 1 : i] = t.y;
    }
#else
    for (int i = 0; i < N; ++i) v[i] = p[i];
#endif
}
// One primitive of a thread's (f, chunk): tab points at its NR * 3 units, uw at its nodes,
// sc at its scalars; fx, fy, fz are f's quanta.
template <class C, int M>
QX_HD inline void tl_prim(const double* tab, const double* uw, int fx, int fy, int fz, const double* sc,
                          const TileQuartet& w, TileThread<C>& th) {
    constexpr int HI = C::Bra::HI, LO = C::Bra::LO;
    // sums over the roots, and (t*) the same weighted with the node
    double LA[3] = {0, 0, 0}, LC[3] = {0, 0, 0}, tA[3] = {0, 0, 0}, tC[3] = {0, 0, 0};
    double E0 = 0.0, tE = 0.0;
#pragma unroll 1
    for (int r = 0; r < C::NR; ++r) {
        const double* t = tab + r * 3 * C::UNIT;
        double X[C::NI], Yv[C::NI], W[C::NI];
        tl_col(t + fx * C::NIP, X);
        tl_col(t + C::UNIT + fy * C::NIP, Yv);
        tl_col(t + 2 * C::UNIT + fz * C::NIP, W);
        if constexpr (!C::DER) {
            int s = 0;
#pragma unroll
            for (int ex = 0; ex <= HI; ++ex) {
                if (!((M >> ex) & 1)) continue;
#pragma unroll
                for (int ey = 0; ey <= HI - ex; ++ey) {
                    const double xy = X[ex] * Yv[ey];
#pragma unroll
                    for (int ez = 0; ez <= HI - ex - ey; ++ez) {
                        if (ex + ey + ez < LO) continue;
                        th.U[s] = fma(xy, W[ez], th.U[s]);
                        ++s;
                    }
                }
            }
        } else {
            double gx[HI + 1], gy[HI + 1], gz[HI + 1];
#pragma unroll
            for (int j = 0; j <= HI; ++j) gx[j] = gy[j] = gz[j] = 0.0;
            int s = 0;
#pragma unroll
            for (int ex = 0; ex <= HI; ++ex) {
                if (!((M >> ex) & 1)) continue;
#pragma unroll
                for (int ey = 0; ey <= HI - ex; ++ey) {
                    const double xy = X[ex] * Yv[ey];
                    double h = 0.0;
#pragma unroll
                    for (int ez = 0; ez <= HI - ex - ey; ++ez) {
                        if (ex + ey + ez < LO) continue;
                        th.U[s] = fma(xy, W[ez], th.U[s]);
                        h = fma(th.G[s], W[ez], h);
                        gz[ez] = fma(th.G[s], xy, gz[ez]);
                        ++s;
                    }
                    gx[ex] = fma(h, Yv[ey], gx[ex]);
                    gy[ey] = fma(h, X[ex], gy[ey]);
                }
            }
            // the largest quanta in y and z a chunk reaches
            constexpr int X0 = (M & 1) ? 0 : (M & 2) ? 1 : (M & 4) ? 2 : (M & 8) ? 3 : (M & 16) ? 4 : (M & 32) ? 5 : 6;
            constexpr int TOP = HI - X0;
            double e = 0.0, l0 = 0.0, l1 = 0.0, l2 = 0.0;
#pragma unroll
            for (int j = 0; j <= HI; ++j) {
                if ((M >> j) & 1) {
                    e = fma(gx[j], X[j], e);
                    if (j > 0) l0 = fma(j * gx[j], X[j > 0 ? j - 1 : 0], l0);
                }
                if (j > 0 && j <= TOP) {
                    l1 = fma(j * gy[j], Yv[j > 0 ? j - 1 : 0], l1);
                    l2 = fma(j * gz[j], W[j > 0 ? j - 1 : 0], l2);
                }
            }
            const double u = uw[r];
            E0 += e;
            tE = fma(u, e, tE);
            LA[0] += l0;
            LA[1] += l1;
            LA[2] += l2;
            tA[0] = fma(u, l0, tA[0]);
            tA[1] = fma(u, l1, tA[1]);
            tA[2] = fma(u, l2, tA[2]);
            // the lowered ket columns (a factor f_x of zero drops the clamped one)
            if constexpr (C::NK > 1) {
                double s0 = 0.0, s1 = 0.0, s2 = 0.0;
                tl_col(t + (fx > 0 ? fx - 1 : 0) * C::NIP, X);
#pragma unroll
                for (int j = 0; j <= HI; ++j)
                    if ((M >> j) & 1) s0 = fma(gx[j], X[j], s0);
                tl_col(t + C::UNIT + (fy > 0 ? fy - 1 : 0) * C::NIP, Yv);
#pragma unroll
                for (int j = 0; j <= TOP; ++j) s1 = fma(gy[j], Yv[j], s1);
                tl_col(t + 2 * C::UNIT + (fz > 0 ? fz - 1 : 0) * C::NIP, W);
#pragma unroll
                for (int j = 0; j <= TOP; ++j) s2 = fma(gz[j], W[j], s2);
                LC[0] += s0;
                LC[1] += s1;
                LC[2] += s2;
                tC[0] = fma(u, s0, tC[0]);
                tC[1] = fma(u, s1, tC[1]);
                tC[2] = fma(u, s2, tC[2]);
            }
        }
    }
    if constexpr (C::DER) {
        const double ra = sc[0], rb = sc[1], a2 = sc[2], rc = sc[3], rd = sc[4], c2 = sc[5], qp = sc[6], pp = sc[7];
        const double AB[3] = {w.P.ABx, w.P.ABy, w.P.ABz}, CD[3] = {w.Q.ABx, w.Q.ABy, w.Q.ABz};
        const int fq[3] = {fx, fy, fz};
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const double lc = fq[x] * LC[x];
            const double tot = fma(sc[8 + x], tE, pp * (fq[x] * tC[x]) - qp * tA[x]);
            const double abE = AB[x] * E0, cdE = CD[x] * E0;
            const double gA = ra * tot - rb * fma(a2, abE, LA[x]);
            th.g[x] += gA;
            th.g[3 + x] += tot - gA;
            th.g[6 + x] -= rc * tot + rd * fma(c2, cdE, lc);
        }
    }
}

template <class C, int K>
QX_HD inline void tl_prim_chunk(int chunk, const double* tab, const double* uw, int fx, int fy, int fz,
                                const double* sc, const TileQuartet& w, TileThread<C>& th) {
    if constexpr (K + 1 < C::NCH) {
        if (chunk != K) {
            tl_prim_chunk<C, K + 1>(chunk, tab, uw, fx, fy, fz, sc, w, th);
            return;
        }
    }
    tl_prim<C, C::MASK(K)>(tab, uw, fx, fy, fz, sc, w, th);
}

// A thread's values to and from the [e][f] arrays.
template <class C, int K>
QX_HD inline void tl_load(int chunk, const double* G, int f, TileThread<C>& th) {
    if constexpr (K + 1 < C::NCH) {
        if (chunk != K) {
            tl_load<C, K + 1>(chunk, G, f, th);
            return;
        }
    }
    tl_each<C, C::MASK(K)>([&](int s, int e, int, int, int) { th.G[s] = G[e * C::NFP + f]; });
}
template <class C, int K>
QX_HD inline void tl_store(int chunk, double* U, int f, const TileThread<C>& th) {
    if constexpr (K + 1 < C::NCH) {
        if (chunk != K) {
            tl_store<C, K + 1>(chunk, U, f, th);
            return;
        }
    }
    tl_each<C, C::MASK(K)>([&](int s, int e, int, int, int) { U[e * C::NFP + f] = th.U[s]; });
}

// Lane roles: chunk by warp, then (primitive of the batch, f).
template <class C>
struct TileRole {
    int chunk, f, sub;
    bool on;
    QX_HD TileRole(int tid, int pass) {
        const int warp = tid / 32, l = (warp / C::NCHB) * 32 + tid % 32;
        chunk = pass * C::NCHB + warp % C::NCHB;
        sub = l / C::NF;
        on = sub < C::NP && chunk < C::NCH;
        f = on ? l - sub * C::NF : 0;
    }
};

#ifndef TILE_HOST
// ------------------------------------------------------------------ device -----
// Registers a thread of the class wants, and the blocks per SM they and the shared
// memory allow.
template <class C>
struct TileBounds {
    static constexpr int VALUES = C::NSLOT * (C::DER ? 2 : 1) + 3 * C::NI + (C::DER ? 2 * (C::Bra::HI + 1) + 4 : 2);
    static constexpr int REGS0 = 2 * VALUES + (C::DER ? 64 : 48);
    static constexpr int REGS = REGS0 > 255 ? 255 : (REGS0 < 64 ? 64 : REGS0);
    static constexpr int BY_REGS = 65536 / (C::NT * REGS), BY_SMEM = 227 * 1024 / (C::SMEM + 1024);
    static constexpr int B0 = BY_REGS < BY_SMEM ? BY_REGS : BY_SMEM;
    static constexpr int MINB = B0 < 1 ? 1 : (B0 > 16 ? 16 : B0);
};

struct TileBlock {
    long long quartet;  // position in the processing order
    int part, parts;
};
__device__ __forceinline__ TileBlock tile_block(const TileArgs& ta) {
    int seg = ta.nseg - 1;  // block-uniform
    const long long bid = ta.block0 + blockIdx.x;
    while (seg > 0 && bid >= ta.start[seg - 1]) --seg;
    const long long rel = bid - ta.start[seg];
    const int lg = ta.lg0 + seg;
    return {ta.first[seg] + (rel >> lg), (int)(rel & ((1LL << lg) - 1)), 1 << lg};
}

// The quartet's pair records to shared memory.
template <int NT>
__device__ __forceinline__ void tile_pairs(const EriArgs& a, int2 pq, TileQuartet& w, int tid) {
    if (tid < 24) {
        reinterpret_cast<int*>(&w.P)[tid] = reinterpret_cast<const int*>(a.pairs + pq.x)[tid];
    } else if (tid < 48 && NT >= 48) {
        reinterpret_cast<int*>(&w.Q)[tid - 24] = reinterpret_cast<const int*>(a.pairs + pq.y)[tid - 24];
    }
    if (NT < 48 && tid < 24) reinterpret_cast<int*>(&w.Q)[tid] = reinterpret_cast<const int*>(a.pairs + pq.y)[tid];
}

template <class C>
__global__ void __launch_bounds__(C::NT, TileBounds<C>::MINB) k_tile(TileArgs ta) {
    static_assert(C::DER, "plain integrals: qx_plain.cuh");
    using Bra = typename C::Bra;
    using Ket = typename C::Ket;
    constexpr int NT = C::NT;
    extern __shared__ __align__(16) double tile_sm[];
    __shared__ TileQuartet w;
    const int tid = threadIdx.x;
    double* coA = tile_sm;
    double* coC = coA + Bra::NCOMBO * (C::DER ? 4 : 1);
    double* den = tile_sm + C::CO;
    double* sc = den + C::NDEN;
    double* uw = sc + C::NSC;
    double* red = uw + C::UW;
    double* region = tile_sm + C::HEAD;
    double* tab = region;
    double* Uy = region;
    double* Hx = region + C::Y;
    const typename Bra::Tab& tb = g_tile_tab<C::la, C::lb>;
    const typename Ket::Tab& tk = g_tile_tab<C::lc, C::ld>;
    const EriArgs& a = ta.e;
    const TileBlock at = tile_block(ta);
    const long long n = a.n;
    const int2 pq = a.quartets[list_index(a, at.quartet)];
    const int ntot = a.pairs[pq.x].nprim * a.pairs[pq.y].nprim;
    const int part = at.part, stride = at.parts * C::PB;
    if (part * C::PB >= ntot) return;  // whole block
    tile_pairs<NT>(a, pq, w, tid);
    __syncthreads();
    const bool sPQ = pq.x != pq.y;
    if (w.P.atom1 == w.P.atom2 && w.P.atom1 == w.Q.atom1 && w.P.atom1 == w.Q.atom2) return;
    {
        const double AB[3] = {w.P.ABx, w.P.ABy, w.P.ABz}, CD[3] = {w.Q.ABx, w.Q.ABy, w.Q.ABz};
        tl_coefs<Bra, true>(tb, AB, coA, tid, NT);
        tl_coefs<Ket, true>(tk, CD, coC, tid, NT);
    }
    const TileRole<C> role(tid, C::NPASS > 1 ? blockIdx.z : 0);
    TileThread<C> th;
#pragma unroll
    for (int s = 0; s < C::NSLOT; ++s) th.U[s] = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) th.g[i] = 0.0;
    TileGamma<C> gam = tl_gamma<C>(den, w.P, w.Q, sPQ, ta.cj, ta.ck);
    tl_density<C>(ta.D, n, w.P, w.Q, den, tid, NT);
    __syncthreads();
    tl_gam_ket<C>(tk, coC, gam, Hx, tid, NT);
    __syncthreads();
    tl_gam_bra<C>(tb, coA, Hx, Uy, tid, NT);
    __syncthreads();
    tl_load<C, 0>(role.on ? role.chunk : 0, Uy, role.f, th);
    __syncthreads();
    const PrimPair* bra = a.prims + w.P.prim_off;
    const PrimPair* ket = a.prims + w.Q.prim_off;
    const int fx = tk.ex[role.f], fy = tk.ey[role.f], fz = tk.ez[role.f];
    double *scp = sc, *uwp = uw;
    for (int t0 = part * C::PB; t0 < ntot; t0 += stride) {
        const int nb = min(C::PB, ntot - t0);
        tl_nodes<C>(ta.rys, w, bra, ket, t0, nb, uwp, scp, tid, NT);
        __syncthreads();  // the previous batch's sums are done, too
        tl_tables<C>(w, bra, ket, t0, nb, uwp, tab, tid, NT);
        __syncthreads();
        if (role.on)
            for (int p = role.sub; p < nb; p += C::NP)
                tl_prim_chunk<C, 0>(role.chunk, tab + (size_t)p * C::PER_PRIM, uwp + 2 * C::NR * p, fx, fy, fz,
                                    scp + C::SCP * p, w, th);
        // the next batch's nodes and scalars beside these
        scp = scp == sc ? sc + C::NSC / 2 : sc;
        uwp = uwp == uw ? uw + C::UWB : uw;
    }
    __syncthreads();
    // U of the NP primitives side by side -> Uy
    if constexpr (C::NPASS > 1) {  // the other passes' values count as zero here
        for (int i = tid; i < C::NE * C::NFP; i += NT) Uy[i] = 0.0;
        __syncthreads();
    }
    if (role.on && role.sub == 0) tl_store<C, 0>(role.chunk, Uy, role.f, th);
    if constexpr (C::NP > 1) {
        double* side = Uy + C::NE * C::NFP;
        for (int s0 = 1; s0 < C::NP; s0 += C::RSUB) {
            const int ns = min(C::RSUB, C::NP - s0);
            if (role.on && role.sub >= s0 && role.sub < s0 + ns)
                tl_store<C, 0>(role.chunk, side + (role.sub - s0) * C::NE * C::NFP, role.f, th);
            __syncthreads();
            for (int i = tid; i < C::NE * C::NFP; i += NT) {
                if (C::NFP != C::NF && i % C::NFP == C::NF) continue;  // padding
                double v = Uy[i];
                for (int k = 0; k < ns; ++k) v += side[k * C::NE * C::NFP + i];
                Uy[i] = v;
            }
            __syncthreads();
        }
    } else {
        __syncthreads();
    }
    if constexpr (C::lb > 0) {
        tl_gam_ket<C>(tk, coC, gam, Hx, tid, NT);
        __syncthreads();
        tl_x_bra<C>(tb, coA, Uy, Hx, th.g, tid, NT);
        if (C::ld > 0) __syncthreads();
    }
    if constexpr (C::ld > 0) {
        tl_gam_bra2<C>(tb, coA, gam, Hx, tid, NT);
        __syncthreads();
        tl_x_ket<C>(tk, coC, Uy, Hx, th.g, tid, NT);
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        for (int off = 16; off > 0; off >>= 1) th.g[i] += __shfl_xor_sync(0xffffffffu, th.g[i], off);
        if ((tid & 31) == 0) red[(tid >> 5) * 9 + i] = th.g[i];
    }
    __syncthreads();
    if (tid < 12) {
        const int x = tid % 3, c = tid / 3;
        double v = 0.0;
        for (int k = 0; k < C::W; ++k)
            v += c < 3 ? red[k * 9 + tid] : -(red[k * 9 + x] + red[k * 9 + 3 + x] + red[k * 9 + 6 + x]);
        const int atom = c == 0 ? w.P.atom1 : (c == 1 ? w.P.atom2 : (c == 2 ? w.Q.atom1 : w.Q.atom2));
        atomicAdd(ta.grad + 3 * atom + x, v);
    }
}

// Blocks of a class.  With one block per quartet the largest ones were the tail of every
// launch (ten atoms, (22|21): the FP64 pipe 45% busy while blocks ran, 26% over the
// launch).  A block takes at most `share` primitives: an eighth of what each of the GPU's
// block slots gets in all, and two batches and 48 primitives at least (about what the
// transfers of Gamma cost).  prefix[k] counts the quartets with more than 2^k
// primitives in the processing order (null: no order).
template <class C>
void launch_tile(TileArgs& ta, long long nq, long long prims, long long max_prims, const long long* prefix,
                 cudaStream_t s) {
    if (nq <= 0) return;
    auto k = k_tile<C>;
    if (C::SMEM > 40 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    const long long share = std::max<long long>(std::max(2 * C::PB, 48), prims / (148LL * TileBounds<C>::MINB * 8) + 1);
    long long blocks;
    ta.nseg = tile_segments(nq, share, max_prims, prefix, 1 << 24, ta.first, ta.start, &blocks);
    for (ta.block0 = 0; ta.block0 < blocks; ta.block0 += TILE_GRID)
        k<<<dim3((unsigned)std::min(TILE_GRID, blocks - ta.block0), 1, C::NPASS), C::NT, C::SMEM, s>>>(ta);
}
#endif  // TILE_HOST

}  // namespace qx
