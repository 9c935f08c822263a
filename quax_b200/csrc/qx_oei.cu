// qx_oei.cu -- one-electron integrals S, T, V and their first nuclear derivatives.
//
// Replaces the one-electron part of the reference's Libint module
// (quax/integrals/libint_interface.cc:232-483 compute_1e_int, :650-788
// compute_1e_deriv, :2403-2579 oei_deriv_core) for the HF energy and gradient.
// O(n^2 natom) work next to the O(n^4) two-electron path: S and T by k_oei (one warp
// per shell pair, one lane per Cartesian component pair, runtime angular momenta),
// the nuclear attraction by k_nai (below) -- except for a lone atom, whose nuclear
// derivatives are zero but for the rounding of their sums: there k_oei adds the
// attraction too, in Hermite form (McMurchie & Davidson, J. Comput. Phys. 26, 218
// (1978)), and the few pairs of one atom leave nothing to gain.
//
// Method (Obara & Saika, J. Chem. Phys. 84, 3963 (1986); Dupuis, Rys & King, J. Chem.
// Phys. 65, 111 (1976)):
//   overlap   1-D Obara-Saika recursion S(i+1,j) = PA S(i,j) + (i S(i-1,j) + j S(i,j-1))/2p
//             (and the j analogue with PB), S(0,0) = sqrt(pi/p);
//   kinetic   T_x(i,j) = -2 b^2 S(i,j+2) + b (2j+1) S(i,j) - j(j-1)/2 S(i,j-2);
//   nuclear   V = -Z_C (2 pi/p) sum_r w_r Ix(u_r) Iy(u_r) Iz(u_r), the Rys rule of
//             T = p |P-C|^2 with 1-D factors I(i+1) = (PA - u PC) I(i) +
//             i (1-u)/(2p) I(i-1) and the transfer I(a,b+1) = I(a+1,b) + AB I(a,b);
//   derivatives d/dA_x g_a = 2 alpha g_{a+1x} - a_x g_{a-1x} (and for B); the
//             derivative of the nuclear term with respect to the nucleus C follows
//             from translational invariance of each term: d/dC = -(d/dA + d/dB).
// Every block is written for both (i,j) and (j,i) by the lane that owns it.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "quax_b200.h"
#include "qx_rys.cuh"

namespace qx {

constexpr int OEI_LMAX = 3;               // shell AM the local tables are sized for
constexpr int OEI_NI = OEI_LMAX + 2;      // i up to la + 1
constexpr int OEI_NJ = OEI_LMAX + 4;      // j up to lb + 3 (kinetic of a B-derivative)
constexpr int OEI_NT = 2 * OEI_LMAX + 3;  // Hermite index t up to la + lb + 2
constexpr int OEI_LR = 2 * OEI_LMAX + 1;  // R_tuv with t + u + v <= la + lb + 1
constexpr int OEI_NR = (OEI_LR + 1) * (OEI_LR + 2) * (OEI_LR + 3) / 6;

struct OeiArgs {
    const PairInfo* pairs;
    int npair;
    const PrimPair* prims;
    const double* boys;
    const double* rys;  // Rys node/weight table
    const double* xyz;  // natom x 3 (bohr)
    const double* Z;    // natom
    int natom;
    int nuc;  // nuclei whose attraction k_oei itself adds (a lone atom), else 0
    long long n;
    double *S, *T, *V;     // n x n (may be null)
    double *dS, *dT, *dV;  // 3N x n x n (may be null)
};

__device__ __forceinline__ void cart_of(int l, int k, int& x, int& y, int& z) {
    // Libint standard order: lx from l down, then ly from l - lx down
    for (int lx = l; lx >= 0; --lx)
        for (int ly = l - lx; ly >= 0; --ly) {
            if (k == 0) {
                x = lx;
                y = ly;
                z = l - lx - ly;
                return;
            }
            --k;
        }
    x = y = z = 0;
}

__device__ __forceinline__ int ridx(int t, int u, int v) {
    // packed index of (t,u,v), t+u+v = s: offset of shell s plus position inside it
    const int s = t + u + v;
    const int k = u + v;
    return s * (s + 1) * (s + 2) / 6 + k * (k + 1) / 2 + v;
}

// 1-D overlaps S(i,j) for i <= ni, j <= nj (without the sqrt(pi/p) factor).
__device__ __forceinline__ void overlap_1d(double PA, double PB, double oo2p, int ni, int nj,
                                           double (&s)[OEI_NI][OEI_NJ]) {
    s[0][0] = 1.0;
    for (int i = 0; i < ni; ++i) s[i + 1][0] = PA * s[i][0] + (i ? i * oo2p * s[i - 1][0] : 0.0);
    for (int j = 0; j < nj; ++j)
        for (int i = 0; i <= ni; ++i)
            s[i][j + 1] = PB * s[i][j] + oo2p * ((i ? i * s[i - 1][j] : 0.0) + (j ? j * s[i][j - 1] : 0.0));
}

// Kinetic 1-D factor acting on the ket index j.
__device__ __forceinline__ double kin_1d(const double (&s)[OEI_NI][OEI_NJ], int i, int j, double b) {
    double t = -2.0 * b * b * s[i][j + 2] + b * (2 * j + 1) * s[i][j];
    if (j >= 2) t -= 0.5 * j * (j - 1) * s[i][j - 2];
    return t;
}

// Hermite coefficients E^{ij}_t for i <= ni, j <= nj (1-D, without exp(-mu X^2)).
__device__ __forceinline__ void hermite_1d(double PA, double PB, double oo2p, int ni, int nj,
                                           double (&E)[OEI_NI][OEI_NI][OEI_NT]) {
    for (int i = 0; i <= ni; ++i)
        for (int j = 0; j <= nj; ++j)
            for (int t = 0; t < OEI_NT; ++t) E[i][j][t] = 0.0;
    E[0][0][0] = 1.0;
    for (int i = 0; i <= ni; ++i)
        for (int j = 0; j <= nj; ++j) {
            if (i == 0 && j == 0) continue;
            const bool up_i = i > 0;
            const int pi = up_i ? i - 1 : i, pj = up_i ? j : j - 1;
            const double X = up_i ? PA : PB;
            for (int t = 0; t <= i + j; ++t) {
                double v = X * E[pi][pj][t];
                if (t > 0) v += oo2p * E[pi][pj][t - 1];
                if (t + 1 <= pi + pj) v += (t + 1) * E[pi][pj][t + 1];
                E[i][j][t] = v;
            }
        }
}

__global__ void __launch_bounds__(128) k_oei(OeiArgs a) {
    const int lane = threadIdx.x & 31;
    const int pidx = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (pidx >= a.npair) return;
    const PairInfo P = a.pairs[pidx];
    const int la = P.l1, lb = P.l2;
    const int na = (la + 1) * (la + 2) / 2, nb = (lb + 1) * (lb + 2) / 2;
    const bool same = P.s1 == P.s2;
    const bool deriv = a.dS != nullptr;
    const double kfac = 5.914967172795613;  // sqrt(2) pi^(5/4), the factor in PrimPair::K
    for (int c = lane; c < na * nb; c += 32) {
        const int ia = c / nb, ib = c % nb;
        if (same && ib > ia) continue;  // the (ia, ib) lane writes (ib, ia) too
        int ax, ay, az, bx, by, bz;
        cart_of(la, ia, ax, ay, az);
        cart_of(lb, ib, bx, by, bz);
        double s = 0.0, t = 0.0, v = 0.0;
        double dsa[3] = {0, 0, 0}, dsb[3] = {0, 0, 0}, dta[3] = {0, 0, 0}, dtb[3] = {0, 0, 0};
        double dva[3] = {0, 0, 0}, dvb[3] = {0, 0, 0};
        const long long i0 = P.bf1 + ia, j0 = P.bf2 + ib;
        for (int k = 0; k < P.nprim; ++k) {
            const PrimPair pp = a.prims[P.prim_off + k];
            const double p = pp.zeta, al = pp.alpha, be = p - al, oo2p = pp.oo2z;
            const double w = pp.K * p / kfac;  // c_a c_b exp(-mu |AB|^2)
            const double PA[3] = {pp.PAx, pp.PAy, pp.PAz};
            const double PB[3] = {pp.PAx + P.ABx, pp.PAy + P.ABy, pp.PAz + P.ABz};
            const int la3[3] = {ax, ay, az}, lb3[3] = {bx, by, bz};
            // overlap and kinetic factors per dimension
            double S0[3], Sa[3], Sb[3], T0[3], Ta[3], Tb[3];
            const double rp = sqrt(3.14159265358979323846 / p);
            for (int d = 0; d < 3; ++d) {
                double tab[OEI_NI][OEI_NJ];
                const int ni = la3[d] + 1, nj = lb3[d] + 3;
                overlap_1d(PA[d], PB[d], oo2p, ni, nj, tab);
                const int i = la3[d], j = lb3[d];
                S0[d] = rp * tab[i][j];
                T0[d] = rp * kin_1d(tab, i, j, be);
                Sa[d] = rp * (2.0 * al * tab[i + 1][j] - (i ? i * tab[i - 1][j] : 0.0));
                Ta[d] = rp * (2.0 * al * kin_1d(tab, i + 1, j, be) - (i ? i * kin_1d(tab, i - 1, j, be) : 0.0));
                Sb[d] = rp * (2.0 * be * tab[i][j + 1] - (j ? j * tab[i][j - 1] : 0.0));
                Tb[d] = rp * (2.0 * be * kin_1d(tab, i, j + 1, be) - (j ? j * kin_1d(tab, i, j - 1, be) : 0.0));
            }
            s += w * S0[0] * S0[1] * S0[2];
            t += w * (T0[0] * S0[1] * S0[2] + S0[0] * T0[1] * S0[2] + S0[0] * S0[1] * T0[2]);
            if (deriv) {
                for (int d = 0; d < 3; ++d) {
                    const int d1 = (d + 1) % 3, d2 = (d + 2) % 3;
                    dsa[d] += w * Sa[d] * S0[d1] * S0[d2];
                    dsb[d] += w * Sb[d] * S0[d1] * S0[d2];
                    dta[d] += w * (Ta[d] * S0[d1] * S0[d2] + Sa[d] * (T0[d1] * S0[d2] + S0[d1] * T0[d2]));
                    dtb[d] += w * (Tb[d] * S0[d1] * S0[d2] + Sb[d] * (T0[d1] * S0[d2] + S0[d1] * T0[d2]));
                }
            }
            if (!a.nuc) continue;  // k_nai's
            // nuclear attraction: Hermite expansion of the pair, one R table per nucleus
            double E[3][OEI_NI][OEI_NI][OEI_NT];
            for (int d = 0; d < 3; ++d) hermite_1d(PA[d], PB[d], oo2p, la3[d] + 1, lb3[d] + 1, E[d]);
            const int L = la + lb + (deriv ? 1 : 0);
            const double Px = pp.Px, Py = pp.Py, Pz = pp.Pz;
            for (int C = 0; C < a.nuc; ++C) {
                const double XPC = Px - a.xyz[3 * C], YPC = Py - a.xyz[3 * C + 1], ZPC = Pz - a.xyz[3 * C + 2];
                const double T = p * (XPC * XPC + YPC * YPC + ZPC * ZPC);
                double F[2 * OEI_LMAX + 2];
                boys<2 * OEI_LMAX + 1>(T, a.boys, F);
                // R^{n}_{tuv}, n from L down to 0 (two packed buffers)
                double Rn[OEI_NR], Rm[OEI_NR];
                double m2p = 1.0;
                for (int q = 0; q < L; ++q) m2p *= -2.0 * p;
                for (int n = L; n >= 0; --n) {
                    const int top = L - n;
                    for (int s3 = 0; s3 <= top; ++s3)
                        for (int tt = s3; tt >= 0; --tt)
                            for (int uu = s3 - tt; uu >= 0; --uu) {
                                const int vv = s3 - tt - uu;
                                double r;
                                if (tt > 0)
                                    r = XPC * Rm[ridx(tt - 1, uu, vv)] + (tt > 1 ? (tt - 1) * Rm[ridx(tt - 2, uu, vv)] : 0.0);
                                else if (uu > 0)
                                    r = YPC * Rm[ridx(tt, uu - 1, vv)] + (uu > 1 ? (uu - 1) * Rm[ridx(tt, uu - 2, vv)] : 0.0);
                                else if (vv > 0)
                                    r = ZPC * Rm[ridx(tt, uu, vv - 1)] + (vv > 1 ? (vv - 1) * Rm[ridx(tt, uu, vv - 2)] : 0.0);
                                else
                                    r = m2p * F[n];
                                Rn[ridx(tt, uu, vv)] = r;
                            }
                    for (int q = 0; q < (top + 1) * (top + 2) * (top + 3) / 6; ++q) Rm[q] = Rn[q];
                    m2p /= -2.0 * p;
                }
                const double* R = Rm;  // R^{0}
                const double pre = -a.Z[C] * 2.0 * 3.14159265358979323846 / p * w;
                // Hermite sum for shifted component indices (sa, sb per dimension)
                auto hsum = [&](int ix, int jx, int iy, int jy, int iz, int jz) {
                    double acc = 0.0;
                    for (int tt = 0; tt <= ix + jx; ++tt) {
                        const double ex = E[0][ix][jx][tt];
                        if (ex == 0.0) continue;
                        for (int uu = 0; uu <= iy + jy; ++uu) {
                            const double exy = ex * E[1][iy][jy][uu];
                            if (exy == 0.0) continue;
                            for (int vv = 0; vv <= iz + jz; ++vv) acc += exy * E[2][iz][jz][vv] * R[ridx(tt, uu, vv)];
                        }
                    }
                    return acc;
                };
                v += pre * hsum(ax, bx, ay, by, az, bz);
                if (deriv) {
                    double ga[3], gb[3];
                    for (int d = 0; d < 3; ++d) {
                        int ia3[3] = {ax, ay, az}, ib3[3] = {bx, by, bz};
                        ia3[d] += 1;
                        double up = hsum(ia3[0], ib3[0], ia3[1], ib3[1], ia3[2], ib3[2]);
                        double dn = 0.0;
                        if (la3[d] > 0) {
                            ia3[d] -= 2;
                            dn = hsum(ia3[0], ib3[0], ia3[1], ib3[1], ia3[2], ib3[2]);
                            ia3[d] += 1;
                        } else {
                            ia3[d] -= 1;
                        }
                        ga[d] = pre * (2.0 * al * up - la3[d] * dn);
                        ib3[d] += 1;
                        up = hsum(ia3[0], ib3[0], ia3[1], ib3[1], ia3[2], ib3[2]);
                        dn = 0.0;
                        if (lb3[d] > 0) {
                            ib3[d] -= 2;
                            dn = hsum(ia3[0], ib3[0], ia3[1], ib3[1], ia3[2], ib3[2]);
                        }
                        gb[d] = pre * (2.0 * be * up - lb3[d] * dn);
                        dva[d] += ga[d];
                        dvb[d] += gb[d];
                    }
                    // nucleus C by invariance of this term
                    const long long nn = a.n * a.n;
                    for (int d = 0; d < 3; ++d) {
                        double* o = a.dV + (3LL * C + d) * nn;
                        o[i0 * a.n + j0] -= ga[d] + gb[d];
                        if (i0 != j0) o[j0 * a.n + i0] -= ga[d] + gb[d];
                    }
                }
            }
        }
        const long long n = a.n;
        auto put = [&](double* M, double x) {
            if (!M) return;
            M[i0 * n + j0] = x;
            M[j0 * n + i0] = x;
        };
        put(a.S, s);
        put(a.T, t);
        if (a.nuc) put(a.V, v);
        if (deriv) {
            const long long nn = n * n;
            auto add = [&](double* base, int atom, int d, double x) {
                double* o = base + (3LL * atom + d) * nn;
                o[i0 * n + j0] += x;
                if (i0 != j0) o[j0 * n + i0] += x;
            };
            for (int d = 0; d < 3; ++d) {
                add(a.dS, P.atom1, d, dsa[d]);
                add(a.dS, P.atom2, d, dsb[d]);
                add(a.dT, P.atom1, d, dta[d]);
                add(a.dT, P.atom2, d, dtb[d]);
                if (!a.nuc) continue;
                add(a.dV, P.atom1, d, dva[d]);
                add(a.dV, P.atom2, d, dvb[d]);
            }
        }
    }
}

// ------------------------------------------------- nuclear attraction (k_nai) ---
// One warp owns (shell pair, slice of the nuclei).  Per nucleus it walks the
// (primitive pair, root) units NAI_UB at a time: three lanes per unit build the three
// directions' 1-D tables (values, and for the derivatives dA and dB) in shared
// memory, then every lane sums the products of its own (component, value) items over
// the units.  The slices of a pair are warps of one block or cluster; their sums meet in
// shared memory, in order, so that one lane writes V(i,j) and V(j,i): symmetric to the bit
// and the same on every call.  (A row of dV takes two atomic adds, the nucleus' own and
// the centres', whose order does not show.)  Bound: shared-memory reads of the product
// step, three per two FP64
// operations; the tables a lane would otherwise recompute per component stay in
// shared memory once per unit.  The Hermite form this replaces kept its E and R tables
// in local memory, once per component and lane: 16 atoms (n = 180), S, T, V and the
// derivatives 129.3 -> 2.3 ms (k_nai 0.98 ms of it).
constexpr int NAI_UB = 10;                                     // units per batch (30 lanes build)
constexpr int NAI_SM = NAI_UB * 9 * (OEI_LMAX + 1) * (OEI_LMAX + 1);  // doubles per warp

template <int LA, int LB, bool DER>
__device__ __forceinline__ void nai_pair(const OeiArgs& a, const PairInfo& P, int c_lo, int c_hi, double* sm,
                                         int lane) {
    constexpr int NR = (LA + LB + (DER ? 1 : 0)) / 2 + 1;
    constexpr int SZ = (LA + 1) * (LB + 1), NT = DER ? 3 : 1, NV = DER ? 6 : 1;
    constexpr int NA = ncart_h(LA), NB = ncart_h(LB), NC = NA * NB, NIT = (NC * NV + 31) / 32;
    constexpr int TOP = LA + LB + (DER ? 1 : 0), NBX = LB + (DER ? 1 : 0);
    constexpr int US = 3 * NT * SZ;  // one unit: [direction][value, dA, dB][a][b]
    constexpr double kfac = 5.914967172795613;
    int off[NIT];  // the item's three table offsets, 10 bits each
#pragma unroll
    for (int j = 0; j < NIT; ++j) {
        const int it = lane + 32 * j, v = it / NC, c = it - v * NC;
        int e[3], f[3];
        off[j] = 0;
        if (it >= NC * NV) continue;
        cart_of(LA, c / NB, e[0], e[1], e[2]);
        cart_of(LB, c % NB, f[0], f[1], f[2]);
        for (int d = 0; d < 3; ++d) {
            const int tab = !DER ? 0 : (v == d ? 1 : (v == d + 3 ? 2 : 0));
            off[j] |= ((d * NT + tab) * SZ + e[d] * (LB + 1) + f[d]) << (10 * d);
        }
    }
    const bool same = P.s1 == P.s2;
    const long long n = a.n, nn = n * n;
    double tot[NIT];  // sums over the nuclei: V, or the dA and dB rows
#pragma unroll
    for (int j = 0; j < NIT; ++j) tot[j] = 0.0;
    const int ul = lane / 3, d = lane - 3 * ul;
    const double PAB = d == 0 ? P.ABx : (d == 1 ? P.ABy : P.ABz);
    const int nu = P.nprim * NR;
    for (int C = c_lo; C < c_hi; ++C) {
        const double Cx = a.xyz[3 * C], Cy = a.xyz[3 * C + 1], Cz = a.xyz[3 * C + 2], Zc = a.Z[C];
        double acc[NIT];
#pragma unroll
        for (int j = 0; j < NIT; ++j) acc[j] = 0.0;
        for (int u0 = 0; u0 < nu; u0 += NAI_UB) {
            const int nb = min(NAI_UB, nu - u0);
            const bool on = ul < nb;
            const int un = u0 + (on ? ul : 0), k = un / NR, r = un - k * NR;
            const PrimPair pp = a.prims[P.prim_off + k];
            const double X = pp.Px - Cx, Y = pp.Py - Cy, W = pp.Pz - Cz;
            const double T = pp.zeta * (X * X + Y * Y + W * W);
            // direction 0's lane evaluates the node, direction 1's the weight
            const double fv = on && d < 2 ? rys_fn<NR>(a.rys, d == 0 ? r : NR + r, T) : 0.0;
            const int src = lane - d < 30 ? lane - d : 0;
            const double u = __shfl_sync(0xffffffffu, fv, src);
            const double wt = __shfl_sync(0xffffffffu, fv, src + 1);
            if (on) {
                const double PC = d == 0 ? X : (d == 1 ? Y : W);
                const double PA = d == 0 ? pp.PAx : (d == 1 ? pp.PAy : pp.PAz);
                const double c00 = PA - u * PC, b10 = pp.oo2z * (1.0 - u);
                double g[NBX + 1][TOP + 1];
                g[0][0] = d == 2 ? -Zc * 2.0 * 3.14159265358979323846 / kfac * pp.K * wt : 1.0;
#pragma unroll
                for (int i = 0; i < TOP; ++i) g[0][i + 1] = c00 * g[0][i] + (i ? i * b10 * g[0][i - 1] : 0.0);
#pragma unroll
                for (int b = 1; b <= NBX; ++b)
#pragma unroll
                    for (int i = 0; i <= TOP - b; ++i) g[b][i] = g[b - 1][i + 1] + PAB * g[b - 1][i];
                double* o = sm + ul * US + d * NT * SZ;
                const double a2 = 2.0 * pp.alpha, b2 = 2.0 * (pp.zeta - pp.alpha);
#pragma unroll
                for (int i = 0; i <= LA; ++i)
#pragma unroll
                    for (int b = 0; b <= LB; ++b) {
                        o[i * (LB + 1) + b] = g[b][i];
                        if constexpr (DER) {
                            o[SZ + i * (LB + 1) + b] = a2 * g[b][i + 1] - (i ? i * g[b][i ? i - 1 : 0] : 0.0);
                            o[2 * SZ + i * (LB + 1) + b] = b2 * g[b + 1][i] - (b ? b * g[b ? b - 1 : 0][i] : 0.0);
                        }
                    }
            }
            __syncwarp();
            for (int q = 0; q < nb; ++q) {
                const double* t = sm + q * US;
#pragma unroll
                for (int j = 0; j < NIT; ++j)
                    acc[j] = fma(t[off[j] & 1023] * t[(off[j] >> 10) & 1023], t[off[j] >> 20], acc[j]);
            }
            __syncwarp();
        }
#pragma unroll
        for (int j = 0; j < NIT; ++j) tot[j] += acc[j];
        if constexpr (DER) {
            // the nucleus by invariance of this term: -(dA + dB)
#pragma unroll
            for (int j = 0; j < NIT; ++j)
                if (lane + 32 * j < NC * NV) sm[lane + 32 * j] = acc[j];
            __syncwarp();
            for (int it = lane; it < 3 * NC; it += 32) {
                const int x = it / NC, c = it - x * NC, ia = c / NB, ib = c - ia * NB;
                if (same && ib > ia) continue;
                const long long i0 = P.bf1 + ia, j0 = P.bf2 + ib;
                const double v = -(sm[it] + sm[it + 3 * NC]);
                double* o = a.dV + (3LL * C + x) * nn;
                atomicAdd(o + i0 * n + j0, v);
                if (i0 != j0) atomicAdd(o + j0 * n + i0, v);
            }
            __syncwarp();
        }
    }
    // the slice's sums, for nai_write
#pragma unroll
    for (int j = 0; j < NIT; ++j)
        if (lane + 32 * j < NC * NV) sm[lane + 32 * j] = tot[j];
}

// A pair's sums over its nslice slices (slice s at part(s)), in order, to V or to the rows
// of its two atoms in dV.
template <bool DER, class Part>
__device__ __forceinline__ void nai_write(const OeiArgs& a, const PairInfo& P, int nslice, int lane, Part&& part) {
    const int nb = ncart_h(P.l2), nc = ncart_h(P.l1) * nb;
    const bool same = P.s1 == P.s2;
    const long long n = a.n, nn = n * n;
    for (int it = lane; it < (DER ? 3 * nc : nc); it += 32) {
        const int x = it / nc, c = it - x * nc, ia = c / nb, ib = c - ia * nb;
        if (same && ib > ia) continue;
        const long long ij = (P.bf1 + ia) * n + P.bf2 + ib, ji = (P.bf2 + ib) * n + P.bf1 + ia;
        double va = 0.0, vb = 0.0;
        for (int s = 0; s < nslice; ++s) {
            const double* q = part(s);
            va += q[it];
            if (DER) vb += q[it + 3 * nc];
        }
        if constexpr (!DER) {
            a.V[ij] = va;
            a.V[ji] = va;
        } else {
            auto add = [&](int atom, double v) {
                double* o = a.dV + (3LL * atom + x) * nn;
                atomicAdd(o + ij, v);
                if (ij != ji) atomicAdd(o + ji, v);
            };
            if (P.atom1 == P.atom2) {
                add(P.atom1, va + vb);
            } else {
                add(P.atom1, va);
                add(P.atom2, vb);
            }
        }
    }
}

// wpp warps of each of ncta blocks (a cluster, if more than one; then wpp = 4) share a
// pair; a slice is `slice` nuclei.
template <bool DER>
__global__ void __launch_bounds__(128) k_nai(OeiArgs a, int slice, int wpp, int ncta) {
    namespace cg = cooperative_groups;
    __shared__ double sm[4][NAI_SM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = blockIdx.x % ncta;
    const int pidx = blockIdx.x / ncta * (4 / wpp) + warp / wpp;
    const int sl = rank * wpp + warp % wpp, nslice = wpp * ncta;
    const int lo = sl * slice, hi = min(a.natom, lo + slice);
    const bool on = pidx < a.npair;
    PairInfo P;
    if (on) {
        P = a.pairs[pidx];
        switch (P.l1 * (OEI_LMAX + 1) + P.l2) {
            case 0: nai_pair<0, 0, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 4: nai_pair<1, 0, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 5: nai_pair<1, 1, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 8: nai_pair<2, 0, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 9: nai_pair<2, 1, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 10: nai_pair<2, 2, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 12: nai_pair<3, 0, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 13: nai_pair<3, 1, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 14: nai_pair<3, 2, DER>(a, P, lo, hi, sm[warp], lane); break;
            case 15: nai_pair<3, 3, DER>(a, P, lo, hi, sm[warp], lane); break;
        }
    }
    // every warp of the block, or cluster, to both barriers
    auto meet = [&] {
        if (ncta > 1) cg::this_cluster().sync();
        else if (wpp > 1) __syncthreads();
        else __syncwarp();
    };
    meet();
    if (on && sl == 0)
        nai_write<DER>(a, P, nslice, lane, [&](int s) {
            double* q = sm[warp + s % wpp];  // this is the pair's first warp
            return (const double*)(s < wpp ? q : cg::this_cluster().map_shared_rank(q, s / wpp));
        });
    if (ncta > 1) cg::this_cluster().sync();  // the other blocks' sums are read before they go
}

}  // namespace qx

template <bool DER>
static void launch_nai(const qx::OeiArgs& a, cudaStream_t s) {
    // slices per pair: a power of two, so that they are warps of one block or whole blocks
    const int want = std::min(a.natom, std::max(1, 148 * 16 / a.npair));
    int nslice = 1;
    while (nslice < want && nslice < 32) nslice *= 2;
    const int wpp = std::min(nslice, 4), ncta = nslice / wpp, ppb = 4 / wpp;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)ncta;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(ncta * ((a.npair + ppb - 1) / ppb)));
    cfg.blockDim = dim3(128);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = ncta > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, qx::k_nai<DER>, a, (a.natom + nslice - 1) / nslice, wpp, ncta);
}

// Launch over every shell pair of a handle; outputs are zeroed by the caller where
// derivatives accumulate.  The nuclei are cut into slices until the warps fill the GPU
// (16 per SM): a small molecule has few pairs, and one warp per pair left most SMs idle.
void qx_launch_oei(const qx::PairInfo* pairs, int npair, const qx::PrimPair* prims, const double* boys, const double* rys,
                   const double* xyz, const double* Z, int natom, long long n, double* S, double* T, double* V,
                   double* dS, double* dT, double* dV, cudaStream_t s) {
    qx::OeiArgs a;
    a.pairs = pairs;
    a.npair = npair;
    a.prims = prims;
    a.boys = boys;
    a.rys = rys;
    a.nuc = natom == 1 ? 1 : 0;
    a.xyz = xyz;
    a.Z = Z;
    a.natom = natom;
    a.n = n;
    a.S = S;
    a.T = T;
    a.V = V;
    a.dS = dS;
    a.dT = dT;
    a.dV = dV;
    const int blocks = (npair + 3) / 4;
    if (!blocks) return;
    if (S || T || dS || a.nuc) qx::k_oei<<<blocks, 128, 0, s>>>(a);
    if (a.nuc) return;
    if (dV) launch_nai<true>(a, s);
    else if (V) launch_nai<false>(a, s);
}
