// Host build of the plain integrals' phases (test infrastructure): the device kernel's
// functions (qx_plain.cuh) over one shell quartet, the threads of a block taking turns
// phase by phase; the same block from the table engine's phases (qx_rys.cuh); and from an
// 80-bit evaluation of the Coulomb kernel's quadrature.
#include <cmath>
#include <vector>

#include "qx_plain.cuh"

using namespace qx;

namespace {

typedef long double ld;
const double g_tab[] = {QX_RYS_TAB_DATA QX_RYS_ASYM_Y_DATA, QX_RYS_ASYM_W_DATA};

struct Quartet {
    const double *cen, *ex, *cw;
    int l[4], n[4], o[4];
    void pair(int s, PairInfo& P, std::vector<PrimPair>& pr) const {
        const double kfac = std::sqrt(2.0) * std::pow(M_PI, 1.25);
        const double *A = cen + 3 * s, *B = A + 3;
        P.Ax = A[0]; P.Ay = A[1]; P.Az = A[2];
        P.ABx = A[0] - B[0]; P.ABy = A[1] - B[1]; P.ABz = A[2] - B[2];
        const double AB2 = P.ABx * P.ABx + P.ABy * P.ABy + P.ABz * P.ABz;
        P.nprim = n[s] * n[s + 1];
        P.prim_off = 0;
        P.l1 = l[s];
        P.l2 = l[s + 1];
        for (int i = 0; i < n[s]; ++i)
            for (int j = 0; j < n[s + 1]; ++j) {
                const double x = ex[o[s] + i], y = ex[o[s + 1] + j];
                PrimPair r;
                r.zeta = x + y;
                r.oo2z = 0.5 / r.zeta;
                r.PAx = -(y / r.zeta) * P.ABx;
                r.PAy = -(y / r.zeta) * P.ABy;
                r.PAz = -(y / r.zeta) * P.ABz;
                r.Px = A[0] + r.PAx; r.Py = A[1] + r.PAy; r.Pz = A[2] + r.PAz;
                r.K = kfac * cw[o[s] + i] * cw[o[s + 1] + j] * std::exp(-x * y / r.zeta * AB2) / r.zeta;
                r.alpha = x;
                pr.push_back(r);
            }
    }
};

template <int LA, int LB, int LC, int LD>
void run_plain(const Quartet& q, int parts, double* out) {
    using C = PlainCls<LA, LB, LC, LD>;
    constexpr int NT = C::NT;
    TileQuartet w;
    std::vector<PrimPair> pp, qq;
    q.pair(0, w.P, pp);
    q.pair(2, w.Q, qq);
    const int ntot = w.P.nprim * w.Q.nprim;
    for (int i = 0; i < C::NCOMP; ++i) out[i] = 0.0;
    std::vector<double> uw(C::UW), one(C::NCOMP);
    for (int part = 0; part < parts; ++part) {
        struct Thread {
            double U[C::NSLOT];
        };
        std::vector<Thread> th(NT, Thread{});
        for (int t0 = part * C::PB; t0 < ntot; t0 += parts * C::PB) {
            const int nb = std::min(C::PB, ntot - t0);
            std::vector<double> tab((size_t)C::TABS, NAN);  // a read of an unbuilt entry shows
            for (int t = 0; t < NT; ++t) tl_nodes<C>(g_tab, w, pp.data(), qq.data(), t0, nb, uw.data(), nullptr, t, NT);
            for (int t = 0; t < NT; ++t) pl_tables<C>(w, pp.data(), qq.data(), t0, nb, uw.data(), tab.data(), t, NT);
            if (LD > 0)
                for (int t = 0; t < NT; ++t) pl_ket<C>(w, nb, tab.data(), t, NT);
            for (int t = 0; t < NT; ++t) {
                const TileRole<C> role(t, 0);
                const PlainLane<C> lane(role.f);
                if (role.on)
                    for (int p = role.sub; p < nb; p += C::NP)
                        pl_prim_chunk<C, 0>(role.chunk, tab.data() + (size_t)p * C::PER_PRIM, lane, th[t].U);
            }
        }
        for (int sub = 0; sub < C::NP; ++sub) {
            for (auto& v : one) v = 0.0;
            for (int t = 0; t < NT; ++t) {
                const TileRole<C> role(t, 0);
                if (role.on && role.sub == sub) pl_store<C, 0>(role.chunk, one.data(), role.f, th[t].U);
            }
            for (int i = 0; i < C::NCOMP; ++i) out[i] += one[i];
        }
    }
}

template <int LA, int LB, int LC, int LD>
void run_table(const Quartet& q, double* out) {
    using C = RysCls<LA, LB, LC, LD, RK_PLAIN>;
    PairInfo P, Q;
    std::vector<PrimPair> pp, qq;
    q.pair(0, P, pp);
    q.pair(2, Q, qq);
    std::vector<double> uw(2 * C::NR), U((size_t)C::NR * 3 * C::USZ);
    for (int i = 0; i < C::NCOMP; ++i) out[i] = 0.0;
    for (const PrimPair& p : pp)
        for (const PrimPair& r : qq) {
            RysPrim st;
            rys_prim(p, r, P, Q, st);
            for (int f = 0; f < 2 * C::NR; ++f) uw[f] = rys_fn<C::NR>(g_tab, f, st.T) * (f >= C::NR ? st.pref : 1.0);
            for (int rb0 = 0; rb0 < C::NR; rb0 += C::RB) {
                const int nrb = std::min(C::RB, C::NR - rb0);
                rys_phase_units<C>(st, uw.data(), rb0, nrb, U.data(), 0, 1);
                for (int kc = 0; kc < C::NCOMP; ++kc)
                    out[kc] += rys_prod_plain<C>(U.data(), nrb, rys_comp_offsets<C, LA, LB, LC, LD, C::RAW>(kc));
            }
        }
}

// Gauss-Legendre rule on [0, 1].
struct Legendre {
    static constexpr int N = 80;
    ld x[N], w[N];
    Legendre() {
        for (int i = 0; i < N; ++i) {
            ld z = cosl(M_PIl * (i + 0.75L) / (N + 0.5L)), d = 0;
            for (int it = 0; it < 20; ++it) {
                ld p = 1, p1 = 0;
                for (int k = 0; k < N; ++k) {
                    const ld p2 = p1;
                    p1 = p;
                    p = ((2 * k + 1) * z * p1 - k * p2) / (k + 1);
                }
                d = N * (z * p - p1) / (z * z - 1);
                z -= p / d;
            }
            x[i] = (1 + z) / 2;
            w[i] = 1 / ((1 - z * z) * d * d);
        }
    }
};

void run_exact(const Quartet& q, double* out) {
    static const Legendre g;
    const int *l = q.l, NI = l[0] + l[1] + 1, NK = l[2] + l[3] + 1;
    int nc[4], ncomp = 1;
    for (int s = 0; s < 4; ++s) ncomp *= nc[s] = (l[s] + 1) * (l[s] + 2) / 2;
    std::vector<ld> sum(ncomp, 0.0L);
    auto at = [&](int a, int b, int c, int d) { return ((a * (l[1] + 1) + b) * (l[2] + 1) + c) * (l[3] + 1) + d; };
    std::vector<ld> T[3];
    for (auto& t : T) t.resize(at(l[0], l[1], l[2], l[3]) + 1);
    for (int i = 0; i < q.n[0]; ++i)
        for (int j = 0; j < q.n[1]; ++j)
            for (int k = 0; k < q.n[2]; ++k)
                for (int m = 0; m < q.n[3]; ++m) {
                    const ld a = q.ex[q.o[0] + i], b = q.ex[q.o[1] + j], c = q.ex[q.o[2] + k], d = q.ex[q.o[3] + m];
                    const ld z = a + b, h = c + d, rho = z * h / (z + h);
                    ld AB[3], CD[3], PA[3], QC[3], PQ[3], ab2 = 0, cd2 = 0, pq2 = 0;
                    for (int x = 0; x < 3; ++x) {
                        AB[x] = (ld)q.cen[x] - q.cen[3 + x];
                        CD[x] = (ld)q.cen[6 + x] - q.cen[9 + x];
                        PA[x] = -b / z * AB[x];
                        QC[x] = -d / h * CD[x];
                        PQ[x] = (ld)q.cen[x] - q.cen[6 + x] + PA[x] - QC[x];
                        ab2 += AB[x] * AB[x];
                        cd2 += CD[x] * CD[x];
                        pq2 += PQ[x] * PQ[x];
                    }
                    const ld pref = 2 * powl(M_PIl, 2.5L) / (z * h * sqrtl(z + h)) * expl(-a * b / z * ab2 - c * d / h * cd2) *
                                    q.cw[q.o[0] + i] * q.cw[q.o[1] + j] * q.cw[q.o[2] + k] * q.cw[q.o[3] + m];
                    const ld top = std::min(1.0L, 7.0L / sqrtl(std::max(rho * pq2, 1e-30L)));
                    for (int n = 0; n < Legendre::N; ++n) {
                        const ld t = top * g.x[n], u = t * t, wt = pref * top * g.w[n] * expl(-rho * pq2 * u);
                        const ld b00 = u / (2 * (z + h)), b10 = (1 - u * h / (z + h)) / (2 * z), b01 = (1 - u * z / (z + h)) / (2 * h);
                        for (int x = 0; x < 3; ++x) {
                            const ld c00 = PA[x] - u * h / (z + h) * PQ[x], d00 = QC[x] + u * z / (z + h) * PQ[x];
                            ld I[8][8];
                            I[0][0] = x == 2 ? wt : 1.0L;
                            for (int e = 1; e < NI; ++e) I[e][0] = c00 * I[e - 1][0] + (e > 1 ? (e - 1) * b10 * I[e - 2][0] : 0);
                            for (int f = 1; f < NK; ++f)
                                for (int e = 0; e < NI; ++e)
                                    I[e][f] = d00 * I[e][f - 1] + (f > 1 ? (f - 1) * b01 * I[e][f - 2] : 0) + (e ? e * b00 * I[e - 1][f - 1] : 0);
                            for (int bb = 0; bb <= l[1]; ++bb) {
                                ld K[8][8];
                                for (int e = 0; e < NI - bb; ++e)
                                    for (int f = 0; f < NK; ++f) K[e][f] = I[e][f];
                                for (int dd = 0; dd <= l[3]; ++dd) {
                                    for (int aa = 0; aa <= l[0]; ++aa)
                                        for (int cc = 0; cc <= l[2]; ++cc) T[x][at(aa, bb, cc, dd)] = K[aa][cc];
                                    for (int e = 0; e <= l[0]; ++e)
                                        for (int f = 0; f + 1 + dd < NK; ++f) K[e][f] = K[e][f + 1] + CD[x] * K[e][f];
                                }
                                for (int f = 0; f < NK; ++f)
                                    for (int e = 0; e + 1 + bb < NI; ++e) I[e][f] = I[e + 1][f] + AB[x] * I[e][f];
                            }
                        }
                        int o = 0;
                        for (int A = 0; A < nc[0]; ++A)
                            for (int B = 0; B < nc[1]; ++B)
                                for (int Cc = 0; Cc < nc[2]; ++Cc)
                                    for (int D = 0; D < nc[3]; ++D, ++o) {
                                        int e[4][3];
                                        pl_cart(l[0], A, e[0][0], e[0][1], e[0][2]);
                                        pl_cart(l[1], B, e[1][0], e[1][1], e[1][2]);
                                        pl_cart(l[2], Cc, e[2][0], e[2][1], e[2][2]);
                                        pl_cart(l[3], D, e[3][0], e[3][1], e[3][2]);
                                        ld v = 1;
                                        for (int x = 0; x < 3; ++x) v *= T[x][at(e[0][x], e[1][x], e[2][x], e[3][x])];
                                        sum[o] += v;
                                    }
                    }
                }
    for (int o = 0; o < ncomp; ++o) out[o] = (double)sum[o];
}

template <int LA, int LB, int LC, int LD>
void pick(const Quartet& q, int what, int parts, double* out) {
    if (what == 0) run_plain<LA, LB, LC, LD>(q, parts, out);
    if (what == 1) run_table<LA, LB, LC, LD>(q, out);
    if (what == 2) run_exact(q, out);
}

}  // namespace

#define PLAIN_HOST_CLASSES(X)                                                                                       \
    X(0, 0, 0, 0) X(1, 1, 1, 0) X(2, 1, 1, 1) X(2, 2, 2, 1) X(3, 0, 0, 0) X(3, 0, 2, 2) X(3, 1, 3, 0) X(3, 2, 1, 0) \
    X(3, 1, 2, 2) X(3, 2, 2, 2) X(3, 3, 2, 0) X(3, 3, 2, 2) X(3, 3, 3, 3)

// what: 0 the phases of qx_plain.cuh (`parts` parts), 1 the table engine's, 2 80 bits.
extern "C" int plain_host(int cls, int what, int* l4, const double* cen, const int* np, const double* ex,
                          const double* cw, int parts, double* out) {
    int k = 0;
#define X(a, b, c, d)                                                              \
    if (k++ == cls) {                                                              \
        l4[0] = a; l4[1] = b; l4[2] = c; l4[3] = d;                                \
        if (!out) return 0;                                                        \
        const Quartet q{cen, ex, cw, {a, b, c, d}, {np[0], np[1], np[2], np[3]},   \
                        {0, np[0], np[0] + np[1], np[0] + np[1] + np[2]}};         \
        pick<a, b, c, d>(q, what, parts, out);                                     \
        return 0;                                                                  \
    }
    PLAIN_HOST_CLASSES(X)
#undef X
    return -1;
}
