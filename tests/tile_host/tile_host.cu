// Host build of the tile engine's phases (test infrastructure).
//
// The device kernel runs the same functions (qx_tile.cuh) over a block with barriers
// between them; here the threads of a block take their turns one after another, phase by
// phase, so a machine without a GPU checks
// the arithmetic and the index tables against the oracle: plain blocks and the adjoint
// gradient of a shell quartet.
#include <cmath>
#include <vector>

#include "qx_tile.cuh"

using namespace qx;

namespace {

const double g_tab[] = {QX_RYS_TAB_DATA QX_RYS_ASYM_Y_DATA, QX_RYS_ASYM_W_DATA};

void make_pair(int l1, int l2, int n1, int n2, const double* A, const double* B, const double* e1, const double* e2,
               const double* w1, const double* w2, PairInfo& P, std::vector<PrimPair>& pr) {
    const double kfac = std::sqrt(2.0) * std::pow(M_PI, 1.25);
    P.Ax = A[0]; P.Ay = A[1]; P.Az = A[2];
    P.ABx = A[0] - B[0]; P.ABy = A[1] - B[1]; P.ABz = A[2] - B[2];
    const double AB2 = P.ABx * P.ABx + P.ABy * P.ABy + P.ABz * P.ABz;
    P.nprim = n1 * n2;
    P.prim_off = 0;
    P.l1 = l1;
    P.l2 = l2;
    for (int i = 0; i < n1; ++i)
        for (int j = 0; j < n2; ++j) {
            PrimPair r;
            const double x = e1[i], y = e2[j];
            r.zeta = x + y;
            r.oo2z = 0.5 / r.zeta;
            r.PAx = -(y / r.zeta) * (A[0] - B[0]);
            r.PAy = -(y / r.zeta) * (A[1] - B[1]);
            r.PAz = -(y / r.zeta) * (A[2] - B[2]);
            r.Px = A[0] + r.PAx; r.Py = A[1] + r.PAy; r.Pz = A[2] + r.PAz;
            r.K = kfac * w1[i] * w2[j] * std::exp(-x * y / r.zeta * AB2) / r.zeta;
            r.alpha = x;
            pr.push_back(r);
        }
}

template <int LA, int LB, int LC, int LD, int KIND>
int run(const double* cen, const int* np, const double* ex, const double* cw, const double* D,
        int parts, double* out) {
    using C = TileCls<LA, LB, LC, LD, KIND>;
    using Bra = typename C::Bra;
    using Ket = typename C::Ket;
    TileQuartet w;
    std::vector<PrimPair> pp, qq;
    const int o[4] = {0, np[0], np[0] + np[1], np[0] + np[1] + np[2]};
    make_pair(LA, LB, np[0], np[1], cen, cen + 3, ex + o[0], ex + o[1], cw + o[0], cw + o[1], w.P, pp);
    make_pair(LC, LD, np[2], np[3], cen + 6, cen + 9, ex + o[2], ex + o[3], cw + o[2], cw + o[3], w.Q, qq);
    w.P.bf1 = 0; w.P.bf2 = Bra::N1; w.Q.bf1 = w.P.bf2 + Bra::N2; w.Q.bf2 = w.Q.bf1 + Ket::N1;
    const long long n = w.Q.bf2 + Ket::N2;
    w.P.s1 = 0; w.P.s2 = 1; w.Q.s1 = 2; w.Q.s2 = 3;
    w.P.atom1 = 0; w.P.atom2 = 1; w.Q.atom1 = 2; w.Q.atom2 = 3;
    std::vector<double> coA(Bra::NCOMBO * (C::DER ? 4 : 1)), coC(Ket::NCOMBO * (C::DER ? 4 : 1));
    std::vector<double> den(C::NDEN + 1), sc(C::NSC + 1), uw(C::UW);
    const auto& tb = g_tile_tab<LA, LB>;
    const auto& tk = g_tile_tab<LC, LD>;
    const double AB[3] = {w.P.ABx, w.P.ABy, w.P.ABz}, CD[3] = {w.Q.ABx, w.Q.ABy, w.Q.ABz};
    constexpr int NT = C::NT;
    for (int t = 0; t < NT; ++t) {
        tl_coefs<Bra, C::DER>(tb, AB, coA.data(), t, NT);
        tl_coefs<Ket, C::DER>(tk, CD, coC.data(), t, NT);
    }
    const TileGamma<C> gam = tl_gamma<C>(den.data(), w.P, w.Q, true, 1.0, -0.5);
    std::vector<double> Gf(C::NE * C::NFP), H(C::X + 1), U(C::NE * C::NFP);
    if (C::DER) {
        for (int t = 0; t < NT; ++t) tl_density<C>(D, n, w.P, w.Q, den.data(), t, NT);
        for (int t = 0; t < NT; ++t) tl_gam_ket<C>(tk, coC.data(), gam, H.data(), t, NT);
        for (int t = 0; t < NT; ++t) tl_gam_bra<C>(tb, coA.data(), H.data(), Gf.data(), t, NT);
    }
    for (int i = 0; i < (KIND == TK_PLAIN ? C::NCOMP : 9); ++i) out[i] = 0.0;
    const int ntot = w.P.nprim * w.Q.nprim;
    for (int blk = 0; blk < parts * C::NPASS; ++blk) {
        const int part = blk / C::NPASS, pass = blk % C::NPASS;
        if (part * C::PB >= ntot) continue;
        std::vector<TileThread<C>> th(NT);
        for (int t = 0; t < NT; ++t) {
            for (auto& u : th[t].U) u = 0.0;
            for (auto& g : th[t].g) g = 0.0;
            const TileRole<C> role(t, pass);
            if constexpr (C::DER) tl_load<C, 0>(role.on ? role.chunk : 0, Gf.data(), role.f, th[t]);
        }
        for (int t0 = part * C::PB; t0 < ntot; t0 += parts * C::PB) {
            const int nb = std::min(C::PB, ntot - t0);
            std::vector<double> tab((size_t)C::PB * C::PER_PRIM, NAN);  // a read of an unbuilt entry shows
            for (int t = 0; t < NT; ++t) tl_nodes<C>(g_tab, w, pp.data(), qq.data(), t0, nb, uw.data(), sc.data(), t, NT);
            for (int t = 0; t < NT; ++t) tl_tables<C>(w, pp.data(), qq.data(), t0, nb, uw.data(), tab.data(), t, NT);
            for (int t = 0; t < NT; ++t) {
                const TileRole<C> role(t, pass);
                if (!role.on) continue;
                const int fx = tk.ex[role.f], fy = tk.ey[role.f], fz = tk.ez[role.f];
                for (int p = role.sub; p < nb; p += C::NP)
                    tl_prim_chunk<C, 0>(role.chunk, tab.data() + (size_t)p * C::PER_PRIM, uw.data() + 2 * C::NR * p, fx, fy,
                                        fz, sc.data() + C::SCP * p, w, th[t]);
            }
        }
        // U of the primitives side by side: sub 0 stores, the others are added
        std::vector<double> one(C::NE * C::NFP);
        for (auto& u : U) u = 0.0;
        for (int sub = 0; sub < C::NP; ++sub) {
            for (auto& u : one) u = 0.0;
            for (int t = 0; t < NT; ++t) {
                const TileRole<C> role(t, pass);
                if (role.on && role.sub == sub) tl_store<C, 0>(role.chunk, one.data(), role.f, th[t]);
            }
            for (int i = 0; i < C::NE * C::NFP; ++i)
                if (i % C::NFP < C::NF) U[i] += one[i];
        }
        if constexpr (C::DER) {
            double g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int t = 0; t < NT; ++t) tl_gam_ket<C>(tk, coC.data(), gam, H.data(), t, NT);
            for (int t = 0; t < NT; ++t) tl_x_bra<C>(tb, coA.data(), U.data(), H.data(), g, t, NT);
            for (int t = 0; t < NT; ++t) tl_gam_bra2<C>(tb, coA.data(), gam, H.data(), t, NT);
            for (int t = 0; t < NT; ++t) tl_x_ket<C>(tk, coC.data(), U.data(), H.data(), g, t, NT);
            for (int t = 0; t < NT; ++t)
                for (int i = 0; i < 9; ++i) g[i] += th[t].g[i];
            for (int i = 0; i < 9; ++i) out[i] += g[i];
        } else {
            for (int t = 0; t < NT; ++t) tl_fwd_bra<C>(tb, coA.data(), U.data(), H.data(), t, NT);
            for (int x = 0; x < C::NCOMP; ++x)
                out[x] += tl_fwd_ket<C>(tk, coC.data(), H.data(), x / C::NCD, x % C::NCD);
        }
    }
    return 0;
}

template <int LA, int LB, int LC, int LD>
int pick(int kind, const double* cen, const int* np, const double* ex, const double* cw, const double* D,
         int parts, double* out) {
    if (kind == 0) return run<LA, LB, LC, LD, TK_PLAIN>(cen, np, ex, cw, D, parts, out);
    return run<LA, LB, LC, LD, TK_GRAD>(cen, np, ex, cw, D, parts, out);
}

}  // namespace

#define TILE_HOST_CLASSES(X)                                                                                        \
    X(0, 0, 0, 0) X(1, 0, 0, 0) X(1, 1, 1, 0) X(2, 0, 1, 1) X(2, 1, 2, 0) X(2, 1, 2, 1) X(2, 2, 1, 0) X(2, 2, 2, 2) \
    X(3, 0, 0, 0) X(3, 0, 2, 2) X(3, 1, 3, 0) X(3, 2, 2, 2) X(3, 3, 3, 1) X(3, 3, 3, 3)

extern "C" int tile_host(int cls, int kind, int* l4, const double* cen, const int* np, const double* ex,
                         const double* cw, const double* D, int parts, double* out) {
    int k = 0;
#define X(a, b, c, d)                                                                      \
    if (k++ == cls) {                                                                      \
        l4[0] = a; l4[1] = b; l4[2] = c; l4[3] = d;                                        \
        return out ? pick<a, b, c, d>(kind, cen, np, ex, cw, D, parts, out) : 0;      \
    }
    TILE_HOST_CLASSES(X)
#undef X
    return -1;
}
