"""The work a user of this package has it do, as measurable cases.

Every case names a kind (an entry point and how it is called) and a molecule: H2O in
STO-3G, or a synthetic molecule of the shapes the benchmark uses (s, p, d shells of 1-8
primitives, with `f` also f shells of 1-3, K and exponents drawn from the case's `mol`).
`prepare` displaces the geometry by 0.05 bohr (the batched workload's displaced
geometries) and draws the density from its own seed, builds the engine -- the handle a
program keeps for a geometry -- and the buffers the call writes; `run` is the call.

`exact` evaluates the same integrals in plain torch FP64, by numerical quadrature of the
Coulomb kernel, for the molecules small enough for that.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from quax_b200.basis import Basis, Molecule, Shell, SyntheticSpec, build_basis, h2o_config1, synthetic_molecule
from quax_b200.integrals.engine import EriEngine
from quax_b200.integrals.spherical import SphericalEngine
from quax_b200.methods.hartree_fock import rhf_gradient

TOL = 1.0e-12  # Schwarz threshold of the benchmark's workloads
SIGMA = 0.05  # bohr, displacement of the geometries

# The cases, smallest calls first.  natom 0 stands for H2O/STO-3G.
_LISTED = [
    # the integral tensor of a tiny molecule: what a first call costs, all latency
    dict(name="eri_h2o", kind="eri", natom=0, mol=0, f=False),
    # second-derivative tensor of a tiny molecule: a Hessian the way the reference forms it
    dict(name="deriv2_h2o", kind="deriv2", natom=0, mol=0, f=False),
    # a whole calculation of a tiny molecule: set-up, SCF and analytic gradient
    dict(name="rhf_h2o", kind="rhf", natom=0, mol=0, f=False),
    # first-derivative tensor with d shells, the input of derivative transforms
    dict(name="deriv1_3", kind="deriv1", natom=3, mol=1, f=False),
    # the throughput workload: every screened unique integral of ten atoms
    dict(name="unique_10", kind="unique", natom=10, mol=0, f=False),
    # the dense tensor a correlated method starts from
    dict(name="eri_8", kind="eri", natom=8, mol=2, f=False),
    # one Fock build of a mid-sized molecule
    dict(name="jk_12", kind="jk", natom=12, mol=3, f=False),
    # one Fock build of a molecule with f shells
    dict(name="jk_f6", kind="jk", natom=6, mol=4, f=True),
    # the two-electron gradient of the benchmark's ten atoms
    dict(name="grad_10", kind="grad", natom=10, mol=0, f=False),
    # the same with f shells
    dict(name="grad_f6", kind="grad", natom=6, mol=4, f=True),
    # a Hessian-vector product of the two-electron energy
    dict(name="hvp_5", kind="hvp", natom=5, mol=5, f=False),
    # overlap, kinetic and nuclear attraction with their derivatives
    dict(name="oei_16", kind="oei", natom=16, mol=6, f=False),
]

# Atoms a drawn case of a kind may have, without and with f shells; and the listed kind
# whose dearest case bounds its cost.
_RANGE = {"eri": ((1, 8), (1, 4), "eri"), "deriv2": ((2, 3), None, "hvp"), "deriv1": ((2, 4), (2, 2), "grad"),
          "unique": ((2, 10), (1, 4), "unique"), "jk": ((2, 12), (1, 6), "jk"),
          "jk_pure": ((2, 12), (1, 6), "jk"), "jk_screened": ((2, 12), (1, 6), "jk"), "grad": ((2, 10), (2, 6), "grad"),
          "hvp": ((2, 5), (2, 2), "hvp"), "oei": ((1, 16), (1, 12), "oei")}


def listed():
    return [dict(c) for c in _LISTED]


def _spec(case) -> SyntheticSpec:
    return SyntheticSpec(natom=case["natom"], f_shell=case["f"], pure=case["kind"] == "jk_pure")


def _molecule(case):
    """(molecule, basis) of a case before its geometry is displaced."""
    if case["natom"] == 0:
        mol = h2o_config1()
        return mol, build_basis(mol, "sto-3g")
    return synthetic_molecule(_spec(case), case["mol"])


@functools.lru_cache
def _dearest(kind, f):
    return max((work(c)["flops"] for c in _LISTED if c["kind"] == kind and c["f"] == f), default=math.inf)


def draw(rng):
    while True:
        kind = rng.choice(list(_RANGE))
        f = _RANGE[kind][1] is not None and rng.random() < 0.4
        lo, hi = _RANGE[kind][f]
        natom = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        case = dict(kind=kind, natom=natom, mol=rng.randrange(10, 1 << 20), f=f)
        if work(case)["flops"] <= min(_dearest(_RANGE[kind][2], False), _dearest(_RANGE[kind][2], f)):
            return case


# ------------------------------------------------------------------- the calls ----
def _displaced(case, seed):
    mol, basis = _molecule(case)
    rng = np.random.default_rng(seed)
    xyz = mol.coords + rng.normal(0.0, SIGMA, size=mol.coords.shape)
    return Molecule(mol.Z, xyz, mol.charge), basis.with_coords(xyz), rng


def _density(n, rng):
    """D = C C^T, C n x n/4 with N(0, 1/n) entries."""
    c = rng.normal(0.0, 1.0 / math.sqrt(n), size=(n, max(1, n // 4)))
    return c @ c.T


def prepare(case, seed):
    mol, basis, rng = _displaced(case, seed)
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "rhf":
        st.update(mol=mol, basis=basis)
        return st
    eng = (SphericalEngine if kind == "jk_pure" else EriEngine)(basis, TOL)
    n = eng.nbf
    st["eng"] = eng
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    empty = lambda *s: torch.empty(s, dtype=torch.float64, device="cuda")  # noqa: E731
    if kind == "eri":
        st["out"] = empty(n, n, n, n)
    elif kind == "unique":
        # room for every unique quartet: how many the screening keeps depends on the geometry
        pairs = [_nc(a.l) * _nc(b.l) for i, a in enumerate(basis.shells) for b in basis.shells[: i + 1]]
        st["out"] = empty((sum(pairs) ** 2 + sum(p * p for p in pairs)) // 2).zero_()
    elif kind in ("deriv1", "deriv2"):
        m = 3 * basis.natom
        st["out"] = empty(m if kind == "deriv1" else m * (m + 1) // 2, n, n, n, n)
    elif kind in ("jk", "jk_pure", "jk_screened", "grad", "hvp"):
        D = _density(n, rng)
        if kind == "jk_screened":  # the density change of a late SCF iteration
            D *= 1.0e-4
        st.update(D=dev(D), J=empty(n, n), K=empty(n, n), g=empty(3 * basis.natom))
        if kind == "hvp":
            st["v"] = dev(rng.normal(size=3 * basis.natom))
    elif kind == "oei":
        eng.set_charges(mol.Z)
    return st


def run(st):
    kind = st["kind"]
    if kind == "rhf":
        e, g = rhf_gradient(st["mol"], st["basis"])
        return {"energy": e, "gradient": g}
    eng = st["eng"]
    if kind == "eri":
        return eng.eri(st["out"])
    if kind == "unique":
        # class by class, quartets in the handle's list order
        return eng.eri_unique(st["out"])
    if kind in ("deriv1", "deriv2"):
        return eng.eri_deriv_core(int(kind[-1]), st["out"])
    if kind == "jk":
        return eng.jk(st["D"], st["J"], st["K"])
    if kind == "jk_pure":
        return eng.jk(st["D"])
    if kind == "jk_screened":
        return eng.jk(st["D"], st["J"], st["K"], screen=1.0e-10)
    if kind == "grad":
        return eng.grad_adjoint(st["D"], 2.0, -1.0, st["g"])
    if kind == "hvp":
        return eng.grad_adjoint_jvp(st["D"], st["v"], 2.0, -1.0)
    S, T, V = eng.oei()
    dS, dT, dV = eng.oei_deriv(1)
    return {"S": S, "T": T, "V": V, "dS": dS, "dT": dT, "dV": dV}


# ------------------------------------------------------------------- the work -----
def _nc(l):
    return (l + 1) * (l + 2) // 2


def _hgp(la, lb):
    """Cartesian functions of the angular momenta la .. la + lb."""
    return sum(_nc(l) for l in range(la, la + lb + 1))


def _quartet_counts(basis):
    """{(la, lb, lc, ld): (quartets, primitive quartets)} of the unique shell quartets
    that an overlap estimate of their size keeps."""
    sh = basis.shells
    groups = {}
    for i, a in enumerate(sh):
        for b in sh[: i + 1]:
            p, q = (a, b) if a.l >= b.l else (b, a)
            ca, cb = p.norm_coefs(), q.norm_coefs()
            z = p.exps[:, None] + q.exps[None, :]
            r2 = float(np.sum((p.center - q.center) ** 2))
            m = np.abs(ca[:, None] * cb[None, :]) * np.exp(-p.exps[:, None] * q.exps[None, :] / z * r2) / z
            groups.setdefault((p.l, q.l), []).append((float(m.sum()), p.nprim * q.nprim))
    out = {}
    keys = sorted(groups)
    for x, kb in enumerate(keys):
        mb, nb = map(np.asarray, zip(*groups[kb]))
        for kk in keys[: x + 1]:
            order = np.argsort([-m for m, _ in groups[kk]])
            mk, nk = (np.asarray([groups[kk][o][t] for o in order]) for t in (0, 1))
            cum = np.concatenate([[0], np.cumsum(nk)])
            kept = np.searchsorted(-mk, -TOL / np.maximum(mb, 1e-300), side="right")
            nq, npq = float(kept.sum()), float((nb * cum[kept]).sum())
            half = 0.5 if kb == kk else 1.0  # both orders of a pair of pairs were counted
            out[kb + kk] = (half * nq, half * npq)
    return out


def work(case):
    """Inputs read once and outputs written once.  Operations: per primitive quartet two
    for every (e0|f0) value its class needs (times the ten values a first and the 45 + 10 a
    second derivative take per value, three where they are contracted), and two per
    output."""
    _, basis = _molecule(case)
    kind, n, m = case["kind"], basis.nbf(), 3 * basis.natom
    shells = 16.0 * sum(s.nprim for s in basis.shells) + 24.0 * basis.natom
    if kind == "oei":
        sh = basis.shells
        prims = sum(_nc(a.l) * _nc(b.l) * a.nprim * b.nprim for i, a in enumerate(sh) for b in sh[: i + 1])
        return {"bytes": shells + 8.0 * 3 * n * n * (1 + m), "flops": 20.0 * prims * basis.natom}
    per_value = {"deriv1": 10.0, "deriv2": 55.0, "grad": 3.0, "hvp": 9.0, "rhf": 12.0}.get(kind, 1.0)
    flops = unique = 0.0
    for (la, lb, lc, ld), (nq, npq) in _quartet_counts(basis).items():
        outs = _nc(la) * _nc(lb) * _nc(lc) * _nc(ld)
        flops += 2.0 * per_value * (npq * _hgp(la, lb) * _hgp(lc, ld) + nq * outs)
        unique += nq * outs
    out = {"eri": n**4, "deriv1": m * n**4, "deriv2": m * (m + 1) // 2 * n**4, "unique": unique,
           "grad": n * n + m, "hvp": n * n + 2 * m, "rhf": m}.get(kind, 3 * n * n)
    return {"bytes": shells + 8.0 * out, "flops": flops}


# --------------------------------------------------- plain FP64 evaluation --------
# (ab|cd) = sum over primitives of pref * int_0^1 Ix Iy Iz exp(-T t^2) dt, with Ix, Iy, Iz
# polynomials in t^2 from one-dimensional recurrences.  The integral is a Gauss-Legendre
# sum over s = t sqrt(T) up to where exp(-s^2) has vanished; derivatives act on one
# direction's factor, d g_a / dA = 2 alpha g_{a+1} - a g_{a-1}.
_NODES = 44


def _components(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


class _Pair:
    """The primitive pairs of one class's shell pairs: flat arrays over (pair, i, j)."""

    def __init__(self, shells, pairs):
        P = {k: [] for k in ("own", "a", "b", "A", "B", "c")}
        for own, (s, t) in enumerate(pairs):
            p, q = shells[s], shells[t]
            for a, ca in zip(p.exps, p.norm_coefs()):
                for b, cb in zip(q.exps, q.norm_coefs()):
                    for k, v in zip(P, (own, a, b, p.center, q.center, ca * cb)):
                        P[k].append(v)
        t = lambda k: torch.as_tensor(np.asarray(P[k]), dtype=torch.float64, device="cuda")  # noqa: E731
        self.own = t("own").long()
        self.a, self.b, self.A, self.B = t("a"), t("b"), t("A"), t("B")
        self.z = self.a + self.b
        self.P = (self.a[:, None] * self.A + self.b[:, None] * self.B) / self.z[:, None]
        self.c = t("c") * torch.exp(-self.a * self.b / self.z * ((self.A - self.B) ** 2).sum(1))


def _legendre():
    x, w = np.polynomial.legendre.leggauss(_NODES)
    return (torch.as_tensor(0.5 * (x + 1.0), device="cuda"), torch.as_tensor(0.5 * w, device="cuda"))


def _transfer(T, n1, n2, D):
    """[a][b] tables from T[a] (a = 0 .. n1 + n2) by I(a, b + 1) = I(a + 1, b) + D I(a, b)."""
    cols = [T]
    for _ in range(n2):
        p = cols[-1]
        cols.append([p[i + 1] + D * p[i] for i in range(len(p) - 1)])
    return [[cols[b][a] for b in range(n2 + 1)] for a in range(n1 + 1)]


def _raise(I, axis, e2):
    """d/dX of a table I[idx] (a dict over (a, b, c, d)) on one centre."""
    out = {}
    for k in I:
        up = k[:axis] + (k[axis] + 1,) + k[axis + 1:]
        if up not in I:
            continue
        v = e2 * I[up]
        if k[axis]:
            v = v - k[axis] * I[k[:axis] + (k[axis] - 1,) + k[axis + 1:]]
        out[k] = v
    return out


def _tables(bra, ket, ib, ik, ls, extra):
    """Per direction {(a, b, c, d): (primitives, nodes)} up to the shells' angular momenta
    plus `extra` on every centre, with the weights in z; and the four factors 2 exponent."""
    z, h = bra.z[ib], ket.z[ik]
    PQ = bra.P[ib] - ket.P[ik]
    rho = z * h / (z + h)
    T = rho * (PQ**2).sum(1)
    x, w = _legendre()
    top = torch.clamp(6.6 / torch.sqrt(torch.clamp(T, min=1e-300)), max=1.0)
    t = top[:, None] * x
    u = t * t
    wt = top[:, None] * w * torch.exp(-T[:, None] * u)
    wt = wt * (2.0 * math.pi**2.5 / (z * h * torch.sqrt(z + h)) * bra.c[ib] * ket.c[ik])[:, None]
    c = lambda v: v[:, None]  # noqa: E731
    b00 = u / c(2.0 * (z + h))
    b10 = (1.0 - u * c(h / (z + h))) / c(2.0 * z)
    b01 = (1.0 - u * c(z / (z + h))) / c(2.0 * h)
    la, lb, lc, ld = (l + extra for l in ls)
    out = []
    for d in range(3):
        c00 = c(bra.P[ib, d] - bra.A[ib, d]) - u * c(h / (z + h) * PQ[:, d])
        d00 = c(ket.P[ik, d] - ket.A[ik, d]) + u * c(z / (z + h) * PQ[:, d])
        g = [[wt if d == 2 else torch.ones_like(u)]]
        for i in range(la + lb):
            g.append([c00 * g[i][0] + (i * b10 * g[i - 1][0] if i else 0.0)])
        for k in range(lc + ld):
            for i in range(la + lb + 1):
                v = d00 * g[i][k]
                if k:
                    v = v + k * b01 * g[i][k - 1]
                if i:
                    v = v + i * b00 * g[i - 1][k]
                g[i].append(v)
        AB, CD = c(bra.A[ib, d] - bra.B[ib, d]), c(ket.A[ik, d] - ket.B[ik, d])
        cols = list(zip(*[_flat(_transfer([r[k] for r in g], la, lb, AB)) for k in range(lc + ld + 1)]))
        I = {}
        for e, col in enumerate(cols):
            K = _transfer(list(col), lc, ld, CD)
            for i in range(lc + 1):
                for j in range(ld + 1):
                    I[(e // (lb + 1), e % (lb + 1), i, j)] = K[i][j]
        out.append(I)
    return out, [c(2.0 * v) for v in (bra.a[ib], bra.b[ib], ket.a[ik], ket.b[ik])]


def _flat(t):
    return [v for row in t for v in row]


def _block(tabs, ls):
    """(primitives, ncomp) of the products of three directions' tables."""
    comps = [_components(l) for l in ls]
    cols = []
    for a in comps[0]:
        for b in comps[1]:
            for c in comps[2]:
                for d in comps[3]:
                    x, y, z = (tabs[k][(a[k], b[k], c[k], d[k])] for k in range(3))
                    cols.append((x * y * z).sum(1))
    return torch.stack(cols, 1)


def _classes(basis):
    """Quartets of shells (as the pairs (s, t), s >= t and pairs in order), by class."""
    sh = basis.shells
    by = {}
    for s in range(len(sh)):
        for t in range(s + 1):
            p = (s, t) if sh[s].l >= sh[t].l else (t, s)
            by.setdefault((sh[p[0]].l, sh[p[1]].l), []).append(p)
    keys = sorted(by)
    for x, kb in enumerate(keys):
        for kk in keys[: x + 1]:
            yield kb, by[kb], kk, by[kk], kb == kk


def _exact_cost(basis, extra):
    c = 0.0
    for (la, lb, lc, ld), (_, npq) in _quartet_counts(basis).items():
        vals = 3.0 * (la + lb + 1 + 2 * extra) * (lc + ld + 1 + 2 * extra) * (lb + ld + 2 + 2 * extra)
        vals += _nc(la) * _nc(lb) * _nc(lc) * _nc(ld) * (1.0, 12.0, 90.0)[extra]
        c += npq * vals * _NODES
    return c


def _dense(basis, order):
    """The dense tensor of derivative order 0, 1 or 2 (slots as the package numbers them)."""
    sh, n, M = basis.shells, basis.nbf(), 3 * basis.natom
    slots = {0: 1, 1: M, 2: M * (M + 1) // 2}[order]
    G = torch.zeros((slots, n, n, n, n), dtype=torch.float64, device="cuda")
    bf = basis.shell2bf()
    for kb, pb, kk, pk, same in _classes(basis):
        ls = kb + kk
        bra, ket = _Pair(sh, pb), _Pair(sh, pk)
        nb, nk = len(bra.a), len(ket.a)
        step = max(1, int(2e8 / (_NODES * nk * math.prod(l + 2 + order for l in ls))))
        ops = _operators(order)
        acc = [torch.zeros((len(pb) * len(pk), math.prod(map(_nc, ls))), dtype=torch.float64, device="cuda")
               for _ in ops]
        for i0 in range(0, nb, step):
            i1 = min(nb, i0 + step)
            ib = torch.arange(i0, i1, device="cuda").repeat_interleave(nk)
            ik = torch.arange(nk, device="cuda").repeat(i1 - i0)
            I, e2 = _tables(bra, ket, ib, ik, ls, order)
            own = bra.own[ib] * len(pk) + ket.own[ik]
            one = {}
            for op, a in zip(ops, acc):
                tabs = []
                for d in range(3):
                    on = tuple(c for c, x in op if x == d)
                    if (d, on) not in one:
                        t = I[d]
                        for c in on:
                            t = _raise(t, c, e2[c])
                        one[(d, on)] = t
                    tabs.append(one[(d, on)])
                a.index_add_(0, own, _block(tabs, ls))
        _scatter(G, basis, bf, pb, pk, same, ls, ops, acc, order)
    return G


def _operators(order):
    """Multisets of (centre, direction) of the order."""
    one = [(c, x) for c in range(4) for x in range(3)]
    if order == 0:
        return [()]
    if order == 1:
        return [(o,) for o in one]
    return [(one[i], one[j]) for i in range(12) for j in range(i, 12)]


def _scatter(G, basis, bf, pb, pk, same, ls, ops, acc, order):
    sh, M = basis.shells, 3 * basis.natom
    nc = [_nc(l) for l in ls]
    sl = lambda s: slice(int(bf[s]), int(bf[s]) + _nc(sh[s].l))  # noqa: E731
    acc = [a.view(len(pb), len(pk), *nc) for a in acc]
    for x, (s, t) in enumerate(pb):
        for y, (u, v) in enumerate(pk):
            if same and y > x:
                continue
            at = [sh[q].atom for q in (s, t, u, v)]
            if order and len(set(at)) == 1:
                continue  # the reference leaves one-centre quartets out of its derivatives
            sums = {}
            for op, a in zip(ops, acc):
                nu = sorted(3 * at[c] + d for c, d in op)
                slot = 0 if not nu else nu[0] if order == 1 else nu[0] * M - nu[0] * (nu[0] - 1) // 2 + nu[1] - nu[0]
                # a mixed derivative is met in both orders of its two centre coordinates
                w = 2.0 if order == 2 and nu[0] == nu[1] and op[0] != op[1] else 1.0
                sums[slot] = sums.get(slot, 0.0) + w * a[x, y]
            for slot, b in sums.items():
                for p, q, r, w, k in ((s, t, u, v, (0, 1, 2, 3)), (t, s, u, v, (1, 0, 2, 3)),
                                      (s, t, v, u, (0, 1, 3, 2)), (t, s, v, u, (1, 0, 3, 2))):
                    e = b.permute(*k)
                    G[slot][sl(p), sl(q), sl(r), sl(w)] = e
                    G[slot][sl(r), sl(w), sl(p), sl(q)] = e.permute(2, 3, 0, 1)


def _one_electron(mol, basis):
    """S, T, V and their first derivatives."""
    sh, n, N = basis.shells, basis.nbf(), basis.natom
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
    out = {"S": z(n, n), "T": z(n, n), "V": z(n, n), "dS": z(3 * N, n, n), "dT": z(3 * N, n, n), "dV": z(3 * N, n, n)}
    bf = basis.shell2bf()
    C = torch.as_tensor(mol.coords, device="cuda")
    Z = torch.as_tensor(np.asarray(mol.Z, dtype=np.float64), device="cuda")
    x, w = _legendre()
    by = {}
    for s in range(len(sh)):
        for t in range(s + 1):
            p = (s, t) if sh[s].l >= sh[t].l else (t, s)
            by.setdefault((sh[p[0]].l, sh[p[1]].l), []).append(p)
    for (la, lb), pairs in by.items():
        B = _Pair(sh, pairs)
        np_, k = len(pairs), _nc(la) * _nc(lb)
        c = lambda v: v[:, None]  # noqa: E731

        def table(c00, b10, first, D):
            g = [first]
            for i in range(la + lb + 4):
                g.append(c00 * g[i] + (i * b10 * g[i - 1] if i else 0.0))
            t = _transfer(g, la + 1, lb + 3, D)
            return {(i, j): t[i][j] for i in range(la + 2) for j in range(lb + 4)}

        def block(t3):
            cols = []
            for a in _components(la):
                for b in _components(lb):
                    v = t3[0][(a[0], b[0])] * t3[1][(a[1], b[1])] * t3[2][(a[2], b[2])]
                    cols.append(v.sum(1))
            return torch.stack(cols, 1)

        def owned(v):
            return z(np_, k).index_add_(0, B.own, v)

        def parts(t3, e2, f):
            """f of the tables, and of their derivatives on A and on B."""
            got = [f(t3)]
            for cen in (0, 1):
                for d in range(3):
                    got.append(f([_raise(t, cen, e2[cen]) if q == d else t for q, t in enumerate(t3)]))
            return got

        e2 = [c(2.0 * B.a), c(2.0 * B.b)]
        norm = c(B.c * (math.pi / B.z) ** 1.5)
        one = torch.ones_like(norm)
        t3 = [table(c(B.P[:, d] - B.A[:, d]), c(0.5 / B.z), norm if d == 2 else one, c(B.A[:, d] - B.B[:, d]))
              for d in range(3)]
        b = c(B.b)

        def kinetic(t3):
            tot = 0.0
            for d in range(3):
                t = t3[d]
                kin = {(i, j): -2.0 * b * b * t[(i, j + 2)] + b * (2 * j + 1) * t[(i, j)]
                       - (0.5 * j * (j - 1) * t[(i, j - 2)] if j > 1 else 0.0) for (i, j) in t if (i, j + 2) in t}
                tot = tot + block([kin if q == d else u for q, u in enumerate(t3)])
            return tot

        res = {"S": [owned(v) for v in parts(t3, e2, block)], "T": [owned(v) for v in parts(t3, e2, kinetic)]}
        nuc = []
        for q in range(N):
            PC = B.P - C[q]
            T = B.z * (PC**2).sum(1)
            top = torch.clamp(6.6 / torch.sqrt(torch.clamp(T, min=1e-300)), max=1.0)
            u = (top[:, None] * x) ** 2
            wt = c(top) * w * torch.exp(-c(T) * u) * c(-Z[q] * 2.0 * math.pi / B.z * B.c)
            v3 = [table(c(B.P[:, d] - B.A[:, d]) - u * c(PC[:, d]), (1.0 - u) * c(0.5 / B.z),
                        wt if d == 2 else torch.ones_like(u), c(B.A[:, d] - B.B[:, d])) for d in range(3)]
            nuc.append([owned(v) for v in parts(v3, e2, block)])
        res["V"] = [sum(nu[i] for nu in nuc) for i in range(7)]
        for p, (s, t) in enumerate(pairs):
            i, j = (slice(int(bf[q]), int(bf[q]) + _nc(sh[q].l)) for q in (s, t))
            sz = (_nc(la), _nc(lb))
            for name, r in res.items():
                out[name][i, j] = r[0][p].view(sz)
                out[name][j, i] = r[0][p].view(sz).T
                slots = {}
                for d in range(3):
                    for cen, q in ((0, s), (1, t)):
                        nu = 3 * sh[q].atom + d
                        slots[nu] = slots.get(nu, 0.0) + r[1 + 3 * cen + d][p]
                    if name == "V":
                        for q in range(N):
                            nu = 3 * q + d
                            slots[nu] = slots.get(nu, 0.0) - nuc[q][1 + d][p] - nuc[q][4 + d][p]
                for nu, v in slots.items():
                    out["d" + name][nu][i, j] = v.view(sz)
                    out["d" + name][nu][j, i] = v.view(sz).T
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rhf", "unique", "jk_pure", "jk_screened"):
        # an iterated result; values in the handle's own list order; functions of another
        # basis; sums that are what the threshold makes them
        return None
    mol, basis, rng = _displaced(case, seed)
    order = {"deriv1": 1, "grad": 1, "deriv2": 2, "hvp": 2}.get(kind, 0)
    if kind == "oei":
        if len(basis.shells) > 60:
            return None
        return _one_electron(mol, basis)
    n, m = basis.nbf(), 3 * basis.natom
    slots = (1, m, m * (m + 1) // 2)[order]
    if _exact_cost(basis, order) > 3.0e11 or slots * n**4 > 1.0e9 or len(basis.shells) > 20:
        return None
    G = _dense(basis, order)
    if kind in ("eri", "deriv1", "deriv2"):
        return G[0] if kind == "eri" else G
    D = _density(n, rng)
    D = torch.as_tensor(D, device="cuda")
    if kind == "jk":
        return torch.einsum("ijkl,kl->ij", G[0], D), torch.einsum("ikjl,kl->ij", G[0], D)
    # sum of (2 D_ij D_kl - D_ik D_jl) times each derivative integral
    E = 2.0 * torch.einsum("xijkl,ij,kl->x", G, D, D) - torch.einsum("xijkl,ik,jl->x", G, D, D)
    if kind == "grad":
        return E
    H = torch.zeros((m, m), dtype=torch.float64, device="cuda")
    i, j = torch.triu_indices(m, m, device="cuda")
    H[i, j] = E
    H[j, i] = E
    return H @ torch.as_tensor(rng.normal(size=m), device="cuda")
