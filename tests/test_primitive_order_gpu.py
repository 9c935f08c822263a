"""Negligible primitive pairs are left out and quartets are processed by decreasing
work: neither may show in what a call returns.

Integrals against the oracle, which sums every primitive: 1e-12 absolute (the ERI bar of
the other tests) for Schwarz thresholds that drop many, few and no primitives of two
separated atoms with exponents up to 5e3; and the screened quartets are the oracle's.
The unique layout is the list's, whatever the processing order: the blocks of a shard,
and of a handle whose precision split was set and taken back, equal the full handle's
blocks of the same shells to 1e-13 of the block's scale (split-mode sums meet in another
order)."""
import numpy as np
import pytest
import torch

from quax_b200.basis import Basis, Shell, SyntheticSpec, synthetic_molecule
from quax_b200.integrals.engine import EriEngine

pytestmark = pytest.mark.gpu


def _mol(seed, natom=2, **kw):
    kw = dict(dict(box=9.0, min_sep=5.0, kmax=6, exp_lo=0.08, exp_hi=5e3, heavy_ls=(0, 1, 2)), **kw)
    return synthetic_molecule(SyntheticSpec(natom=natom, **kw), seed)[1]


@pytest.mark.parametrize("tol", [1e-6, 1e-12, 1e-30])
def test_dropped_primitives(oracle_lib, tol):
    b = _mol(1)
    eng = EriEngine(b, tol)
    ob = oracle_lib.OracleBasis(b)
    assert eng.unique_quartets() == oracle_lib.count_unique(ob, tol)
    full = sum(a.nprim * c.nprim for i, a in enumerate(b.shells) for c in b.shells[: i + 1]) ** 2
    used = sum(c["prims"] for c in eng.class_info())
    assert used < full
    G = eng.eri().cpu().numpy()
    assert np.abs(G - oracle_lib.compute_2e_int(ob, tol)).max() < 1e-12


def test_dropped_primitives_second_derivatives():
    """Hessian-vector products of s and p shells, whose programs cancel sums of (2 alpha)^2
    weights, do not depend on the primitives a threshold drops.  Shells with a diffuse and
    tight primitives on close atoms, so that both thresholds keep every quartet: the same
    sums in the same order but for the atomics, 1e-12 of the largest entry (grouping them
    otherwise moved five atoms' product by 2.8e-9)."""
    xyz = np.array([[0.0, 0.0, 0.0], [0.0, 1.1, 2.6], [2.4, 0.4, -1.3]])
    exps, coef = np.array([3000.0, 400.0, 60.0, 9.0, 0.3]), np.array([0.1, 0.2, 0.4, 0.6, 1.0])
    b = Basis([Shell(l, exps, coef, x.copy(), a) for a, x in enumerate(xyz) for l in (0, 0, 1)], 3)
    n = b.nbf()
    rng = np.random.default_rng(3)
    C = rng.normal(0.0, 1.0 / np.sqrt(n), size=(n, max(1, n // 4)))
    D, v = torch.from_numpy(C @ C.T).cuda(), torch.from_numpy(rng.normal(size=3 * b.natom)).cuda()
    e = [EriEngine(b, tol) for tol in (1e-12, 1e-60)]
    assert e[0].unique_quartets() == e[1].unique_quartets()
    assert sum(c["prims"] for c in e[0].class_info()) < sum(c["prims"] for c in e[1].class_info())
    h = [x.grad_adjoint_jvp(D, v, 2.0, -1.0).cpu().numpy() for x in e]
    assert np.abs(h[0] - h[1]).max() < 1e-12 * np.abs(h[1]).max()


def test_layout_of_views():
    b = _mol(2, natom=4, min_sep=1.8, kmax=4)
    eng = EriEngine(b, 1e-12)

    def blocks(e):
        return {(c, tuple(s)): v for c, (sh, blk) in e.unique_blocks().items()
                for s, v in zip(sh.tolist(), blk.cpu().numpy())}

    ref = blocks(eng)
    seen = 0
    for r in range(3):
        eng.set_shard(r, 3)
        got = blocks(eng)
        seen += len(got)
        for k, v in got.items():
            assert np.abs(v - ref[k]).max() <= 1e-13 * max(1.0, np.abs(ref[k]).max()), k
    assert seen == len(ref)
    eng.set_shard(0, 1)
    eng.set_precision(1e-6)
    eng.set_precision(0.0)
    got = blocks(eng)
    assert sorted(got) == sorted(ref)
    for k, v in got.items():
        assert np.abs(v - ref[k]).max() <= 1e-13 * max(1.0, np.abs(ref[k]).max()), k


def test_order_without_room():
    """A device with room for the quartet lists but not for their processing order: the
    handle works, in list order."""
    rng = np.random.default_rng(31)
    xyz = 1.6 * np.array(list(np.ndindex(5, 5, 5)))[:110] + rng.uniform(-0.2, 0.2, (110, 3))
    shells = [Shell(0, rng.uniform(0.08, 0.4, size=1 + a % 3), np.ones(1 + a % 3), xyz[a], a) for a in range(110)]
    b = Basis(shells, 110)

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    D = torch.eye(110, dtype=torch.float64, device="cuda")
    warm = EriEngine(b, 1e-12)  # what the first calls of a process allocate
    warm.jk(D)
    warm.close()
    f0 = free()
    ref = EriEngine(b, 1e-12)
    used = f0 - free()
    nq = ref.unique_quartets()
    assert used > 12 * nq > 100 << 20  # lists of 8 bytes and orders of 4 per quartet
    J, K = ref.jk(D)
    ref.close()
    fill = torch.empty(free() - used + 2 * nq, dtype=torch.uint8, device="cuda")
    eng = EriEngine(b, 1e-12)
    J2, K2 = eng.jk(D)
    eng.set_precision(1e-9)  # lists rebuilt, with no more room than before
    eng.set_precision(0.0)
    J3, K3 = eng.jk(D)
    del fill
    for x, y in ((J, J2), (K, K2), (J, J3), (K, K3)):
        assert (x - y).abs().max().item() < 1e-11 * J.abs().max().item()
