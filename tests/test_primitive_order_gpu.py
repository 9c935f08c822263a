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

from quax_b200.basis import SyntheticSpec, synthetic_molecule
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
