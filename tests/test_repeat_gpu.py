"""Outputs that one thread writes are the same to the bit from call to call, and equal
where symmetry makes them equal."""
import itertools

import numpy as np
import pytest
import torch

from quax_b200.basis import Basis, Shell
from quax_b200.integrals.engine import EriEngine

pytestmark = pytest.mark.gpu


def _basis(ks, ls=(0, 1, 2, 3)):
    """Two centres, shells of ks primitives in turn (f shells at most 3)."""
    rng = np.random.default_rng(17)
    shells = []
    for a, x in enumerate(([0.0, 0.0, 0.0], [0.4, -1.1, 1.9])):
        for l in ls:
            k = ks[(l + a) % len(ks)] if l < 3 else min(3, max(ks))
            e = np.sort(np.exp(rng.uniform(np.log(0.2), np.log(20.0 if l < 3 else 4.0), size=k)))[::-1].copy()
            shells.append(Shell(l, e, rng.uniform(0.2, 1.0, size=k), np.array(x), a))
    return Basis(shells, 2)


@pytest.mark.parametrize("engine", ["default", "rys"])
@pytest.mark.parametrize("ks", [(5,), (1, 8)])
def test_integrals(ks, engine):
    """Dense and unique integrals, with 1 to 4,096 primitives per quartet: one and several
    parts per quartet.  (Of the default engines, those that sum a quartet's primitives
    with atomics, for the large classes up to d, repeat to rounding only.)"""
    eng = EriEngine(_basis(ks), 1e-12)
    if engine == "rys":
        for c in eng.class_info():
            eng.set_engine(c["cls"], plain="rys")
    G = eng.eri()
    blocks = {cls: b.clone() for cls, (_, b) in eng.unique_blocks().items()}
    exact = {c["cls"] for c in eng.class_info() if engine == "rys" or max(c["l"]) == 3}
    for _ in range(3):
        for cls, (_, b) in eng.unique_blocks().items():
            assert cls not in exact or torch.equal(b, blocks[cls]), cls
        assert engine != "rys" or torch.equal(eng.eri(), G)
    # images of one integral; a quartet with two equal shells or pairs holds some of its
    # images as components of their own, each with its own rounding
    b = eng.basis
    sh = torch.cat([torch.full(((s.l + 1) * (s.l + 2) // 2,), i) for i, s in enumerate(b.shells)]).cuda()
    i, j, k, l = (sh.view([-1 if a == x else 1 for a in range(4)]) for x in range(4))
    own = (i == j) | (k == l) | ((torch.minimum(i, j) == torch.minimum(k, l)) & (torch.maximum(i, j) == torch.maximum(k, l)))
    for p in itertools.permutations(range(4)):
        if {p[0], p[1]} in ({0, 1}, {2, 3}):
            assert bool(((G.permute(p) == G) | own).all()), p
