"""Outputs that one thread writes are the same to the bit from call to call, and equal
where symmetry makes them equal."""
import itertools

import numpy as np
import pytest
import torch

from quax_b200.basis import Basis, Shell
from quax_b200.integrals.engine import EriEngine
from quax_b200.oei import one_electron

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
    _images(eng.basis, G)


def _images(b, G):
    """The images of one integral are equal; a quartet with two equal shells or pairs holds
    some of its images as components of their own, each with its own rounding."""
    sh = torch.cat([torch.full(((s.l + 1) * (s.l + 2) // 2,), i) for i, s in enumerate(b.shells)]).cuda()
    i, j, k, l = (sh.view([-1 if a == x else 1 for a in range(4)]) for x in range(4))
    own = (i == j) | (k == l) | ((torch.minimum(i, j) == torch.minimum(k, l)) & (torch.maximum(i, j) == torch.maximum(k, l)))
    for p in itertools.permutations(range(4)):
        if {p[0], p[1]} in ({0, 1}, {2, 3}):
            assert bool(((G.permute(p) == G) | own).all()), p


@pytest.mark.parametrize("ks,ls", [((5,), (0, 1, 2, 3)), ((1, 8), (0, 1, 3)), ((2,), (0, 3))])
def test_first_derivatives(ks, ls):
    """First-derivative tensors of the Rys engine, a quartet's primitives in one and in
    several parts: the tensor, its slices, and both after the parts' buffer was given back
    and after it was planned anew for more classes."""
    eng = EriEngine(_basis(ks, ls), 1e-12)
    first = eng.eri_deriv_core(1).clone()  # f classes by the Rys engine
    for c in eng.class_info():
        eng.set_engine(c["cls"], deriv="rys")
    dG = eng.eri_deriv_core(1).clone()
    scale = dG.abs().max()
    assert (first - dG).abs().max() < 1e-9 * max(1.0, scale.item())
    for x in range(dG.shape[0]):
        _images(eng.basis, dG[x])
    for _ in range(2):
        assert torch.equal(eng.eri_deriv_core(1), dG)
        eng.release_scratch()
    nu = np.zeros(dG.shape[0], dtype=int)
    for x in (0, 4):
        nu[:] = 0
        nu[x] = 1
        assert torch.equal(eng.eri_deriv(nu), dG[x])


def test_first_derivatives_under_capture():
    """A captured tensor: before the parts' buffer exists (one team per quartet), and with it."""
    eng = EriEngine(_basis((3,), (0, 3)), 1e-12)
    for c in eng.class_info():
        eng.set_engine(c["cls"], deriv="rys")
    out = torch.empty((3 * eng.natom,) + (eng.nbf,) * 4, dtype=torch.float64, device="cuda")

    def captured():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            eng.eri_deriv_core(1, out)
        out.fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        return out.clone()

    alone = captured()
    dG = eng.eri_deriv_core(1).clone()
    assert (alone - dG).abs().max() < 1e-12 * max(1.0, dG.abs().max().item())
    assert torch.equal(captured(), dG)


# atoms, how many of them carry shells: nuclei in 2, 4, 16 and 32 slices (one to eight
# blocks per shell pair), some of them empty, and in one slice
@pytest.mark.parametrize("natom,carry,ls", [(2, 2, (0, 1, 2)), (3, 3, (0, 1, 2)), (12, 4, (0, 1)), (24, 3, (0, 1, 2)),
                                            (10, 10, (0,) * 5)])
def test_attraction(natom, carry, ls):
    """V and dV: every image and every call to the bit (each pair's sums over the nuclei
    meet in order), and right."""
    rng = np.random.default_rng(natom)
    xyz = 1.7 * np.array(list(np.ndindex(3, 3, 3)))[rng.permutation(27)[:natom]] + rng.uniform(-0.2, 0.2, (natom, 3))
    k = 2 if natom < 10 else 1
    shells = [Shell(l, rng.uniform(0.2, 20.0, size=k), rng.uniform(0.2, 1.0, size=k), xyz[a], a)
              for a in range(carry) for l in ls]
    b = Basis(shells, natom)
    Z = rng.integers(1, 9, size=natom).astype(float)
    eng = EriEngine(b, 1e-12)
    eng.set_charges(Z)
    V, dV = eng.oei()[2].clone(), eng.oei_deriv(1)[2].clone()
    assert torch.equal(V, V.T) and torch.equal(dV, dV.transpose(1, 2))
    for _ in range(5):
        assert torch.equal(eng.oei()[2], V) and torch.equal(eng.oei_deriv(1)[2], dV)
    ref = one_electron(b, Z, b.atom_coords(), deriv=True)
    assert np.abs(V.cpu().numpy() - ref[2]).max() < 1e-12 * max(1.0, np.abs(ref[2]).max())
    assert np.abs(dV.cpu().numpy() - ref[5]).max() < 1e-11 * max(1.0, np.abs(ref[5]).max())
