"""The tile kernels where a quartet's primitives are split over blocks, and the
straight-line J/K kernels with every lane count, against the oracle.  Tolerances as in the
Rys and J/K tests: ERI 1e-12 absolute, J/K 1e-10, gradients 1e-9 of max(1, |g|)."""
import numpy as np
import pytest
import torch

from quax_b200.basis import Basis, Shell, SyntheticSpec, synthetic_molecule
from quax_b200.integrals.engine import EriEngine

pytestmark = pytest.mark.gpu


def _density(n, seed):
    rng = np.random.default_rng(seed)
    C = rng.normal(0.0, 1.0 / np.sqrt(n), size=(n, max(1, n // 4)))
    return C @ C.T


@pytest.mark.parametrize("ks", [(1,), (5,), (1, 8)])
def test_split_primitives(oracle_lib, ks):
    """Two centres with s, p, d and f shells of equal (no processing order) and of very
    unequal primitive counts, 1 to 4,096 per quartet: every output that parts of a quartet
    meet in (dense, unique, J/K, gradient)."""
    rng = np.random.default_rng(7)
    shells = []
    for a, x in enumerate(([0.0, 0.0, 0.0], [0.4, -1.1, 1.9])):
        for l in (0, 1, 2, 3):
            k = ks[(l + a) % len(ks)] if l < 3 else min(3, ks[0])
            e = np.sort(np.exp(rng.uniform(np.log(0.2), np.log(20.0 if l < 3 else 4.0), size=k)))[::-1].copy()
            shells.append(Shell(l, e, rng.uniform(0.2, 1.0, size=k), np.array(x), a))
    b = Basis(shells, 2)
    ob = oracle_lib.OracleBasis(b)
    eng = EriEngine(b, 1e-12)
    for c in eng.class_info():
        eng.set_engine(c["cls"], plain="rys", deriv="rys")
    G = oracle_lib.compute_2e_int(ob, 1e-12)
    assert np.abs(eng.eri().cpu().numpy() - G).max() < 1e-12
    D = _density(eng.nbf, 1)
    Dg = torch.from_numpy(D).cuda()
    J, K = (x.cpu().numpy() for x in eng.jk(Dg))
    assert np.abs(J - np.einsum("ijkl,kl->ij", G, D)).max() < 1e-10
    assert np.abs(K - np.einsum("ikjl,kl->ij", G, D)).max() < 1e-10
    for cls, (sh, blk) in eng.unique_blocks().items():
        for s, v in zip(sh[:3], blk[:3].cpu().numpy()):
            assert np.abs(v - oracle_lib.shell_quartet(ob, *map(int, s)).reshape(-1)).max() < 1e-12, cls
    g = eng.grad_adjoint(Dg, 2.0, -1.0).cpu().numpy()
    gr = oracle_lib.grad_contract(ob, 1e-12, D, 2.0, -1.0)
    assert np.abs(g - gr).max() < 1e-9 * max(1.0, np.abs(gr).max())


@pytest.mark.parametrize("ks", [(8,), (1, 8), (1, 3, 8)])
def test_straight_line_segments(oracle_lib, ks):
    """The default lanes per quartet, by its primitives: 1 to 4,096 per quartet, equal
    counts (one segment, no processing order) and mixed ones, in every output mode."""
    rng = np.random.default_rng(11)
    shells = []
    for a, x in enumerate(([0.0, 0.0, 0.0], [0.4, -1.1, 1.9], [1.7, 1.2, -0.6])):
        for i, l in enumerate((0, 0, 1, 2) if a else (0, 1, 1)):
            k = ks[(i + a) % len(ks)]
            e = np.sort(np.exp(rng.uniform(np.log(0.2), np.log(20.0), size=k)))[::-1].copy()
            shells.append(Shell(l, e, rng.uniform(0.2, 1.0, size=k), np.array(x), a))
    b = Basis(shells, 3)
    ob = oracle_lib.OracleBasis(b)
    eng = EriEngine(b, 1e-12)
    assert sum(v[0] == "sl" for v in eng.engine_config().values()) >= 8
    G = oracle_lib.compute_2e_int(ob, 1e-12)
    assert np.abs(eng.eri().cpu().numpy() - G).max() < 1e-12
    D = _density(eng.nbf, 4)
    J, K = (x.cpu().numpy() for x in eng.jk(torch.from_numpy(D).cuda()))
    assert np.abs(J - np.einsum("ijkl,kl->ij", G, D)).max() < 1e-10
    assert np.abs(K - np.einsum("ikjl,kl->ij", G, D)).max() < 1e-10
    for cls, (sh, blk) in eng.unique_blocks().items():
        for s, v in zip(sh[:40], blk[:40].cpu().numpy()):
            assert np.abs(v - oracle_lib.shell_quartet(ob, *map(int, s)).reshape(-1)).max() < 1e-12, cls


@pytest.mark.parametrize("lg", [0, 2, 5])
def test_straight_line_jk(oracle_lib, lg):
    """J/K of every class with a straight-line kernel, 2^lg lanes per quartet: accumulators
    in registers and in shared memory, full and screened builds."""
    b = synthetic_molecule(SyntheticSpec(natom=4, box=5.0, min_sep=1.2, kmax=2, exp_lo=0.1, exp_hi=50.0,
                                         heavy_ls=(0, 0, 1, 1, 2), h_ls=(0, 0, 1)), 5)[1]
    eng = EriEngine(b, 1e-12)
    for c in eng.class_info():
        if "%d%d%d%d" % c["l"] not in ("2121", "2211", "2221", "2222") and max(c["l"]) <= 2:
            eng.set_engine(c["cls"], plain="sl", plain_param=lg)
    G = oracle_lib.compute_2e_int(oracle_lib.OracleBasis(b), 1e-12)
    D = _density(eng.nbf, 2)
    for kw in ({}, {"screen": 1e-14}):
        J, K = (x.cpu().numpy() for x in eng.jk(torch.from_numpy(D).cuda(), **kw))
        assert np.abs(J - np.einsum("ijkl,kl->ij", G, D)).max() < 1e-10
        assert np.abs(K - np.einsum("ikjl,kl->ij", G, D)).max() < 1e-10


@pytest.mark.parametrize("engine", ["default", "rys"])
def test_long_contractions(oracle_lib, engine):
    """Shells of 1, 9 and 12 primitives: quartets of up to 20,736, past the counts that
    have an order key of their own, in every output that their parts meet in."""
    rng = np.random.default_rng(23)
    shells = []
    for a, x in enumerate(([0.0, 0.0, 0.0], [0.4, -1.1, 1.9])):
        for l, k in ((0, 12), (1, 9), (1, 12), (2, 1)) if a else ((0, 1), (0, 12), (1, 12)):
            e = np.sort(np.exp(rng.uniform(np.log(0.2), np.log(20.0), size=k)))[::-1].copy()
            shells.append(Shell(l, e, rng.uniform(0.2, 1.0, size=k), np.array(x), a))
    b = Basis(shells, 2)
    ob = oracle_lib.OracleBasis(b)
    eng = EriEngine(b, 1e-12)
    if engine == "rys":
        for c in eng.class_info():
            eng.set_engine(c["cls"], plain="rys", deriv="rys")
    G = oracle_lib.compute_2e_int(ob, 1e-12)
    assert np.abs(eng.eri().cpu().numpy() - G).max() < 1e-12
    D = _density(eng.nbf, 6)
    Dg = torch.from_numpy(D).cuda()
    J, K = (x.cpu().numpy() for x in eng.jk(Dg))
    assert np.abs(J - np.einsum("ijkl,kl->ij", G, D)).max() < 1e-10
    assert np.abs(K - np.einsum("ikjl,kl->ij", G, D)).max() < 1e-10
    g = eng.grad_adjoint(Dg, 2.0, -1.0).cpu().numpy()
    gr = oracle_lib.grad_contract(ob, 1e-12, D, 2.0, -1.0)
    assert np.abs(g - gr).max() < 1e-9 * max(1.0, np.abs(gr).max())


def test_engine_config_round_trip():
    """What engine_config reports, given back to set_engine, changes nothing: the lanes a
    straight-line kernel chooses itself, and tensors on another engine than the gradient."""
    b = synthetic_molecule(SyntheticSpec(natom=3, box=5.0, min_sep=1.2, kmax=3, exp_lo=0.1, exp_hi=50.0, f_shell=True,
                                         f_kmax=1), 5)[1]
    eng = EriEngine(b, 1e-12)
    classes = {"%d%d%d%d" % c["l"]: c["cls"] for c in eng.class_info() if c["nq"]}
    names = EriEngine.ENGINE_NAMES

    def apply(cfg):
        for k, (plain, p, deriv, d) in cfg.items():
            eng.set_engine(classes[k], plain=plain, plain_param=p, deriv=deriv, deriv_param=d)

    default = eng.engine_config()
    assert all(v[1] == -1 for v in default.values() if v[0] == "sl")
    # the tiles' gradient from L = 4 on; tensors of the classes up to d stay on their engine
    for k, v in default.items():
        if v[2] == "rys":
            assert (v[3] in (0, 1)) == ("3" in k)
            assert "3" in k or names[v[3] // 8] in ("warp", "coop", "wvrr", "dsplit")
    apply(default)
    assert eng.engine_config() == default
    for lg in (0, 5):  # fixed lanes, and tensors and gradient on one engine
        apply({k: (v[0], lg if v[0] == "sl" else v[1], "rys", 0) for k, v in default.items()})
        fixed = eng.engine_config()
        assert all(v[2:] == ("rys", 0) and (v[0] != "sl" or v[1] == lg) for v in fixed.values())
        apply(fixed)
        assert eng.engine_config() == fixed
    apply(default)
    assert eng.engine_config() == default
    eng.autotune()
    tuned = eng.engine_config()
    apply(tuned)
    assert eng.engine_config() == tuned
    for plain_param, deriv_param in ((-2, 0), (6, 0), (-1, 2), (-1, 48), (-1, 8 + 2)):
        with pytest.raises(NotImplementedError):
            eng.set_engine(classes["1010"], plain="sl", plain_param=plain_param, deriv="rys", deriv_param=deriv_param)
