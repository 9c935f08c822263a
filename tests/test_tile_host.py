"""The tile engine's arithmetic and index tables on the CPU (no GPU needed).

tests/tile_host/tile_host.cu runs the phases of qx_tile.cuh for a shell quartet, one
thread of the block after another, for classes that cover one and several chunks of e
values, one and several primitives side by side, and empty transfers; the primitives in
one part and in three.  Against the oracle: the plain block (1e-11) and the nine gradient
sums of Gamma = D_ij D_kl - D_ik D_jl / 2 summed over images (1e-10), each relative to
max(1, largest value) -- the bounds of the Rys phases' test, from the oracle's own
rounding (~1e-13 on (ff|ff) quartets).
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from quax_b200.basis import Basis, Shell

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
_dp, _ip = C.POINTER(C.c_double), C.POINTER(C.c_int)
NCLS = 14


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("tile_host") / "libtile_host.so")
    cmd = [nvcc, "-x", "cu", "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-shared",
           "-Xcompiler", "-fPIC", "-DTILE_HOST", "-I" + os.path.join(ROOT, "quax_b200", "csrc"),
           "-I" + os.path.join(ROOT, "include"), os.path.join(HERE, "tile_host", "tile_host.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lib = C.CDLL(out)
    lib.tile_host.argtypes = [C.c_int, C.c_int, _ip, _dp, _ip, _dp, _dp, _dp, C.c_int, _dp]
    return lib


def _ncart(l):
    return (l + 1) * (l + 2) // 2


def _gamma(D, off, nc):
    """Gamma of the quartet's components, summed over the eight images (four shells)."""
    A, B, Cc, Dd = (slice(o, o + k) for o, k in zip(off, nc))
    j = 8.0 * np.einsum("ab,cd->abcd", D[A, B], D[Cc, Dd])
    k = 4.0 * (np.einsum("ac,bd->abcd", D[A, Cc], D[B, Dd]) + np.einsum("ad,bc->abcd", D[A, Dd], D[B, Cc]))
    return (j - 0.5 * k).reshape(-1)


@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("cls", range(NCLS))
def test_tile_phases_against_oracle(host_lib, oracle_lib, cls, parts):
    l4 = np.zeros(4, dtype=np.int32)
    lp = l4.ctypes.data_as(_ip)
    assert host_lib.tile_host(cls, 0, lp, None, None, None, None, None, 1, None) == 0
    rng = np.random.default_rng(300 + cls)
    kmax = 3 if l4.sum() < 10 else 2
    shells = []
    for c in range(4):
        k = int(rng.integers(1, kmax + 1))
        e = np.sort(np.exp(rng.uniform(np.log(0.1), np.log(20.0), size=k)))[::-1].copy()
        shells.append(Shell(int(l4[c]), e, rng.uniform(0.1, 1.0, size=k), rng.uniform(0.0, 3.0, size=3), c))
    ob = oracle_lib.OracleBasis(Basis(shells, 4, False))
    nc = [_ncart(int(l)) for l in l4]
    off = np.concatenate([[0], np.cumsum(nc)])
    n = int(off[-1])
    cen = np.ascontiguousarray(np.concatenate([s.center for s in shells]))
    npr = np.array([s.nprim for s in shells], dtype=np.int32)
    ex = np.ascontiguousarray(np.concatenate([s.exps for s in shells]))
    w = np.ascontiguousarray(ob.coef.copy())
    D = rng.normal(size=(n, n))
    D = np.ascontiguousarray(D + D.T)
    ncomp = int(np.prod(nc))

    def run(kind):
        out = np.zeros(ncomp if kind == 0 else 9)
        args = [x.ctypes.data_as(t) for x, t in ((cen, _dp), (npr, _ip), (ex, _dp), (w, _dp), (D, _dp))]
        assert host_lib.tile_host(cls, kind, lp, *args, parts, out.ctypes.data_as(_dp)) == 0
        return out

    ref = oracle_lib.shell_quartet(ob, 0, 1, 2, 3).reshape(-1)
    assert np.abs(run(0) - ref).max() < 1e-11 * max(1.0, np.abs(ref).max()), tuple(l4)
    gam = _gamma(D, off, nc)
    ref1 = oracle_lib.shell_quartet(ob, 0, 1, 2, 3, deriv=True).reshape(12, -1)
    terms = ref1[:9] * gam
    g = run(1)
    assert np.abs(g - terms.sum(1)).max() < 1e-10 * max(1.0, np.abs(terms).max()), tuple(l4)
