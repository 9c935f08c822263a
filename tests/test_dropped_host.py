"""Primitive pairs left out at set-up (build_pairs in qx_setup.cu), on the CPU: what the
rule drops, with up to four nuclear derivatives, lies below the rounding of any integral
that passes the Schwarz threshold.

The rule drops a primitive pair whose bound, raised by a factor for four derivatives, is
below 1e-18 of the threshold.  The oracle evaluates the dropped pair alone against a
Gaussian charge at its own place: the value and every derivative has to stay below the
cut, two decades under the rounding of an integral as large as the threshold."""
import ctypes as C
import os
import shutil
import subprocess
from itertools import combinations_with_replacement

import numpy as np
import pytest

from quax_b200.basis import Basis, Shell

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
_dp, _ip = C.POINTER(C.c_double), C.POINTER(C.c_int)


@pytest.fixture(scope="module")
def setup_lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("setup_host") / "libsetup_host.so")
    csrc = os.path.join(ROOT, "quax_b200", "csrc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC", "-I" + csrc, "-I" + os.path.join(ROOT, "include"), os.path.join(csrc, "qx_setup.cu"),
                        os.path.join(HERE, "setup_host", "setup_host.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lib = C.CDLL(out)
    lib.kept_pairs.argtypes = [_dp, _ip, _ip, _dp, _dp, C.c_double, _dp]
    return lib


@pytest.mark.parametrize("tol", [1e-12, 1e-6])
@pytest.mark.parametrize("l0,l1", [(0, 0), (1, 0), (1, 1), (2, 0), (1, 2), (2, 2), (3, 0), (1, 3), (3, 2), (3, 3)])
def test_dropped_bound(oracle_lib, setup_lib, l0, l1, tol):
    rng = np.random.default_rng(100 * l0 + l1)
    cut, seen, worst = 1e-18 * min(tol, 1e-10), 0, 0.0
    for R in (1.0, 2.0, 4.0, 8.0):
        xyz = np.array([[0.1, -0.2, 0.3], [0.1, -0.2, 0.3]])
        xyz[1] += R * np.array([0.48, 0.64, 0.6])
        exps = [np.exp(rng.uniform(np.log(0.08), np.log(5e3), size=6)) for _ in range(2)]
        coef = [rng.uniform(0.2, 1.0, size=6) for _ in range(2)]
        shells = [Shell(l, e, c, x, a) for a, (l, e, c, x) in enumerate(zip((l0, l1), exps, coef, xyz))]
        ob = oracle_lib.OracleBasis(Basis(shells, 2))
        fl = Basis(shells, 2).flat()
        out = np.zeros(72)
        p = lambda a, t=_dp: a.ctypes.data_as(t)  # noqa: E731
        n = setup_lib.kept_pairs(p(np.ascontiguousarray(xyz)), p(fl["l"], _ip), p(fl["nprim"], _ip), p(fl["exps"]),
                                 p(fl["coefs"]), tol, p(out))
        kept = out[: 2 * n].reshape(-1, 2)
        ca, cb = ob.coef[:6], ob.coef[6:]  # coefficients of the normalised contractions
        dropped = [(i, j) for i in range(6) for j in range(6)
                   if not np.any(np.all(np.abs(kept / (exps[0][i], exps[1][j]) - 1.0) < 1e-9, axis=1))]
        assert n + len(dropped) == 36
        rng.shuffle(dropped)
        # the largest of those left out are the ones next to the cut
        mu = [exps[0][i] * exps[1][j] / (exps[0][i] + exps[1][j]) for i, j in dropped]
        for i, j in [dropped[k] for k in np.argsort(mu)[:3]]:
            a, b = exps[0][i], exps[1][j]
            at = (a * xyz[0] + b * xyz[1]) / (a + b)
            one = Basis([Shell(l0, np.array([a]), np.ones(1), xyz[0], 0), Shell(l1, np.array([b]), np.ones(1), xyz[1], 1),
                         Shell(0, np.array([1.0]), np.ones(1), at, 2)], 3)
            o = oracle_lib.OracleBasis(one)
            w = abs(ca[i] * cb[j] / (o.coef[0] * o.coef[1]))
            q = max(1e-300, oracle_lib.shell_quartet(o, 2, 2, 2, 2).max()) ** 0.5
            for k in range(5 if l0 + l1 <= 3 else 3):
                if k == 0:
                    v = np.abs(oracle_lib.shell_quartet(o, 0, 1, 2, 2)).max()
                else:
                    rows = [r for r, t in enumerate(combinations_with_replacement(range(12), k)) if max(t) < 6]
                    v = np.abs(oracle_lib.shell_quartet_derivk(o, 0, 1, 2, 2, k)[rows]).max()
                worst = max(worst, w * v / q / cut)
                seen += 1
    assert seen and worst < 1.0
