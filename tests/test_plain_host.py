"""The plain integrals' arithmetic on the CPU (no GPU needed).

tests/plain_host/plain_host.cu runs the phases of qx_plain.cuh for a shell quartet, one
thread of the block after another: against the oracle (1e-11 of max(1, largest value), the
oracle's own rounding being about 1e-13 on (ff|ff)), with the primitives in one part and in
three; and for accuracy, error against an 80-bit evaluation next to the error of the table
engine's phases (qx_rys.cuh).  Both transfer each 1-D factor, so their roundings are of
one kind and number; over 24 quartets the medians may differ by half, and the worst, a
heavy tail, fourfold.  A transfer after the contraction misses both: (ff|ff) 3.6 times
(median) and 65 times (worst) beyond the table engine."""
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
NCLS = 13


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("plain_host") / "libplain_host.so")
    cmd = [nvcc, "-x", "cu", "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-shared",
           "-Xcompiler", "-fPIC", "-DTILE_HOST", "-I" + os.path.join(ROOT, "quax_b200", "csrc"),
           "-I" + os.path.join(ROOT, "include"), os.path.join(HERE, "plain_host", "plain_host.cu"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    lib = C.CDLL(out)
    lib.plain_host.argtypes = [C.c_int, C.c_int, _ip, _dp, _ip, _dp, _dp, C.c_int, _dp]
    return lib


def _class(lib, cls):
    l4 = np.zeros(4, dtype=np.int32)
    assert lib.plain_host(cls, 0, l4.ctypes.data_as(_ip), None, None, None, None, 1, None) == 0
    return [int(l) for l in l4]


def _shells(rng, l4, kmax, spread, emax):
    out = []
    for c, l in enumerate(l4):
        k = int(rng.integers(1, kmax + 1))
        e = np.sort(np.exp(rng.uniform(np.log(0.1), np.log(emax), size=k)))[::-1].copy()
        out.append(Shell(l, e, rng.uniform(0.1, 1.0, size=k), rng.uniform(0.0, spread, size=3), c))
    return out


def _run(lib, cls, what, shells, w, parts=1):
    out = np.zeros(int(np.prod([(s.l + 1) * (s.l + 2) // 2 for s in shells])))
    arr = (np.ascontiguousarray(np.concatenate([s.center for s in shells])),
           np.array([s.nprim for s in shells], dtype=np.int32),
           np.ascontiguousarray(np.concatenate([s.exps for s in shells])), np.ascontiguousarray(w))
    p = [a.ctypes.data_as(t) for a, t in zip(arr, (_dp, _ip, _dp, _dp))]
    l4 = np.zeros(4, dtype=np.int32)
    assert lib.plain_host(cls, what, l4.ctypes.data_as(_ip), *p, parts, out.ctypes.data_as(_dp)) == 0
    return out


@pytest.mark.parametrize("parts", [1, 3])
@pytest.mark.parametrize("cls", range(NCLS))
def test_plain_phases_against_oracle(host_lib, oracle_lib, cls, parts):
    l4 = _class(host_lib, cls)
    shells = _shells(np.random.default_rng(500 + cls), l4, 3 if sum(l4) < 10 else 2, 3.0, 20.0)
    ob = oracle_lib.OracleBasis(Basis(shells, 4, False))
    ref = oracle_lib.shell_quartet(ob, 0, 1, 2, 3).reshape(-1)
    v = _run(host_lib, cls, 0, shells, ob.coef, parts)
    assert np.abs(v - ref).max() < 1e-11 * max(1.0, np.abs(ref).max()), l4


@pytest.mark.parametrize("cls", [3, 8, 9, 10, 11, 12])
def test_plain_accuracy(host_lib, oracle_lib, cls):
    l4 = _class(host_lib, cls)
    rng = np.random.default_rng(900 + cls)
    err = {0: [], 1: []}
    for q in range(24):
        shells = _shells(rng, l4, 1, (1.0, 3.0, 6.0)[q % 3], (5.0, 20.0, 50.0)[q // 3 % 3])
        w = oracle_lib.OracleBasis(Basis(shells, 4, False)).coef
        ref = _run(host_lib, cls, 2, shells, w)
        for k in err:
            err[k].append(np.abs(_run(host_lib, cls, k, shells, w) - ref).max() / np.abs(ref).max())
    plain, table = np.array(err[0]), np.array(err[1])
    assert np.median(plain) < 1.5 * np.median(table), (l4, np.median(plain), np.median(table))
    assert plain.max() < 4.0 * table.max(), (l4, plain.max(), table.max())
