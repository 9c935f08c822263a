"""Launch segments of a class's quartets (qx_segments.h), on the CPU: whatever the counts,
the segments hold every quartet once, in order, and no lane or block is left more
primitives than its share -- for classes of more than 2^31 quartets too."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
_lp, _ip = C.POINTER(C.c_longlong), C.POINTER(C.c_int)


@pytest.fixture(scope="module")
def seg(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is not available")
    out = str(tmp_path_factory.mktemp("segments") / "libseg.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "quax_b200", "csrc"),
                    os.path.join(HERE, "segments_host", "segments_host.cpp"), "-o", out], check=True)
    lib = C.CDLL(out)
    lib.seg_key_of.argtypes = [C.c_longlong]
    lib.seg_prefix_of.argtypes = [_lp, C.c_int, _lp]
    lib.sl_segs.argtypes = [C.c_longlong, C.c_longlong, C.c_longlong, _lp, C.c_int, _lp, _ip]
    lib.tile_segs.argtypes = [C.c_longlong, C.c_longlong, C.c_longlong, _lp, C.c_int, _lp, _lp, _lp]
    return lib


def _prefix(seg, counts):
    """counts: {primitives per quartet: quartets}."""
    nkey = max(seg.seg_key_of(n) for n in counts) + 1
    hist = np.zeros(nkey, dtype=np.int64)
    for n, q in counts.items():
        hist[seg.seg_key_of(n)] += q
    prefix = np.zeros(seg.seg_pow(), dtype=np.int64)
    seg.seg_prefix_of(hist.ctypes.data_as(_lp), nkey, prefix.ctypes.data_as(_lp))
    return prefix


# quartets per primitive count: small, ordinary, and beyond 32 bits in all or in one count
COUNTS = [{1: 7}, {1: 100, 64: 3}, {1: 5, 3: 5, 9: 5, 27: 5, 81: 5}, {1: 1 << 20, 30: 1 << 18, 4096: 2000},
          {1: 3 << 30, 8: 1 << 29, 512: 1 << 20}, {16: 5 << 30}, {1: 1 << 31, 4096: (1 << 31) + 5},
          # shells of more than 8 primitives, up to four of 64
          {1: 300, 4097: 20, 10000: 1000, 1 << 24: 3}, {8: 100, 20736: 4, 20737: 4, 40000: 4}, {1 << 24: 1 << 20}]


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("case", range(len(COUNTS)))
def test_segments(seg, case, ordered):
    counts = COUNTS[case]
    nq, prims, mx = sum(counts.values()), sum(n * q for n, q in counts.items()), max(counts)
    prefix = _prefix(seg, counts)
    for k in range(seg.seg_pow()):
        assert prefix[k] == sum(q for n, q in counts.items() if n > 1 << k)
    pp = prefix.ctypes.data_as(_lp) if ordered else None
    desc = sorted(counts, reverse=True)
    at = np.concatenate([[0], np.cumsum([counts[n] for n in desc])])  # desc[i]: quartets at[i] .. at[i + 1]

    def largest(lo, hi):
        return max(n for i, n in enumerate(desc) if at[i] < hi and at[i + 1] > lo)

    first, lg = np.zeros(8, dtype=np.int64), np.zeros(8, dtype=np.int32)
    ns = seg.sl_segs(nq, prims, mx, pp, -1, first.ctypes.data_as(_lp), lg.ctypes.data_as(_ip))
    assert 1 <= ns <= 6 and first[0] == 0 and first[ns] == nq
    share = max(64, prims // (148 * 768)) if prims >= 148 * 768 else 16
    for k in range(ns):
        assert first[k + 1] >= first[k] and 0 <= lg[k] <= 5
        if ordered and first[k + 1] > first[k]:
            assert lg[k] == 5 or largest(first[k], first[k + 1]) <= share << int(lg[k])
    for share, cap in ((2, 1 << 24), (48, 1 << 24), (48, 8), (1000, 1), (1 << 30, 1 << 24)):
        f, st, nb = np.zeros(32, dtype=np.int64), np.zeros(32, dtype=np.int64), C.c_longlong()
        ns = seg.tile_segs(nq, share, mx, pp, cap, f.ctypes.data_as(_lp), st.ctypes.data_as(_lp), C.byref(nb))
        assert f[ns - 1] == 0 and st[ns - 1] == 0 and 1 << (ns - 1) <= cap
        for j in range(ns - 1, -1, -1):
            hi = f[j - 1] if j else nq
            assert hi >= f[j]
            assert (st[j - 1] if j else nb.value) == st[j] + ((hi - f[j]) << j)
            if ordered and hi > f[j]:
                assert j == ns - 1 and 1 << (j + 1) > cap or largest(f[j], hi) <= share << j


def test_keys(seg):
    """Keys order counts and keep apart those at a power of two; above 64 they span at most
    1/64 of the count."""
    ns = sorted({max(1, (1 << k) + d) for k in range(25) for d in (-1, 0, 1)} | set(range(1, 9000, 7)))
    ns = [n for n in ns if n <= 1 << 24]
    keys = [seg.seg_key_of(n) for n in ns]
    assert keys == sorted(keys)
    for a, b, ka, kb in zip(ns, ns[1:], keys, keys[1:]):
        assert ka < kb or (b > 64 and b - a <= b / 64 and (a - 1).bit_length() == (b - 1).bit_length())


def test_lanes_by_average(seg):
    """A class of unequal counts without an order: one segment, the caller's lanes."""
    first, lg = np.zeros(8, dtype=np.int64), np.zeros(8, dtype=np.int32)
    nq = 3 << 30
    assert seg.sl_segs(nq, 20 * nq, 4096, None, 2, first.ctypes.data_as(_lp), lg.ctypes.data_as(_ip)) == 1
    assert first[1] == nq and lg[0] == 2
