"""The conversions between double, float and pairs of floats that csrc/pair_arith.cuh takes
from the bits, against numpy's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
EDGE = [0.0, -0.0, 1.0, 1 + 2.0**-24, 1 + 3 * 2.0**-24, 1 + 2.0**-23, 2 - 2.0**-52, 2.0**-74, 2.0**-126, 2.0**-127,
        2.0**-149, 2.0**-150, 1.5 * 2.0**-150, 3 * 2.0**-150, 2.0**-151, 5e-324, 2.0**126, 2.0**127,
        2.0**128 - 2.0**103, 2.0**128 - 2.0**104, 2.0**128, 1e300, np.inf, -np.inf, np.nan]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pair") / "pair.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "pair_host_check.cpp")],
                   check=True)
    r = C.CDLL(so)
    r.pair_host_max.restype = C.c_ulonglong
    return r


@pytest.mark.parametrize("s", [0, 40, -40, 800])
def test_conversions(lib, s):
    rng = np.random.default_rng(7)
    x = np.concatenate([EDGE, rng.standard_normal(20000) * 2.0 ** rng.integers(-160, 130, 20000),
                        rng.standard_normal(20000) * 2.0 ** (rng.integers(-70, 100, 20000) - s)])
    y = np.concatenate([np.array(EDGE[:-6] + EDGE[-3:] + [0.0] * 3).astype(np.float32), rng.integers(0, 2**32, len(x) - len(EDGE), dtype=np.uint32).view(np.float32)])
    n = len(x)
    hi, lo, f = (np.zeros(n, np.float32) for _ in range(3))
    d, scale = np.zeros(n), np.zeros(n, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    y = np.ascontiguousarray(y, np.float32)
    lib.pair_host_check(n, p(x), p(y), s, p(hi), p(lo), p(f), p(d), p(scale))
    with np.errstate(all="ignore"):
        assert np.array_equal(f, x.astype(np.float32), equal_nan=True)
        assert np.array_equal(np.signbit(f[x == x]), np.signbit(x[x == x]))
        z = np.ldexp(x, s)
        want = np.ldexp(y.astype(np.float64), s)
        normal = ~(np.abs(want) < np.finfo(np.float64).tiny)
        assert np.array_equal(d[normal], want[normal], equal_nan=True)
        # a pair: 24 leading bits to nearest, 24 of the 29 others
        r = (np.abs(z) >= 2.0**-74) & (np.abs(z) < 2.0**127) & (np.abs(x) >= np.finfo(np.float64).tiny)
        assert np.all(np.abs(hi[r].astype(np.float64) - z[r]) <= np.abs(z[r]) * 2.0**-24)
        assert np.all(np.abs(hi[r].astype(np.float64) + lo[r].astype(np.float64) - z[r]) <= np.abs(z[r]) * 2.0**-49)
        small = np.abs(z) < 2.0**-74
        assert np.all(np.abs(hi[small].astype(np.float64) + lo[small] - z[small]) <= 2.0**-98)
        big = ~(np.abs(z) < 2.0**128)
        assert np.array_equal(hi[big & (x == x)], np.where(z[big & (x == x)] > 0, np.inf, -np.inf))
        assert np.all(np.isnan(hi[x != x]))
    k = np.isfinite(x) & (np.abs(x) > 2.0**-900)
    m = np.ldexp(np.abs(x[k]), scale[k])
    assert np.all(((m >= 1) & (m < 2)) | (np.abs(scale[k]) == 900))


def test_largest(lib):
    x = np.array([0.0, -3.0, np.nan, 2.5, -0.0, 5e-324])
    for v in (x, np.append(x, -np.inf), np.array([0.0, -0.0, np.nan])):
        got = np.array([lib.pair_host_max(len(v), v.ctypes.data_as(C.c_void_p))], np.uint64).view(np.float64)[0]
        assert got == np.fmax.reduce(np.abs(v), initial=0.0)
