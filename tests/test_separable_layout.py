"""Where a point's unit sums lie (csrc/separable.cuh, ``sep_sums``)."""
import ctypes as C
import itertools
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("seplayout") / "layout.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "sep_layout_check.cpp")], check=True)
    return C.CDLL(so)


def test_places_are_aligned_and_apart(lib):
    """Every point starts on four values (16 bytes in FP32, the projection's reads), also
    with an odd number of radial points and structures of unequal size; the parts of a point
    do not overlap."""
    for ngl, nf, x, y in itertools.product((1, 7, 20, 40), (1, 5, 36), ((3, 2), (4, 4), (7, 1)), ((2, 2), (6, 9))):
        nu = np.array([nf, x[0], y[0], x[1], y[1]], np.int64)
        at = np.zeros(4, np.int64)
        p = lambda a: a.ctypes.data_as(C.c_void_p)
        lib.sep_layout_check(C.c_longlong(ngl), p(nu), p(at))
        assert at[2] % 4 == 0 and at[0] % 2 == 0 and at[1] % 2 == 0 and at[3] % 4 == 0
        assert at[0] >= 2 * ngl * nf * at[3]
        assert at[1] >= at[0] + 2 * ngl * max(x)
        assert at[2] >= at[1] + 2 * ngl * max(y)
