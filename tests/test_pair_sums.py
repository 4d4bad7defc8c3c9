"""The Broyden dots' sums across a warp (csrc/pair_arith.cuh) are FP64 sums."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_sums_across_the_lanes(tmp_path):
    """Against sums in extended precision: 2^-50 of the sum of the magnitudes (five levels of
    FP64 additions, the sum of a lane's parts and the comparison: 7 times 2^-53), where sums of
    pairs of floats keep about 2^-48."""
    from pynfam_gb300 import build
    so = str(tmp_path / "sum.so")
    subprocess.run([build.nvcc_path(), build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", so,
                    os.path.join(HERE, "pair_sum_check.cu")], check=True)
    rng = np.random.default_rng(2)
    n = 4096
    v = rng.standard_normal((2, n, 32)) * 10.0 ** rng.uniform(-9, 3, (2, n, 1))
    v[:, ::2] = np.abs(v[:, ::2])
    hi = v.astype(np.float32)
    lo = (v - hi).astype(np.float32)
    a, b = (np.ascontiguousarray(np.stack([hi[k], lo[k]], axis=-1)) for k in range(2))
    out = np.zeros((n, 2))
    p = lambda x: x.ctypes.data_as(C.c_void_p)
    assert C.CDLL(so).pair_sum_check(n, p(a), p(b), p(out)) == 0
    for k, x in enumerate((a, b)):
        exact = x.astype(np.longdouble).sum(axis=(1, 2))
        size = np.abs(x.astype(np.float64)).sum(axis=(1, 2))
        assert np.all(np.abs(out[:, k] - exact.astype(np.float64)) <= 2.0**-50 * size)
