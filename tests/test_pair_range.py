"""Pairs of floats of small numbers (csrc/pair_arith.cuh): nothing is dropped above the least
denormal float."""
import ctypes as C

import numpy as np
import pytest

from test_pair_arith import lib  # noqa: F401 (fixture)


@pytest.mark.parametrize("s", [0, 60, -60])
def test_small_values(lib, s):  # noqa: F811
    """|hi + lo - x 2^s| within 2^-49 of the value, or 2^-148 (both parts rounded to multiples
    of 2^-149) where that is more: what a conversion to float and that of the remainder give."""
    rng = np.random.default_rng(11)
    x = np.ldexp(rng.uniform(1, 2, 60000) * rng.choice([-1.0, 1.0], 60000), rng.integers(-160, 5, 60000) - s)
    n = len(x)
    y, hi, lo, f = (np.zeros(n, np.float32) for _ in range(4))
    d, scale = np.zeros(n), np.zeros(n, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    lib.pair_host_check(n, p(x), p(y), s, p(hi), p(lo), p(f), p(d), p(scale))
    z = np.ldexp(x, s)
    err = np.abs((z - hi.astype(np.float64)) - lo.astype(np.float64))
    assert np.all(err <= np.maximum(2.0**-49 * np.abs(z), 2.0**-148))
