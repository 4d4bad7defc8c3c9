"""Strength sums (k_contract): more cross terms than one pass of the kernel takes, and vectors
from less than one chunk to many."""
import numpy as np
import pytest

from test_separable import _case


@pytest.mark.gpu
@pytest.mark.parametrize("terms", [1, 7, 8, 9, 17])
@pytest.mark.parametrize("name,nsh", [("omega", 2), ("S40", 7)])
def test_repeated_terms(name, nsh, terms):
    """A cross term equal to the operator has its strength, wherever it stands in the list."""
    from pynfam_gb300.solver import GPUSolver
    c = _case(name, nsh, "GT-K0")
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, [c.F] * terms)
    kw = dict(max_iter=3, eps=1e-13, quench=c.quench)
    for precision in (0, 1):
        r = gpu.solve(np.array([9.0 + 2.0j, 12.0 + 1.0j]), precision=precision, **kw)
        S = r.re_S + 1j * r.im_S
        assert S.shape == (2, terms + 1) and np.all(np.abs(S[:, 0]) > 0)
        assert np.array_equal(S[:, 1:], np.repeat(S[:, :1], terms, axis=1))
    gpu.close()
