"""The FP64 field projection and densities over the whole mesh (k_hproj_fp64, k_density_fp64)
at the edges of their tables, against the product-basis kernels."""
import numpy as np
import pytest

from test_separable import _case, _fields


@pytest.mark.gpu
@pytest.mark.parametrize("name,nsh,op", [
    ("omega", 2, "GT-K0"),     # groups of a few outputs, blocks of one state
    ("S40", 5, "RS2-K2"),      # blocks without a partner, odd sizes
    ("Gd162", 13, "GT-K1"),    # pieces of 256 outputs and their remainders
    ("omega", 15, "GT-K0"),    # more than 64 rows of one spin: two pieces per tile, chunks of 8
])
def test_field_matches_product_basis(monkeypatch, name, nsh, op):
    """1e-12 of the largest element: sums of up to 1e4 products in another order."""
    c = _case(name, nsh, op)
    want = _fields(c, 6, False)
    monkeypatch.setenv("PNFAM_GB300_SEPARABLE", "0")
    got = _fields(c, 6, False)
    for g, w in zip(got, want):
        assert np.max(np.abs(g - w)) <= 1e-12 * np.max(np.abs(w))
