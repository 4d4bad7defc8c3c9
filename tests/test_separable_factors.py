"""The search for the factors of a product basis (csrc/separable.cuh, ``sep_factors``) where a
block's time-reversed partner does not hold the same states in the same places."""
import numpy as np
import pytest

from test_separable import _case, _host_sums, host  # noqa: F401 (fixture)


@pytest.mark.parametrize("change", ["order", "sign", "scale"])
def test_partner_blocks_of_another_kind(host, change):  # noqa: F811
    """States of a partner block in reverse order, with the other sign, or (all functions of one
    z function) scaled: still a product basis, and its tables give the sums over the mesh
    (1e-12 of the largest value, as for the recorded order)."""
    c = _case("Gd162", 9, "GT-K1")
    h = c.hfb
    phi = np.stack([h.wf, h.wfdr, h.wfdp, h.wfdz, h.wfd2_all])
    for i in range(h.nb // 2, h.nb):
        s, u, e = int(h.isstart[i]), int(h.isstart[i] + h.num_spin_up[i]), int(h.isstart[i] + h.db[i])
        for lo, hi in ((s, u), (u, e)):
            if change == "order":
                phi[:, lo:hi] = phi[:, lo:hi][:, ::-1].copy()
            elif change == "sign":
                phi[:, lo:hi] *= -1.0
            else:
                phi[:, lo:hi] *= np.where(h.nz[lo:hi] == 2, 1.5, 1.0)[None, :, None]
    ngh, s, ws, x, wx = _host_sums(host, h, np.asarray(c.F.mat.cols), phi, 3)
    assert ngh == 20
    assert np.max(np.abs(s - ws)) <= 1e-12 * np.max(np.abs(ws))
    assert np.max(np.abs(x - wx)) <= 1e-12 * np.max(np.abs(wx))
