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


@pytest.mark.gpu
@pytest.mark.parametrize("change", ["component", "value", "nan"])
def test_other_bases_keep_the_general_kernels(monkeypatch, change):
    """A basis that is a product but for one state's z derivative, one value or a NaN: the field is that
    of the kernels over the mesh, to the last bit, and not that of the unit sums."""
    import copy
    import dataclasses
    from test_separable import _fields
    c = _case("S40", 6, "GT-K0")
    h, k = c.hfb, c.hfb.dqp // 2 + 3
    wf, wfdz, wfd2 = h.wf.copy(), h.wfdz.copy(), h.wfd2_all.copy()
    if change == "component":
        wfdz[k] *= 1.0 + 1e-9
    elif change == "value":
        wf[k, 37] += 1e-9
    else:
        wfd2[k, 5] = np.nan
    c = copy.copy(c)
    c.hfb = dataclasses.replace(h, wf=wf, wfdz=wfdz, wfd2_all=wfd2)
    got = _fields(c, 4, False)
    monkeypatch.setenv("PNFAM_GB300_SEPARABLE", "0")
    want = _fields(c, 4, False)
    assert all(np.array_equal(g, w, equal_nan=True) for g, w in zip(got, want))
    monkeypatch.delenv("PNFAM_GB300_SEPARABLE")
    units = _fields(_case("S40", 6, "GT-K0"), 4, False)
    assert any(not np.array_equal(g, w) for g, w in zip(got, units))
