"""The unit sums (csrc/separable.cuh) on meshes other than the recorded 20 x 20 one: a larger
square one, odd ones with different numbers of points along z and r, and one whose radial
points need more of the projection's shared memory than a launch takes by default (307)."""
import copy
import functools
import os

import numpy as np
import pytest

from golden_cases import GOLDEN, golden, namelist_for
from test_separable import _fields, _host_sums, host  # noqa: F401 (fixture)

# (points along z, radial points): the no-alloc entry's largest mesh, odd numbers, few and many
MESHES = [(40, 40), (13, 21), (22, 9), (4, 320)]


@functools.lru_cache(maxsize=None)
def _case(ngh, ngl):
    """A synthetic Bogoliubov state of N_sh = 6 on a mesh of ngh x ngl points: Gauss nodes, or
    equidistant radial ones where there are too many for those."""
    import pynfam_gb300.hel as hel
    from pynfam_gb300.pnfam_setup import setup_case
    from pynfam_gb300.synthetic import bogoliubov_nucleus
    path = os.path.join(GOLDEN, "S40.hel")
    g = copy.copy(hel.read_hel(path))
    x, w = np.polynomial.hermite.hermgauss(2 * ngh)
    g.xh, g.wh = x[ngh:], 2 * w[ngh:] * np.exp(x[ngh:] ** 2)
    if ngl <= 60:
        g.xl, w = np.polynomial.laguerre.laggauss(ngl)
        g.wl = w * np.exp(g.xl)
    else:
        g.xl, g.wl = np.linspace(0.05, 30.0, ngl), np.full(ngl, 30.0 / ngl)
    g.ngh, g.ngl = ngh, ngl
    read = hel.read_hel
    hel.read_hel = lambda p: g
    try:
        h = bogoliubov_nucleus(path, 6, seed=3, parity=True)
    finally:
        hel.read_hel = read
    nml = namelist_for("S40", golden("S40")["operators"]["RS1-K1"][0])
    nml["interaction"]["require_self_consistency"] = False
    return setup_case(nml, None, hfb=h)


@pytest.mark.parametrize("ngh,ngl", MESHES)
def test_tables_reproduce_direct_sums(host, ngh, ngl):  # noqa: F811
    """As on the recorded mesh: 1e-12 of the largest value."""
    c = _case(ngh, ngl)
    h = c.hfb
    phi = np.stack([h.wf, h.wfdr, h.wfdp, h.wfdz, h.wfd2_all])
    got, s, ws, x, wx = _host_sums(host, h, np.asarray(c.F.mat.cols), phi, 3)
    assert got == ngh
    assert np.max(np.abs(s - ws)) <= 1e-12 * np.max(np.abs(ws))
    assert np.max(np.abs(x - wx)) <= 1e-12 * np.max(np.abs(wx))


@pytest.mark.gpu
@pytest.mark.parametrize("ngh,ngl", MESHES)
@pytest.mark.parametrize("mixed", [False, True])
def test_field_matches_general_kernels(monkeypatch, ngh, ngl, mixed):
    """1e-12 (FP64) and 1e-5 (FP32) of the largest value, as on the recorded mesh."""
    c = _case(ngh, ngl)
    got = _fields(c, 4, mixed)
    monkeypatch.setenv("PNFAM_GB300_SEPARABLE", "0")
    want = _fields(c, 4, False)
    for g, w in zip(got, want):
        assert np.max(np.abs(g - w)) <= (1e-5 if mixed else 1e-12) * np.max(np.abs(w))


@pytest.mark.gpu
@pytest.mark.parametrize("ngh,ngl", MESHES)
def test_iterations_match_general_kernels(monkeypatch, ngh, ngl):
    """Five points (two or four per CTA leave one over): the FP64 iteration table to 1e-9 and
    the mixed form's strengths after the same few steps to 1e-5, as on the recorded mesh."""
    from pynfam_gb300.solver import GPUSolver
    c = _case(ngh, ngl)
    w = 8.0 + 2.0 * np.arange(5) + 3.0j
    res = []
    for env in (None, "0"):
        if env:
            monkeypatch.setenv("PNFAM_GB300_SEPARABLE", env)
        gpu = GPUSolver(c.hfb, c.couplings)
        gpu.set_operator(c.F, c.G)
        kw = dict(max_iter=4, eps=1e-13, quench=c.quench)
        res.append((gpu.solve(w, history=True, **kw).hist, gpu.solve(w, precision=1, settle=8, **kw)))
        gpu.close()
    (h0, m0), (h1, m1) = res
    np.testing.assert_allclose(h0, h1, rtol=1e-9, atol=1e-12)
    s0, s1 = m0.re_S + 1j * m0.im_S, m1.re_S + 1j * m1.im_S
    assert np.max(np.abs(s0 - s1)) <= 1e-5 * np.max(np.abs(s1))
