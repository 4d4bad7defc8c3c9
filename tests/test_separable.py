"""The densities and the field projection of a z x radial product basis
(csrc/separable.cuh): factors and tables on the host, kernels against the general ones."""
import ctypes as C
import functools
import os
import subprocess

import numpy as np
import pytest

from golden_cases import GOLDEN, case_for

HERE = os.path.dirname(os.path.abspath(__file__))
# (ground state, N_sh, operator): parity blocks in the recorded basis, larger ones, and
# Omega-only blocks (every pair of n_z in a class)
CASES = [("S40", 6, "GT-K0"), ("Gd162", 9, "GT-K1"), ("S40", 6, "RS2-K2"), ("omega", 7, "GT-K1")]


@functools.lru_cache(maxsize=None)
def _case(name, nsh, op):
    from golden_cases import golden, namelist_for
    from pynfam_gb300.pnfam_setup import setup_case
    from pynfam_gb300.synthetic import bogoliubov_nucleus, ground_state
    hel = "Gd162" if name == "omega" else name
    path = os.path.join(GOLDEN, f"{hel}.hel")
    hfb = bogoliubov_nucleus(path, nsh, seed=5, parity=False) if name == "omega" else ground_state(path, nsh)
    nml = namelist_for(hel, golden(hel)["operators"][op][0])
    nml["interaction"]["require_self_consistency"] = False
    return setup_case(nml, None, hfb=hfb)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sep") / "sep.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "sep_host_check.cpp")], check=True)
    return C.CDLL(so)


def _host_sums(lib, h, cols, phi, seed):
    """(ngh, C, direct C, h, direct h) of random rho and fields."""
    rng = np.random.default_rng(seed)
    db = np.ascontiguousarray(h.db, np.int32)
    nup = np.ascontiguousarray(h.num_spin_up, np.int32)
    cols = np.ascontiguousarray(cols, np.int32)
    n = int(h.nghl)
    nxy = sum(int(db[i]) * int(db[j]) for i, j in enumerate(cols) if j >= 0)
    rho = rng.standard_normal(nxy)
    m = rng.standard_normal((4, 17, n))
    out_c = np.zeros((4, 16, n))
    out_h = np.zeros(nxy)
    phi = np.ascontiguousarray(phi)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    ngh = lib.sep_host_check(len(db), p(db), p(nup), n, p(phi), p(cols), p(rho), p(m), p(out_c), p(out_h))
    want_c, want_h = np.zeros_like(out_c), np.zeros_like(out_h)
    st, o = np.concatenate([[0], np.cumsum(db)]), 0
    for i, j in enumerate(cols):
        if j < 0:
            continue
        d, e = int(db[i]), int(db[j])
        blk = rho[o:o + d * e].reshape(d, e, order="F")
        hb = np.zeros((d, e))
        for s, ra in enumerate((slice(0, nup[i]), slice(nup[i], d))):
            for t, rb in enumerate((slice(0, nup[j]), slice(nup[j], e))):
                a, b = phi[:, st[i]:st[i] + d][:, ra], phi[:, st[j]:st[j] + e][:, rb]
                k = 2 * s + t
                want_c[k] += np.einsum("qar,ab,pbr->qpr", a[:4], blk[ra, rb], b[:4], optimize=True).reshape(16, n)
                f = m[k, :16].reshape(4, 4, n)
                x = np.einsum("qar,qpr,pbr->ab", a[:4], f, b[:4], optimize=True)
                x += np.einsum("ar,r,br->ab", a[0], m[k, 16], b[4], optimize=True)
                x += np.einsum("ar,r,br->ab", a[4], m[k, 16], b[0], optimize=True)
                hb[ra, rb] = 2 * x
        want_h[o:o + d * e] = hb.reshape(-1, order="F")
        o += d * e
    return ngh, out_c, want_c, out_h, want_h


@pytest.mark.parametrize("name,nsh,op", CASES)
def test_tables_reproduce_direct_sums(host, name, nsh, op):
    """Density and projection through the units and items equal the sums over the whole
    mesh to rounding: 1e-12 of the largest value (a few hundred terms of size one, each
    rounded at 1e-16)."""
    h = _case(name, nsh, op).hfb
    phi = np.stack([h.wf, h.wfdr, h.wfdp, h.wfdz, h.wfd2_all])
    fc = np.asarray(_case(name, nsh, op).F.mat.cols)
    tr = np.array([h.partner(i) for i in range(h.nb)])
    for cols in (fc, fc[tr]):   # the operator's structure and the Y quadrant's
        ngh, c, wc, x, wx = _host_sums(host, h, cols, phi, 3)
        assert ngh == 20
        assert np.max(np.abs(c - wc)) <= 1e-12 * np.max(np.abs(wc))
        assert np.max(np.abs(x - wx)) <= 1e-12 * np.max(np.abs(wx))


@pytest.mark.parametrize("change", ["value", "component", "energy", "nan", "zero"])
def test_other_bases_are_not_accepted(host, change):
    """A basis that is a product everywhere but in one value, one component, one state's
    Laplacian, or with a NaN or a vanishing state, keeps the general kernels."""
    h = _case("S40", 6, "GT-K0").hfb
    phi = np.stack([h.wf, h.wfdr, h.wfdp, h.wfdz, h.wfd2_all])
    k = h.dqp // 2 + 3
    if change == "value":
        phi[0, k, 37] += 1e-9
    elif change == "component":
        phi[3, k] *= 1.0 + 1e-9
    elif change == "energy":
        phi[4, k, ::2] += 1e-9 * phi[0, k, ::2]
    elif change == "nan":
        phi[1, k, 5] = np.nan
    else:
        phi[:, k] = 0.0
    assert _host_sums(host, h, np.asarray(_case("S40", 6, "GT-K0").F.mat.cols), phi, 3)[0] == 0


def _fields(c, seed, mixed, scale=1.0):
    from pynfam_gb300.solver import GPUSolver
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, c.G)
    rng = np.random.default_rng(seed)
    ins = [scale * (rng.standard_normal(gpu.nxy) + 1j * rng.standard_normal(gpu.nxy)) for _ in range(4)]
    out = gpu.calc_hamiltonian(*ins, mixed=mixed)
    gpu.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name,nsh,op", CASES)
@pytest.mark.parametrize("mixed", [False, True])
def test_field_matches_general_kernels(monkeypatch, name, nsh, op, mixed):
    """The field through the product basis against the FP64 kernels over the whole mesh:
    1e-12 (FP64, rounding) and 1e-5 (FP32, the bound of the other FP32 paths)."""
    c = _case(name, nsh, op)
    got = _fields(c, 4, mixed)
    monkeypatch.setenv("PNFAM_GB300_SEPARABLE", "0")
    want = _fields(c, 4, False)
    for g, w in zip(got, want):
        assert np.max(np.abs(g - w)) <= (1e-5 if mixed else 1e-12) * np.max(np.abs(w))


@pytest.mark.gpu
@pytest.mark.parametrize("points", [1, 2, 7])
def test_batches_match_general_kernels(monkeypatch, points):
    """FP64 and mixed iterations of a few points (odd counts: two points per CTA leave
    one over) against the general kernels: the FP64 iteration table to 1e-9, the mixed
    form's strengths after the same number of steps to 1e-5."""
    from pynfam_gb300.solver import GPUSolver
    c, _ = case_for("S40", "RS1-K1", 0)
    w = 8.0 + 2.0 * np.arange(points) + 3.0j
    res = []
    for env in (None, "0"):
        if env:
            monkeypatch.setenv("PNFAM_GB300_SEPARABLE", env)
        gpu = GPUSolver(c.hfb, c.couplings)
        gpu.set_operator(c.F, c.G)
        kw = dict(max_iter=6, eps=1e-13, quench=c.quench)
        res.append((gpu.solve(w, history=True, **kw).hist, gpu.solve(w, precision=1, settle=8, **kw)))
        gpu.close()
    (h0, m0), (h1, m1) = res
    np.testing.assert_allclose(h0, h1, rtol=1e-9, atol=1e-12)
    s0, s1 = m0.re_S + 1j * m0.im_S, m1.re_S + 1j * m1.im_S
    assert np.max(np.abs(s0 - s1)) <= 1e-5 * np.max(np.abs(s1))
