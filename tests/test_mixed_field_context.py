"""Single-precision fields on contexts that hold buffers of several points: the field entry
points take neither the block GEMMs nor the pair tensor, and the tuner, whose trials take
both, belongs to the first run that does."""
import numpy as np
import pytest

from golden_cases import case_for


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(4)]


@pytest.mark.gpu
@pytest.mark.parametrize("setting", ["PNFAM_GB300_SEPARABLE=0", "PNFAM_GB300_PAIR_MIN=2", "PNFAM_GB300_TC_DENSITY=0"])
def test_field_between_solves(monkeypatch, setting):
    """FP64 solve of four points, mixed field, a larger operator, mixed field again, a mixed
    solve: fields within 1e-5 of the FP64 ones (the bound of the FP32 paths), and the mixed
    solve finds what it finds on a fresh context (1e-6, its own convergence)."""
    from pynfam_gb300.solver import GPUSolver
    name, value = setting.split("=")
    monkeypatch.setenv(name, value)
    small, _ = case_for("S40", "RS2-K2", 0)
    large, _ = case_for("S40", "GT-K0", 0)
    assert small.F.mat.nelem < large.F.mat.nelem
    w = 8.0 + 2.0 * np.arange(4) + 3.0j
    kw = dict(max_iter=40, eps=1e-8, quench=large.quench, precision=1, settle=7)
    gpu = GPUSolver(small.hfb, small.couplings)
    gpu.set_operator(small.F, small.G)
    gpu.solve(w, max_iter=3, quench=small.quench)
    for c in (small, large):
        if c is large:
            gpu.set_operator(c.F, c.G)
        ins = _inputs(gpu.nxy, 3)
        for g, f in zip(gpu.calc_hamiltonian(*ins, mixed=True), gpu.calc_hamiltonian(*ins)):
            assert np.max(np.abs(g - f)) <= 1e-5 * np.max(np.abs(f))
    got = gpu.solve(w, **kw)
    gpu.close()
    fresh = GPUSolver(large.hfb, large.couplings)
    fresh.set_operator(large.F, large.G)
    want = fresh.solve(w, **kw)
    fresh.close()
    s, r = (x.re_S + 1j * x.im_S for x in (got, want))
    assert np.max(np.abs(s - r)) <= 1e-6 * np.max(np.abs(r))
