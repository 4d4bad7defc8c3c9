"""Runs of every form on one context, in several orders and over two operators: each finds
what it finds on a context of its own, whichever tables and buffers the runs before it left."""
import itertools

import numpy as np
import pytest

from golden_cases import case_for

W = 8.0 + 2.0 * np.arange(4) + 3.0j
RUNS = {"fp64": dict(), "short": dict(broyden_m=7), "settled": dict(precision=1, settle=8),
        "unsettled": dict(precision=1), "none": dict(broyden_m=0)}


def _solve(gpu, c, run):
    r = gpu.solve(W, max_iter=4, eps=1e-13, quench=c.quench, **RUNS[run])
    return np.concatenate([r.re_S.ravel(), r.im_S.ravel(), r.si])


def _field(gpu, mixed):
    rng = np.random.default_rng(4)
    ins = [rng.standard_normal(gpu.nxy) + 1j * rng.standard_normal(gpu.nxy) for _ in range(4)]
    return np.concatenate(gpu.calc_hamiltonian(*ins, mixed=mixed))


@pytest.mark.gpu
@pytest.mark.parametrize("separable", ["1", "0"])
def test_runs_do_not_depend_on_earlier_ones(monkeypatch, separable):
    """To the last bit (the tuner's choices are kept per process)."""
    from pynfam_gb300.solver import GPUSolver
    monkeypatch.setenv("PNFAM_GB300_SEPARABLE", separable)
    cases = [case_for("S40", op, 0)[0] for op in ("RS2-K2", "GT-K0")]
    want = {}
    for k, c in enumerate(cases):
        for run in RUNS:
            for _ in range(2):   # the first may tune
                gpu = GPUSolver(c.hfb, c.couplings)
                gpu.set_operator(c.F, c.G)
                want[k, run] = _solve(gpu, c, run)
                want[k, "field"], want[k, "field32"] = _field(gpu, False), _field(gpu, True)
                gpu.close()
    for order in list(itertools.permutations(RUNS))[::17]:
        gpu = GPUSolver(cases[0].hfb, cases[0].couplings)
        for k, c in ((0, cases[0]), (1, cases[1]), (0, cases[0])):
            gpu.set_operator(c.F, c.G)
            for run in order:
                assert np.array_equal(_solve(gpu, c, run), want[k, run]), (order, k, run)
                assert np.array_equal(_field(gpu, False), want[k, "field"]), (order, k, run)
                assert np.array_equal(_field(gpu, True), want[k, "field32"]), (order, k, run)
        gpu.close()
