"""A context's operator changed while an engine holds the context."""
import numpy as np
import pytest

from pynfam_gb300.pnfam_setup import setup_case
from test_separable import _case

W = 5.0 + 0.7 * np.arange(6) + 2.0j
KW = dict(max_iter=60, eps=1e-8)


def _run(eng, n):
    out = {}
    while eng.active:
        eng.launch()
        for r in eng.finish():
            out[r.tag] = (r.iters, r.S[0])
    assert sorted(out) == list(range(n))
    return np.array([out[k][0] for k in range(n)]), np.array([out[k][1] for k in range(n)])


def _engine(c, **kw):
    from pynfam_gb300.solver import GPUSolver
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, c.G)
    return gpu, gpu.engine(len(W), quench=c.quench, **KW, **kw)


def _other(c):
    """The same ground state with an operator of other blocks."""
    import copy
    nml = copy.deepcopy(c.nml)
    nml["ext_field"]["operator_k"] = 0
    o = setup_case(nml, None, hfb=c.hfb)
    assert not np.array_equal(o.F.mat.cols, c.F.mat.cols)
    return o


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(), dict(broyden_m=7), dict(precision=1, settle=7), dict(precision=1)],
                         ids=["fp64", "short", "settled", "unsettled"])
def test_operator_changes_under_an_engine(kw):
    """162Gd at N_sh = 12, where 0.89 of the pairs are active: the engine solves for the
    operator that is set while it is empty, goes on when the same one is set between two of
    its evaluations, and its points refuse one of other blocks; results as on a context of
    their own, to the last bit."""
    from pynfam_gb300._lib import PnfamGPUError
    c = _case("Gd162", 12, "GT-K1")
    o = _other(c)
    want = {}
    for name, x in (("c", c), ("o", o)):
        gpu, eng = _engine(x, **kw)
        eng.admit(W, np.arange(len(W)))
        want[name] = _run(eng, len(W))
        eng.close()
        gpu.close()
    gpu, eng = _engine(c, **kw)
    for name, x in (("c", c), ("o", o), ("c", c)):
        gpu.set_operator(x.F, x.G)
        eng.admit(W, np.arange(len(W)))
        eng.launch()
        assert eng.finish() == []
        gpu.set_operator(x.F, x.G)
        with pytest.raises(PnfamGPUError):
            gpu.set_operator(*((o.F, o.G) if x is c else (c.F, c.G)))
        its, S = _run(eng, len(W))
        assert np.array_equal(its, want[name][0]) and np.array_equal(S, want[name][1]), name
    eng.close()
    gpu.close()
