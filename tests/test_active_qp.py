"""Runs that iterate the active quasiparticles only: N_sh = 8, where the pairing window
erases a sixth of the quasiparticles, against the oracle on whole blocks."""
import os

import numpy as np
import pytest

from golden_cases import GOLDEN, golden, namelist_for
from oracle.fam_oracle import FAMOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op,start", [("GT-K0", None), ("RS1-K1", None), ("GT-K1", "erased"), ("GT-K1", "active")])
def test_history_and_state_match_oracle(op, start):
    """Four iterations from X = 0, from a start vector that vanishes on the erased
    quasiparticles, and from one that does not (whole blocks are iterated then): the
    iteration table and the final vector to 1e-9, as the other tests against the oracle."""
    from pynfam_gb300.hfb_solution import load_hfb_solution
    from pynfam_gb300.pnfam_setup import setup_case
    from pynfam_gb300.solver import GPUSolver
    hfb = load_hfb_solution(os.path.join(GOLDEN, "S40_nsh8.hel"))
    nml = namelist_for("S40", golden("S40")["operators"][op][0])
    nml["interaction"]["require_self_consistency"] = False
    c = setup_case(nml, None, hfb=hfb)
    w = 7.0 + 6.0j
    orc = FAMOracle(c.hfb, c.couplings, c.F, c.G, quench=c.quench)
    x0 = None
    if start:
        x0 = 1e-3 * np.random.default_rng(2).standard_normal(4 * orc.nxy)
        if start == "active":
            full = orc.solve(w, max_iter=1, eps=1e-30, broyden_m=50).vector
            x0[full == 0.0] = 0.0
            assert np.any(x0 == 0.0)
    kw = {} if x0 is None else dict(x0=x0, si0=1.0)
    ref = orc.solve(w, max_iter=4, eps=1e-30, broyden_m=50, **kw)
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, c.G)
    r = gpu.solve([w], max_iter=4, eps=1e-30, broyden_m=50, quench=c.quench, history=True, x0=x0, return_state=True)
    gpu.close()
    for h in ref.history[1:]:
        g = r.hist[0, h[0]]
        for a, b in ((g[0], h[2]), (g[1], h[3]), (g[2], h[4])):
            assert abs(a - b) <= 1e-9 * max(abs(b), 1e-6), (h, g)
    assert np.max(np.abs(r.state[0] - ref.vector)) <= 1e-9 * np.max(np.abs(ref.vector))
