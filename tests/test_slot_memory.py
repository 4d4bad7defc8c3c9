"""The memory estimate of a serving slot against what an engine allocates."""
import numpy as np
import pytest

from pynfam_gb300.serve import field_bytes, slot_bytes
from test_separable import _case


def test_field_part_counts_the_units():
    """The part that does not grow with nxy at N_sh = 6 (20 x 20 mesh, 7 n_z in two parities):
    density shares of at least 4 groups, 104 mean-field components and the unit sums."""
    c = _case("S40", 6, "GT-K0")
    b = field_bytes(c.hfb, c.F.mat.cols, True)
    n = c.hfb.nghl
    fixed = 12 * (2 * 4 * 56 * n + 208 * 2 * n)
    assert b >= fixed
    assert b - field_bytes(c.hfb, c.F.mat.cols, False) == b // 3
    # every class at most 7 x 7 units of 22 sums at 20 radial points
    assert b <= 12 * (2 * 24 * 56 * n + 208 * 2 * n + 2 * 20 * 22 * 4 * 49 + 3)


@pytest.mark.gpu
@pytest.mark.parametrize("name,nsh,op,mixed", [("S40", 6, "GT-K0", True), ("S40", 6, "GT-K0", False),
                                               ("Gd162", 9, "GT-K1", True)])
def test_estimate_matches_engine(name, nsh, op, mixed):
    """64 slots: within 10 % of the estimate (all quasiparticles are active in these bases)
    beside 32 MB of tables and allocation granularity."""
    import torch
    from pynfam_gb300.solver import GPUSolver
    c = _case(name, nsh, op)
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, c.G)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    eng = gpu.engine(64, max_iter=10, eps=1e-8, quench=c.quench, precision=int(mixed), settle=8 if mixed else 0)
    used = before - torch.cuda.mem_get_info()[0]
    eng.close()
    gpu.close()
    want = 64 * slot_bytes(c.F.mat.nelem, 50, mixed, field=field_bytes(c.hfb, c.F.mat.cols, mixed))
    assert 0.9 * want - (32 << 20) <= used <= 1.1 * want + (32 << 20)
