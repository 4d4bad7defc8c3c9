"""Device memory of a context that changes its operator: buffers only grow for what a call
needs."""
import numpy as np
import pytest

from test_separable import _case


@pytest.mark.gpu
def test_next_operator_leaves_run_buffers():
    """After a run in the active form (162Gd at N_sh = 12: 0.89 of the pairs) setting the
    operator again, and a field of either precision, take what one point needs: less than 16
    MB, where whole-block buffers of the run's 16 points and 50 history columns would be 150
    MB more. The run then repeats to the last bit."""
    import torch
    from pynfam_gb300.solver import GPUSolver
    c = _case("Gd162", 12, "GT-K1")
    gpu = GPUSolver(c.hfb, c.couplings)
    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
    w = 5.0 + 0.5 * np.arange(16) + 2.0j
    gpu.set_operator(c.F, c.G)
    ins = [np.ones(gpu.nxy, complex)] * 4
    gpu.calc_hamiltonian(*ins, mixed=True)
    first = gpu.solve(w, max_iter=3, quench=c.quench)
    before = free()
    gpu.set_operator(c.F, c.G)
    gpu.calc_hamiltonian(*ins)
    gpu.calc_hamiltonian(*ins, mixed=True)
    assert before - free() < 16 << 20
    again = gpu.solve(w, max_iter=3, quench=c.quench)
    gpu.close()
    assert np.array_equal(first.re_S, again.re_S) and np.array_equal(first.im_S, again.im_S)
