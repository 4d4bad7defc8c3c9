"""The field evaluation on complex arrays (pnfam_gpu_calc_hamiltonian_z) against the entry
points on separate planes: the same numbers, whatever the arrays' place and order."""
import ctypes as C

import numpy as np
import pytest

from test_separable import _case

pytestmark = pytest.mark.gpu


def _planes(gpu, ins, mixed):
    from pynfam_gb300 import _lib
    parts = [np.ascontiguousarray(p) for a in ins for p in (a.real, a.imag)]
    outs = [np.zeros(gpu.nxy) for _ in range(8)]
    fn = gpu.lib.pnfam_gpu_calc_hamiltonian_mixed if mixed else gpu.lib.pnfam_gpu_calc_hamiltonian
    _lib.check(fn(gpu.ctx, *[_lib.dptr(x) for x in parts + outs]))
    return [outs[2 * k] + 1j * outs[2 * k + 1] for k in range(4)]


@pytest.mark.parametrize("separable", [True, False])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("name,nsh,op", [("omega", 2, "GT-K0"), ("S40", 6, "RS2-K2"), ("Gd162", 9, "GT-K1")])
def test_same_as_planes(monkeypatch, name, nsh, op, mixed, separable):
    from pynfam_gb300 import _lib
    from pynfam_gb300.solver import GPUSolver
    if not separable:
        monkeypatch.setenv("PNFAM_GB300_SEPARABLE", "0")
    c = _case(name, nsh, op)
    gpu = GPUSolver(c.hfb, c.couplings)
    gpu.set_operator(c.F, c.G)
    n = gpu.nxy
    rng = np.random.default_rng(9)
    ins = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(4)]
    want = _planes(gpu, ins, mixed)
    for args in (ins, [np.repeat(a, 2)[::2] for a in ins], [a.tolist() for a in ins]):
        got = gpu.calc_hamiltonian(*args, mixed=mixed)
        assert len(got) == 4
        for g, w in zip(got, want):
            assert g.shape == (n,) and g.dtype == complex and np.array_equal(g, w)
    # results in four places
    outs = [np.zeros(n + 1, dtype=complex) for _ in range(4)]
    ptrs = [(C.c_void_p * 4)(*[a.ctypes.data for a in group]) for group in (ins, outs)]
    _lib.check(gpu.lib.pnfam_gpu_calc_hamiltonian_z(gpu.ctx, int(mixed), *ptrs))
    for g, w in zip(outs, want):
        assert np.array_equal(g[:n], w) and g[n] == 0
    with pytest.raises(ValueError):
        gpu.calc_hamiltonian(ins[0][:-1], *ins[1:])
    gpu.close()
