"""What a caller of the FP64 path may count on besides the values: null grids are
refused before anything is launched, and integrate and backward give the same bits
from call to call."""
import ctypes as C

import numpy as np
import pytest

from libgpw_gb300 import capi, tasks as T

pytestmark = pytest.mark.gpu

INVALID_ARG = 1  # GPW_ERR_INVALID_ARG


def _zeros(*n):
    import torch

    return torch.zeros(n, dtype=torch.float64, device="cuda:0")


def _dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")


@pytest.mark.parametrize("ortho", [True, False])
@pytest.mark.parametrize("null_level", [0, 1])
def test_backward_null_grid(null_level, ortho):
    """Every pair on level 0.  The matrix elements need every grid, the gradients those with pairs."""
    wl = T.synthetic("null", 3, 1, (1.0, 2.0), 8.0 if ortho else T.lattice_15(length=8.0), [(24,) * 3, (12,) * 3], 1,
                     ortho=ortho)
    ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
    V = [_dev(v) for v in wl.potentials(seed=1)]
    grids = (C.c_void_p * 2)(*[None if l == null_level else V[l].data_ptr() for l in range(2)])
    pab, hab, grad = _dev(wl.pab), _zeros(wl.pab.size), _zeros(3, 3)

    def backward(h, g):
        return capi.lib().gpw_backward(ts.handle, pab.data_ptr(), grids, h, g, None, None, None, None)

    assert backward(hab.data_ptr(), grad.data_ptr()) == INVALID_ARG
    assert backward(hab.data_ptr(), None) == INVALID_ARG
    assert backward(None, grad.data_ptr()) == (INVALID_ARG if null_level == 0 else 0)
    ts.check()
    assert not hab.any() and bool(grad.any()) == (null_level == 1)


# undivided pairs, pairs divided into items, both kinds of cell, and the float-float kernel of untiled general cells
@pytest.mark.parametrize("n,zeta", [(200, (2.0, 50.0)), (40, (0.3, 20.0)), (2, (0.2, 0.3))])
@pytest.mark.parametrize("ortho,precision", [(True, "fp64"), (False, "fp64"), (False, "mixed")])
def test_integrate_repeats_bit_for_bit(n, zeta, ortho, precision):
    import torch

    cell = 10.0 if ortho else T.lattice_15(length=10.0)
    wl = T.synthetic("repeat", n, 3, zeta, cell, [(64,) * 3], 5, ortho=ortho)
    ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
    V, pab = [_dev(v) for v in wl.potentials(seed=3)], _dev(wl.pab)

    def outputs():
        hab = _zeros(wl.pab.size)
        ts.integrate(V, hab, precision)
        out = [hab]
        if precision == "fp64":
            out += [_zeros(wl.pab.size), _zeros(n, 3), _zeros(n, 3), _zeros(n), _zeros(n)]
            ts.backward(pab, V, *out[1:])
        return out

    first = outputs()
    for _ in range(12):
        assert all(torch.equal(a, b) for a, b in zip(first, outputs()))
    ts.check()
