"""What a caller of the FP64 path may count on besides the values: null grids are
refused before anything is launched."""
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
