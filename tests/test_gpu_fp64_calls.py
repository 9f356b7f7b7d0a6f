"""What a caller of the FP64 path may count on besides the values: null grids are
refused before anything is launched, and integrate and backward give the same bits
from call to call; the longest cubes accepted run."""
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


# The longest cubes accepted (one pair, l = 0, 4 points on the short axes): what a CTA held
# when it kept a whole pair's tables, 8 bytes a column or plane and 24 a row of 227 KB.
LONGEST = {0: 29038, 1: 9678, 2: 29038}


def _long(axis, n):
    """One pair whose cube is n points long on axis, on a grid that it does not wrap around."""
    r = 1.5
    h = np.full(3, 1.2)
    h[axis] = r / (n // 2 - 0.5)
    npts = np.full(3, 5)
    npts[axis] = n + 9
    wl = T.synthetic("long", 1, 0, (4.0, 4.0), h * npts, [npts], 3)
    wl.tasks["radius"] = r
    return wl


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_longest_cubes(axis, oracle_lib):
    from gpu_util import run_collocate, run_integrate

    wl = _long(axis, LONGEST[axis])
    V = wl.potentials(seed=axis)
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    assert np.linalg.norm(run_collocate(wl)[0] - want) <= 1e-12 * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V) - hab).max() <= 1e-12 * np.abs(hab).max()
    grid = _zeros(*want.shape)
    level, tasks = np.array([wl.levels[0]], dtype=T.GRID_DTYPE), np.ascontiguousarray(wl.tasks)
    pab = _dev(wl.pab)
    capi.check(capi.lib().gpw_collocate_noalloc(level.ctypes.data, tasks.ctypes.data, 1, 0, pab.data_ptr(),
                                                grid.data_ptr(), None))
    assert np.linalg.norm(grid.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)
    one = np.zeros(want.shape)
    capi.collocate_pgf_product_rspace(oracle_lib.task_dict(wl, 0), one)
    assert np.linalg.norm(one - want) <= 1e-12 * np.linalg.norm(want)
    # the gradients' moments have two more powers: 8 (l + 3) bytes of table a row do not fit
    V, hab2, grad = [_dev(v) for v in V], _zeros(1), _zeros(1, 3)
    if axis == 1:
        with pytest.raises(capi.GpwError) as e:
            ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
            ts.backward(pab, V, hab2, grad)
        assert e.value.status == 4  # GPW_ERR_UNSUPPORTED, with the matrix elements
        assert np.abs(hab2.cpu().numpy() - hab).max() <= 1e-12 * np.abs(hab).max()


@pytest.mark.parametrize("axis,n", [(0, 9000), (0, 29038), (2, 9000)])
def test_long_cubes_backward(axis, n, oracle_lib):
    """s functions: dE/dRa_d = 2 zeta sum V (x_d - Ra_d) phi_a phi_b over the cube."""
    wl = _long(axis, n)
    V = wl.potentials(seed=1)
    ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
    hab, dra, dza = _zeros(1), _zeros(1, 3), _zeros(1)
    ts.backward(_dev(wl.pab), [_dev(v) for v in V], hab, dra=dra, dzeta=dza)
    ts.check()
    t, g = wl.tasks[0], wl.levels[0]
    phi = oracle_lib.batch(wl)[0]  # pab phi_a phi_b on the cube, each grid point once
    h, n3, rp = np.diag(g["dh"]), np.array(g["npts"]), t["ra"] + t["zetb"] / (t["zeta"] + t["zetb"]) * t["rab"]
    x = []  # the coordinate of each grid index: its image nearest to the product centre, relative to centre a
    for d in range(3):
        off = (np.arange(n3[d]) - np.floor(rp[d] / h[d]) + n3[d] // 2 - 1) % n3[d] - (n3[d] // 2 - 1)
        x.append((np.floor(rp[d] / h[d]) + off) * h[d] - t["ra"][d])
    X, Y, Z = x[0][None, None, :], x[1][None, :, None], x[2][:, None, None]
    w = phi * V[0]
    want = 2.0 * t["zeta"] * np.array([(w * X).sum(), (w * Y).sum(), (w * Z).sum()])
    size = 2.0 * t["zeta"] * np.abs(w).sum()  # sums of alternating signs: relative to their terms
    assert np.abs(dra.cpu().numpy()[0] - want).max() <= 1e-12 * 3.0 * size
    assert abs(float(dza) + (w * (X * X + Y * Y + Z * Z)).sum()) <= 1e-12 * 9.0 * size
    assert np.abs(hab.cpu().numpy() - oracle_lib.batch(wl, V=V)).max() <= 1e-12 * np.abs(w).sum() / abs(wl.pab[0])


@pytest.mark.parametrize("ortho", [True, False])
def test_captured_integrate_between_mixed_calls(ortho):
    """The parts' moments share their memory with the tiled integrate kernel's V slots: a captured FP64
    call gives the same bits after mixed calls, new tiles (general cells: the slots' first use) and a backward pass."""
    import torch

    cell = 10.0 if ortho else T.lattice_15(length=10.0)
    wl = T.synthetic("captured", 6, 2, (0.2, 0.4), cell, [(64,) * 3], 9, ortho=ortho)
    ts = capi.TaskSet.from_workload(capi.Plan(wl.levels), wl)
    V, pab, hab, other = [_dev(v) for v in wl.potentials(seed=3)], _dev(wl.pab), _zeros(wl.pab.size), _zeros(wl.pab.size)
    ts.integrate(V, hab)
    torch.cuda.synchronize()
    want = hab.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ts.integrate(V, hab)
    for tz in (8, 4):
        ts.set_tiles([tz])
        ts.integrate(V, other, "mixed")
        ts.backward(pab, V, other, dra := _zeros(6, 3))
        hab.zero_()
        graph.replay()
        ts.check()
        assert torch.equal(hab, want) and bool(dra.any())
