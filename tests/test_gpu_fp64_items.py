"""The FP64 kernels' items at the edges of their blocks: cubes whose width is
just below, at and above the 8, 16 and 32 columns of a block, few and many planes,
one and several items per pair, every l, against the CPU oracle (1e-12, the FP64
path's bar)."""
import numpy as np
import pytest

from gpu_util import run_collocate, run_integrate
from libgpw_gb300 import capi, tasks as T

pytestmark = pytest.mark.gpu

H = 0.25  # grid step


def _pairs(half, lmax, func, ortho, n=3, npts=(40, 36, 44)):
    """n pairs whose cubes are 2 half + 2 points wide (every l up to lmax)."""
    zeta = np.log(1e10) / ((half + 0.5) * H) ** 2 / 2.0
    cell = np.array(npts) * H if ortho else T.lattice_15(length=npts[0] * H)
    return T.synthetic("items", n, lmax, (zeta, zeta), cell, [npts if ortho else (npts[0],) * 3], 11 + half + lmax,
                       ortho=ortho, compute_tau=func, lmin=max(0, lmax - 1))


@pytest.mark.parametrize("half", [0, 1, 2, 3, 4, 7, 8, 15, 16, 24])
@pytest.mark.parametrize("lmax,func", [(0, 0), (2, 1), (4, 0), (4, 1)])
def test_ortho_items(half, lmax, func, oracle_lib):
    wl = _pairs(half, lmax, func, True)
    V = wl.potentials(seed=half)
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    got = run_collocate(wl)[0]
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V) - hab).max() <= 1e-12 * np.abs(hab).max()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("half", [1, 6, 17])
def test_general_items(half, precision, tol, oracle_lib):
    wl = _pairs(half, 3, 0, False)
    V = wl.potentials(seed=half)
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    got = run_collocate(wl, precision)[0]
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V, precision) - hab).max() <= tol * np.abs(hab).max()


@pytest.mark.parametrize("n", [1, 60, 64])
def test_few_planes_per_cta(n, oracle_lib):
    """20 planes of a pair in CTAs of one, two, and two or three (152 SMs): warps share a plane's rows."""
    import torch

    wl = _pairs(9, 2, 0, True, n=n)
    level, tasks = np.array([wl.levels[0]], dtype=T.GRID_DTYPE), np.ascontiguousarray(wl.tasks)
    pab = torch.from_numpy(wl.pab).cuda()
    grid = torch.zeros(T.grid_shape(wl.levels[0]), dtype=torch.float64, device="cuda")
    capi.check(capi.lib().gpw_collocate_noalloc(level.ctypes.data, tasks.ctypes.data, n, 0, pab.data_ptr(),
                                                grid.data_ptr(), torch.cuda.current_stream().cuda_stream))
    want = oracle_lib.batch(wl)[0]
    assert np.linalg.norm(grid.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)
