"""The dense cube contractions at the edges of their blocks: fewer, exactly and more
rows than a CTA takes (8 and 1024), more planes than a cluster, one point per axis,
L up to 16; against numpy, within FP64 rounding of the sums' lengths."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import torch_dev
from libgpw_gb300 import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (3, 8, 5, 16), (9, 9, 33, 2), (17, 7, 64, 9), (2, 1023, 3, 4),
                                   (2, 1025, 2, 3), (40, 60, 60, 9), (65, 256, 3, 1)])
def test_core_shapes(shape):
    torch, dev = torch_dev()
    nz, ny, nx, L = shape
    rng = np.random.default_rng(7)
    ld = max(nz, ny, nx)
    pol, co = rng.uniform(-1, 1, size=(3, L, ld)), rng.uniform(-1, 1, size=(L, L, L))
    V = rng.uniform(-1, 1, size=(nz, ny, nx))
    Z, Y, X = pol[0, :, :nz], pol[1, :, :ny], pol[2, :, :nx]
    d = lambda a: torch.from_numpy(a).to(dev)  # noqa: E731
    d_co, d_pol, d_V = d(co), d(pol), d(V)
    out, back = torch.full((nz, ny, nx), 9.0, dtype=torch.float64, device=dev), d(np.full((L, L, L), 9.0))
    length, s = (C.c_int * 3)(nz, ny, nx), torch.cuda.current_stream().cuda_stream
    capi.check(capi.lib().gpw_collocate_core(length, L, d_co.data_ptr(), d_pol.data_ptr(), ld, out.data_ptr(), s))
    capi.check(capi.lib().gpw_integrate_core(length, L, d_pol.data_ptr(), ld, d_V.data_ptr(), back.data_ptr(), s))
    eps = 2.0 ** -53
    # every product is at most 1: L^3 terms and nz ny nx terms of three factors each
    want = np.einsum("agb,gz,by,ax->zyx", co, Z, Y, X, optimize=True)
    assert np.abs(out.cpu().numpy() - want).max() <= 4 * eps * L**3 * (3 * L + 3)
    want = np.einsum("zyx,gz,by,ax->gba", V, Z, Y, X, optimize=True)
    assert np.abs(back.cpu().numpy() - want).max() <= 4 * eps * nz * ny * nx * 8


@pytest.mark.parametrize("nz,ny,L,ok", [(3, 0, 2, True), (3, -1, 2, True), (3, -5, 1, False), (0, 4, 2, False)])
def test_core_no_points(nz, ny, L, ok):
    """Calls without points: nothing is written; a negative need of shared memory (8 L (L + ny)
    bytes for a plane's rows) and an empty grid of planes are errors."""
    torch, dev = torch_dev()
    pol, co = torch.ones(3 * L * 8, dtype=torch.float64, device=dev), torch.ones(L**3, dtype=torch.float64, device=dev)
    out = torch.full((64,), 9.0, dtype=torch.float64, device=dev)
    s = torch.cuda.current_stream().cuda_stream
    st = capi.lib().gpw_collocate_core((C.c_int * 3)(nz, ny, 3), L, co.data_ptr(), pol.data_ptr(), 8, out.data_ptr(), s)
    assert (st == 0) == ok
    torch.cuda.synchronize()
    assert bool((out == 9.0).all())
