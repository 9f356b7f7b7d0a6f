"""Periodic images of a cube over one tile as items of their own: cells smaller
than the cubes (1 to 4 images per axis), tiles that the grid does not fill, both
tile shapes, explicit cube lists, and the error for more images than the tiled
path takes.  Against the CPU oracle at the mixed path's bar (1e-8)."""
import numpy as np
import pytest

from gpu_util import run_collocate, run_integrate
from libgpw_gb300 import capi, tasks as T

pytestmark = pytest.mark.gpu

TOL = 1e-8


def _check(wl, tz, oracle_lib):
    plan = capi.Plan(wl.levels)
    ts = capi.TaskSet.from_workload(plan, wl)
    ts.set_tiles([tz])
    V = wl.potentials(seed=3)
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    got = run_collocate(wl, "mixed", ts=ts, plan=plan)[0]
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V, "mixed", ts=ts, plan=plan) - hab).max() <= TOL * np.abs(hab).max()


# (radius / cell, npts): from cubes inside the cell to four images of an axis
@pytest.mark.parametrize("ratio,npts", [(0.2, (33, 31, 9)), (0.6, (20, 17, 8)), (1.1, (32, 16, 16)), (1.4, (30, 45, 21))])
@pytest.mark.parametrize("tz", [4, 8])
@pytest.mark.parametrize("ortho", [True, False])
def test_images(ratio, npts, tz, ortho, oracle_lib):
    cell = 6.0
    zp = np.log(1e10) / (ratio * cell) ** 2
    npts = npts if ortho else (npts[0],) * 3
    wl = T.synthetic("images", 12, 2, (0.5 * zp, 0.5 * zp), cell if ortho else T.lattice_15(length=cell), [npts],
                     int(100 * ratio) + tz, ortho=ortho)
    _check(wl, tz, oracle_lib)


def test_images_explicit_lists(oracle_lib):
    cell, npts = 5.0, (24, 24, 24)
    wl = T.synthetic("lists", 6, 1, (0.3, 0.4), cell, [npts], 17)
    table = []
    for t in wl.tasks:
        t["lb_cube"], t["ub_cube"], sb = capi.sphere_bounds(float(t["radius"]), np.eye(3) * cell / 24)
        t["sphere_offset"] = sum(len(x) for x in table)
        table.append(sb)
    wl.sphere_table = np.concatenate(table).astype(np.int32)
    _check(wl, 8, oracle_lib)


def test_too_many_images():
    wl = T.synthetic("many", 4, 0, (0.05, 0.06), 3.0, [(16, 16, 16)], 5)
    with pytest.raises(capi.GpwError) as e:
        run_collocate(wl, "mixed")
    assert e.value.status == 4  # GPW_ERR_UNSUPPORTED


# every degree of the summed moments, both tile shapes
@pytest.mark.parametrize("l", range(5))
@pytest.mark.parametrize("tz", [4, 8])
@pytest.mark.parametrize("ortho", [True, False])
def test_integrate_degrees(l, tz, ortho, oracle_lib):
    cell = 9.0 if ortho else T.lattice_15(length=9.0)
    wl = T.synthetic("degrees", 10, l, (0.4, 2.0), cell, [(35, 40, 27)], 50 + l, lmin=max(l - 1, 0), ortho=ortho)
    plan = capi.Plan(wl.levels)
    ts = capi.TaskSet.from_workload(plan, wl)
    ts.set_tiles([tz])
    V = wl.potentials(seed=3)
    hab = oracle_lib.batch(wl, V=V)
    assert np.abs(run_integrate(wl, V, "mixed", ts=ts, plan=plan) - hab).max() <= TOL * np.abs(hab).max()


def test_too_many_images_bounded(oracle_lib):
    """Cubes of about ten cells a side beside ordinary ones: no items for them (they would have
    hundreds per tile), the same status from tiled calls, and plain FP64 calls are not affected."""
    wl = T.synthetic("some", 40, 0, (0.05, 0.06), 3.0, [(16, 16, 16)], 5)
    wl.tasks["radius"][::2] = 1.4
    plan = capi.Plan(wl.levels)
    ts = capi.TaskSet.from_workload(plan, wl)
    items = ts.bins()[0]
    assert 20 <= items <= 20 * 2 * 8  # 20 pairs, 2 tiles, at most two images of an axis
    V = wl.potentials(seed=3)
    for run in (lambda: run_collocate(wl, "mixed", ts=ts, plan=plan), lambda: run_integrate(wl, V, "mixed", ts=ts, plan=plan)):
        with pytest.raises(capi.GpwError) as e:
            run()
        assert e.value.status == 4  # GPW_ERR_UNSUPPORTED
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    assert np.linalg.norm(run_collocate(wl, "fp64", ts=ts, plan=plan)[0] - want) <= 1e-12 * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V, "fp64", ts=ts, plan=plan) - hab).max() <= 1e-12 * np.abs(hab).max()
