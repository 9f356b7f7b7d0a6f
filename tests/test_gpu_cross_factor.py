"""Tiled general cells with radii beyond the synthetic workloads' exp(-zetp r^2) = 1e-10:
the cross factor of the Gaussian reaches exp(1.5 zetp r^2) at the sphere's edge and must not
leave float's range, on the row's points or beside them.  Against the CPU oracle."""
import numpy as np
import pytest

from gpu_util import run_collocate, run_integrate
from libgpw_gb300 import capi, tasks as T

pytestmark = pytest.mark.gpu

RADIUS = 1.5
# Grid: the mixed path's bar.  Matrix elements: a row's slices carry 2^-35 of its largest
# V E X, which exceeds the values at its points by at most exp((k - 1) zetp r^2), k =
# G_00 (G^-1)_00 = 1.188 of this lattice, zetp r^2 <= 46 the points that are taken: 1.7e-7.
TOL_GRID, TOL_HAB = 1e-8, 2e-7


@pytest.mark.parametrize("exponent", [23, 46, 47, 60, 92, 150, 400])
@pytest.mark.parametrize("tz", [4, 8])
def test_wide_radii(exponent, tz, oracle_lib):
    zp = exponent / RADIUS**2
    wl = T.synthetic("wide", 40, 1, (0.5 * zp, 0.5 * zp), T.lattice_15(length=6.0), [(24, 24, 24)], exponent, ortho=False)
    wl.tasks["radius"] = RADIUS
    wl.tasks["rab"] *= 0.1  # (prefactors of order one)
    plan = capi.Plan(wl.levels)
    ts = capi.TaskSet.from_workload(plan, wl)
    ts.set_tiles([tz])
    V = wl.potentials(seed=3)
    want, hab = oracle_lib.batch(wl)[0], oracle_lib.batch(wl, V=V)
    got = run_collocate(wl, "mixed", ts=ts, plan=plan)[0]
    assert np.linalg.norm(got - want) <= TOL_GRID * np.linalg.norm(want)
    assert np.abs(run_integrate(wl, V, "mixed", ts=ts, plan=plan) - hab).max() <= TOL_HAB * np.abs(hab).max()
