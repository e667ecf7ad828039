"""The caller's limit on a linear solve's iterations (gmres_max_it) over Newton steps
that keep the multigrid hierarchy: a solve whose tolerance is out of reach ends at
the limit, kept hierarchy or not, so the load step takes at most
newton_its * gmres_max_it iterations.  The limit is a whole number of restart
cycles here, since a cycle is not cut short.  The load step converges all the
same: the iterations it is given reduce each linear residual far enough."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("forcing", [0, 1])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_bulk"])
def test_a_solve_keeps_to_its_iterations(precision, forcing):
    from biofem.gpu import GpuShell
    w = configs.Workload("flat", 24, 18, z_sigma=1e-3, z_smooth=True, activation="smooth", index=260, pressure=1e-4)
    m = w.build_mesh()
    sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0, precision=precision)
    x0 = w.initial_x(m, sh.topology()["xyz0_full"])
    x, st = sh.newton(x0, rtol=1e-10, gmres_rtol=1e-15, gmres_restart=10, gmres_max_it=20, max_newton=20, forcing=forcing)
    ref, sr = sh.newton(x0, rtol=1e-10)
    sh.close()
    print(st)
    assert st["converged"] == 1 and sr["converged"] == 1
    assert st["gmres_its_last"] <= 20 and st["gmres_its_total"] <= 20 * st["newton_its"], st
    assert np.linalg.norm(x - ref) <= 1e-7 * np.linalg.norm(ref - x0)
