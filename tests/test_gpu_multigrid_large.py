"""The multigrid cycle on meshes whose finest level smooths with A after the coarse
correction (A, P and A P together above the 96 MB that stay in L2: from some
200 x 150 cells; 36 bytes a block of A, and A P and P together 1.5 times as much)
and below.  A load step must converge on either side, its root checked by the
residual alone, and a linear solve to 1e-9 take no more than 60 iterations: it
takes 18 on 128 x 96 cells and 41 on 256 x 192 with a sound cycle, and block-Jacobi
takes some thousand."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,large", [(150, 112, False), (232, 174, True)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_bulk"])
def test_load_step_on_either_side_of_the_cycles_rule(nx, ny, large, precision):
    from biofem.gpu import GpuShell
    w = configs.Workload("sheet", nx, ny, z_sigma=1e-3, z_smooth=True, activation="smooth", index=270, pressure=1e-4)
    m = w.build_mesh()
    sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0, precision=precision)
    assert (36 * sh.nnzb * 2.5 > 1.2 * (96 << 20)) == large
    x0 = w.initial_x(m, sh.topology()["xyz0_full"])
    x, st = sh.newton(x0, rtol=1e-10, gmres_rtol=1e-9)
    R = sh.form_function(x)
    sh.close()
    print(st)
    assert st["converged"] == 1 and np.linalg.norm(R) <= 1.0001e-10 * st["r0"]
    assert st["gmres_its_total"] <= 60 * st["newton_its"] and st["gmres_its_last"] <= 60
