"""The Newton solve's kernels over the sizes where their launches change: a
mesh with one, two, three and four multigrid levels, chunks shorter and longer than a
block, restart cycles that end before convergence, FP64 and FP32 tangents.  The
multigrid solve ends at block-Jacobi's root (1e-7 of the step, the linear
conditioning of the tests beside), on the handle's stream, where a cycle is one graph,
and on the legacy default stream, where it is enqueued, bit for bit the same."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,restart", [(2, 2, 30), (5, 3, 30), (13, 9, 4), (33, 25, 30), (64, 48, 7), (131, 96, 30)])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_bulk"])
def test_multigrid_solve_over_the_sizes(nx, ny, restart, precision):
    import torch
    from biofem.gpu import GpuShell, BIOFEM_PC_AMG, BIOFEM_PC_BJACOBI
    w = configs.Workload(f"flat_{nx}x{ny}", nx, ny, z_sigma=1e-3, activation="smooth", index=220, pressure=2e-4)
    m = w.build_mesh()
    sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0, precision=precision)
    x0 = w.initial_x(m, sh.topology()["xyz0_full"])
    kw = dict(rtol=1e-10, gmres_max_it=2000, max_newton=20)
    xa, sa = sh.newton(x0, preconditioner=BIOFEM_PC_AMG, gmres_restart=restart, **kw)
    assert sa["converged"] == 1, sa
    xd = torch.tensor(x0, device="cuda")
    sd = sh.newton_device(xd.data_ptr(), 0, preconditioner=BIOFEM_PC_AMG, gmres_restart=restart, **kw)
    assert sd["gmres_its_total"] == sa["gmres_its_total"]
    np.testing.assert_array_equal(xd.cpu().numpy(), xa)
    xb, sb = sh.newton(x0, preconditioner=BIOFEM_PC_BJACOBI, gmres_restart=60, **{**kw, "gmres_max_it": 20000})
    assert sb["converged"] == 1, sb
    assert np.linalg.norm(xa - xb) <= 1e-7 * max(np.linalg.norm(xb - x0), 1e-30)
    sh.close()
