"""The multigrid setup where a diagonal block of the tangent is nearly singular: a
flat sheet compressed in its plane until the bending stiffness of an interior
node against its own normal displacement (positive) and the membrane force's
share (negative) cancel to 1e-4, 1e-8 and 1e-10 of its in-plane stiffness.  D^-1 A,
whose largest eigenvalue the setup estimates in FP32, then has eigenvalues of
some 1e3, 1e5 and 1e6 (the off-diagonal couplings of that row and of its column,
over the root of the vanishing entry).  The tangent is indefinite and the solve
stops at its 60 iterations; what it is asked for is a step: finite, and taking the
in-plane compression (all of the residual, 0.26) out of the sheet to a tenth."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ratio", [1e-4, 1e-8, 1e-10])
def test_setup_with_a_nearly_singular_diagonal_block(ratio):
    from biofem.gpu import GpuShell, BIOFEM_PC_AMG
    w = configs.Workload("flat", 14, 12, pressure=0.0, lambda_a=1.0, index=250)
    m = w.build_mesh()
    sh = GpuShell(m, w, configs.MU, configs.BULK, 3 * configs.H0)
    X = np.asarray(sh.topology()["xyz0_full"], float).reshape(-1, 3)
    mid = int(np.argmin(np.linalg.norm(m.xyz0 - m.xyz0.mean(0), axis=1)))

    def state(c):
        return (X * [c, c, 1.0]).ravel()

    def stiffness(c):
        k = sh.to_scipy(sh.form_jacobian(state(c))[1]).tocsr()
        return k[3 * mid + 2, 3 * mid + 2] / k[3 * mid, 3 * mid]

    lo, hi = 0.9, 1.0                     # indefinite, definite
    assert stiffness(lo) < 0 < stiffness(hi)
    s = 1.0
    while not 0 < s < ratio:
        c = 0.5 * (lo + hi)
        s = stiffness(c)
        lo, hi = (c, hi) if s < 0 else (lo, c)
    x, st = sh.newton(state(c), preconditioner=BIOFEM_PC_AMG, max_newton=1, rtol=1e-12, gmres_rtol=1e-8, gmres_max_it=60)
    sh.close()
    assert np.isfinite(x).all()
    assert st["rfinal"] <= 0.1 * st["r0"], st
