"""The residual kernel's two forms (one lane an element, or three for meshes
that leave FP64 units idle) and the FP32-bulk residual's, on both sides of
each rule's line and where the last warp is ragged, against the oracle.
Bounds as in the parity tests: 1e-10 ||R||; the tangent call returns the same R
bit for bit."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,kw", [
    (2, 2, {}),                                     # 8 triangles, less than a warp's ten
    (7, 3, dict(n_qp=1, pressure=1e-3)),            # 42: four warps and two elements
    (9, 5, dict(n_qp=2, c33_iters=1)),              # fewer points than lanes
    (8, 5, dict(n_qp=6, basis=1, tnormal=1)),       # two points a lane
    (80, 76, dict(pressure=1e-4)),                  # 12,160: the last size of the three-lane FP64 form
    (79, 77, dict(pressure=1e-4)),                  # 12,166: the first of the one-lane form
    (96, 95, {}),                                   # 18,240: the last of the three-lane float-float form
    (107, 86, {}),                                  # 18,404: beyond
])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_bulk"])
def test_residual_forms_match_the_oracle(oracle_lib, nx, ny, kw, precision):
    from biofem.gpu import GpuShell
    w = configs.small(nx, ny, activation="random", index=210, **kw)
    m = w.build_mesh()
    sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0, precision=precision)
    t = sh.topology()
    x = w.initial_x(m, t["xyz0_full"])
    x[: 3 * m.n_v] += 1e-3 / nx * np.random.default_rng(3).standard_normal(3 * m.n_v)
    o = oracle_lib.setup_given_topology(m, w, t, configs.MU, configs.BULK, configs.H0)
    o.set_threads(8)
    Ro = o.residual(x)
    R = sh.form_function(x)
    assert np.linalg.norm(R - Ro) <= 1e-10 * np.linalg.norm(Ro)
    Rj, _ = sh.form_jacobian(x)
    np.testing.assert_array_equal(Rj, R)
    sh.close()
