"""The FP64 row assembly's two ways: exact integer sums, and plain FP64 for rows
near an end of the exponent range.  A stiffness scaled by 2^980 scales K by 2^980
and takes its rows past the integers' range, so the two must agree: chains of
some 400 double operations (24 contributions, 15 products and sums each) of 1.1e-16
against sums rounded at 2^-57 of a row's largest entry.  Bound 1e-12 of the
Frobenius norm, over real, ghost and irregular patches and both kinds of tables."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [configs.small(9, 7, index=230, activation="random", pressure=0.0),
                               configs.small(8, 5, index=231, basis=1, tnormal=1, n_qp=2, pressure=0.0),
                               configs.SphereWorkload("sphere_f4", 4, index=232, pressure=0.0)],
                         ids=["flat", "flat_exact", "sphere"])
def test_integer_rows_equal_double_rows(w):
    from biofem.gpu import GpuShell
    m = w.build_mesh()
    K = []
    for scale in (1.0, 2.0 ** 980):
        sh = GpuShell(m, w, configs.MU * scale, configs.BULK * scale, configs.H0)
        x = w.initial_x(m, sh.topology()["xyz0_full"])
        x[: 3 * m.n_v] += 1e-4 * np.random.default_rng(7).standard_normal(3 * m.n_v)
        k = np.asarray(sh.form_jacobian(x)[1], np.float64)
        K.append((k, sh.to_scipy(k)))
        sh.close()
    (k1, s1), (k2, s2) = K
    assert np.isfinite(k2).all()
    nreal = 3 * m.n_v
    a, b = s1.toarray()[:nreal, :nreal], s2.toarray()[:nreal, :nreal]
    big = np.abs(b) > 2.0 ** 900                # identity rows stay as they are
    assert big.any()
    d = np.where(big, b * 2.0 ** -980, 0.0) - np.where(big, a, 0.0)
    assert np.linalg.norm(d) <= 1e-12 * np.linalg.norm(np.where(big, a, 0.0))
