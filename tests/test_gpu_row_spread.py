"""The FP64 row assembly's two forms: integer sums in one unit a row, and sums in
double for rows whose elements lie far apart, whose load lies far above the
stiffness, with elements that are not finite, or near an end of the exponent range.

A stiffness scaled by 2^990 scales every element's tangent by exactly 2^990 (the
largest entry of these meshes is near 1e-2, field 2006 of at most 1998 for the
integers), so that handle sums all its rows in double, and its K times 2^-990 is
that form's K of the unscaled mesh.  Rows that leave the integers for one of the
other reasons must equal it bit for bit: the same sums of the same numbers.
Where the integers serve, the two forms agree within 1e-12 of the Frobenius norm
(24 additions of 1.1e-16 against sums rounded at 2^-57 of a row's largest entry)
and differ in some last bit, which shows that both have run."""
import numpy as np
import pytest

from biofem import configs

pytestmark = pytest.mark.gpu

S = 2.0 ** 990


def blocks(m, w, x=None, scale=1.0):
    """(K as n x n x 3 x 3 of the real nodes, patches, real row kinds) of one handle."""
    from biofem.gpu import GpuShell
    sh = GpuShell(m, w, configs.MU * scale, configs.BULK * scale, configs.H0)
    t = sh.topology()
    if x is None:
        x = w.initial_x(m, t["xyz0_full"])
    K = sh.to_scipy(np.asarray(sh.form_jacobian(x)[1], np.float64)).toarray()
    sh.close()
    n = m.n_v
    return K[: 3 * n, : 3 * n].reshape(n, 3, n, 3).transpose(0, 2, 1, 3), t, x


def patches(m, t):
    nen = np.where(t["ire"] != 0, t["val"] + 6, 12)
    return [set(p[:k]) for p, k in zip(t["patch"], nen)]


def free_rows(m):
    free = np.ones(m.n_v, bool)
    if m.n_edge:
        free[m.bnodes[: m.n_bnodes[0]]] = False
    return free


def smooth(m, full):
    x = full.reshape(-1, 3).copy()
    p = x[: m.n_v]
    x[: m.n_v] += 0.02 * np.stack([np.sin(2 * p[:, 1]), np.sin(3 * p[:, 0]), 2 * np.sin(3 * p[:, 0]) * np.cos(2 * p[:, 1])], 1)
    return x.ravel()


def flat(pressure, **kw):
    return configs.Workload("flat", 12, 9, pressure=pressure, activation="smooth", index=240, **kw)


def test_rows_of_uneven_elements_are_summed_in_double():
    """One column of cells 2^-10 as wide as the others: rows that hold both kinds."""
    w = flat(0.0)
    m = w.build_mesh()
    h = m.meta["lx"] / 12
    m.xyz0[:, 0] = np.where(m.xyz0[:, 0] > 5.5 * h, m.xyz0[:, 0] - h * (1 - 2.0 ** -10), m.xyz0[:, 0])
    _, t, _ = blocks(m, w)
    x = smooth(m, np.asarray(t["xyz0_full"], float))
    k1, _, _ = blocks(m, w, x)
    k2, _, _ = blocks(m, w, x, S)
    assert np.isfinite(k2).all()
    width = np.ptp(m.xyz0[m.tri][:, :, 0], axis=1)
    kinds = [set() for _ in range(m.n_v)]
    for e, p in enumerate(patches(m, t)):
        for i in p:
            if i < m.n_v:
                kinds[i].add(bool(width[e] < 0.1 * h))
    rows = np.array([len(k) == 2 for k in kinds]) & free_rows(m)
    assert rows.sum() > 30
    np.testing.assert_array_equal(k1[rows], k2[rows] / S)


def test_a_load_far_above_the_stiffness_leaves_it_its_digits():
    """Follower pressure 2^8 times the stiffness: blocks of nodes that share a patch but no triangle carry no load."""
    w = flat(64.0)
    m = w.build_mesh()
    _, t, _ = blocks(m, w)
    x = smooth(m, np.asarray(t["xyz0_full"], float))
    k1, _, _ = blocks(m, w, x)
    k0, _, _ = blocks(m, flat(0.0), x, S)
    apart = np.ones((m.n_v, m.n_v), bool)
    for a in range(3):
        for b in range(3):
            apart[m.tri[:, a], m.tri[:, b]] = False
    # a ghost's load goes to its parents: interior rows
    apart[[i for p in patches(m, t) if max(p) >= m.n_v for i in p if i < m.n_v]] = False
    apart &= free_rows(m)[:, None]
    assert np.abs(k1[free_rows(m)]).max() > 2.0 ** 3 * np.abs(k0[apart]).max() / S
    assert (k0[apart] != 0).any(axis=(1, 2)).sum() > 300
    np.testing.assert_array_equal(k1[apart], k0[apart] / S)


@pytest.mark.parametrize("w", [configs.small(9, 7, index=241, activation="random", pressure=0.0),
                               configs.small(8, 5, index=242, basis=1, tnormal=1, n_qp=2, pressure=0.0),
                               configs.small(10, 6, index=243, pressure=1e-3),
                               configs.SphereWorkload("sphere_f4", 4, index=244, pressure=1e-3),
                               configs.cone(8, pressure=1e-3), configs.capped(16, 8, True, pressure=1e-3)],
                         ids=["flat", "flat_exact", "flat_pressure", "sphere", "cone_v8", "capped"])
def test_both_forms_agree(w):
    import dataclasses
    m = w.build_mesh()
    k1, _, x = blocks(m, w)
    k2, _, _ = blocks(m, dataclasses.replace(w, pressure=w.pressure * S), x, S)
    assert np.isfinite(k2).all()
    rows = free_rows(m)
    a, b = k1[rows], k2[rows]
    if w.pressure:                 # K is divided by the largest external force where that is above 1
        b = b / np.abs(b).max()
        b *= np.vdot(a, b) / np.vdot(b, b)
    else:
        b = b / S
        assert (a != b).any()
    assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)


def test_an_element_that_is_not_finite_stays_in_its_blocks():
    """One element's activation is NaN; with one C33 sub-iteration its stress is, too."""
    import torch
    from biofem.gpu import GpuShell
    w = flat(0.0, c33_iters=1)
    m = w.build_mesh()
    _, t, _ = blocks(m, w)
    x = smooth(m, np.asarray(t["xyz0_full"], float))
    k0, _, _ = blocks(m, w, x, S)
    p = patches(m, t)
    e = next(i for i in range(m.n_elmt // 2, m.n_elmt) if max(p[i]) < m.n_v and len(p[i]) == 12)
    m.gamma_scale[e] = np.nan
    sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0)
    d_x = torch.tensor(x, device="cuda")
    d_R = torch.empty_like(d_x)
    d_K = torch.empty((sh.nnzb, 3, 3), dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    sh.jacobian_device(d_x.data_ptr(), d_R.data_ptr(), d_K.data_ptr(), s)
    torch.cuda.synchronize()
    n = m.n_v
    k = sh.to_scipy(d_K.cpu().numpy()).toarray()[: 3 * n, : 3 * n].reshape(n, 3, n, 3).transpose(0, 2, 1, 3)
    sh.close()
    nodes = sorted(p[e])
    free = free_rows(m)
    hit = np.zeros((n, n), bool)
    hit[np.ix_(nodes, nodes)] = True
    hit &= free[:, None]
    assert np.isnan(k[hit]).any(axis=(1, 2)).all()
    assert np.isfinite(k[~hit]).all()
    others = ~hit & free[:, None] & np.isin(np.arange(n), nodes)[:, None]
    np.testing.assert_array_equal(k[others], k0[others] / S)
