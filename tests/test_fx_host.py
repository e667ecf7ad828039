"""The fixed-point contraction of the FP64 row assembly (fx.cuh), run on the
host over one row of contributions: against extended-precision numpy, for
every subdivision table, for magnitudes across the double range, for Cartesian
pairs of very different size and for elements of very different size.

Tolerance (in units of 2^(E-31) / den^2, E the row's exponent of the (i, j) pair
plus the bits dropped for growth): each contribution rounds its sum (1/2) and
leaves out five lo.lo products of at most 1/2 each; w's own error (1/2 + 5, and
1/2 more where it is shifted to the row's exponent) reaches it times the column
sum of |N| (2.26) times den / 2^15; D's and N's own roundings add 0.8: at most
8 a contribution and slot.  With integer table values (the regular table)
nothing is left out and the table's own rounding adds 0.06.  The fixed-point row
(all its entries, each relative to its pair's size) must also be no further from the extended-precision one than the double chain
of fused multiply-adds it replaces, on a row of 24 contributions with blocks of
their own (an interior row of a regular mesh)."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from biofem.gpu import basis_tables

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
NBLK = 36


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if NVCC is None:
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("fx") / "fx_host"
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    str(ROOT / "tests" / "fx_host.cu"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("table,ints", [(0, 1), (0, 0), (3, 0), (5, 0), (7, 0), (10, 0)])
@pytest.mark.parametrize("scale,nc,shared", [(1.0, 24, 0), (1e-250, 24, 0), (1e290, 24, 0), (1e-3, 1, 0),
                                             (1e-3, 24, 1), (1e-3, 48, 1), (1e-3, 200, 1)])
def test_fixed_point_row_matches_extended_precision(driver, tmp_path, table, ints, scale, nc, shared):
    rng = np.random.default_rng(100 * table + nc)
    N = basis_tables()[table]
    nen = 12 if table == 0 else table + 6
    D = rng.standard_normal((nc, 15, 15)) * scale
    pair = 10.0 ** rng.uniform(-8, 0, (3, 3))                    # membrane, bending and coupling pairs
    D *= np.kron(np.ones((5, 5)), pair)
    D *= 10.0 ** rng.uniform(-2, 0, (nc, 1, 1))                  # elements of different size
    D[:, 3, 4] = 0.0
    a = rng.integers(0, nen, nc).astype(np.int32)
    # shared: several slots of a contribution add to one block, as ghost slots do
    tgt = np.array([rng.integers(0, NBLK, 16) if shared else rng.permutation(NBLK)[:16] for _ in range(nc)], np.int32)
    inp, out = tmp_path / "in.bin", tmp_path / "out.bin"
    with open(inp, "wb") as f:
        for x in (np.array([nc, nen, NBLK, ints], np.int32), a, tgt, D.astype(np.float64), N.astype(np.float64)):
            f.write(np.ascontiguousarray(x).tobytes())
    subprocess.run([str(driver), str(inp), str(out)], check=True)
    res = np.fromfile(out, np.float64)
    grow = int(res[0])
    kx, kd = res[1:].reshape(2, NBLK, 3, 3)
    L = np.longdouble
    ref = np.zeros((NBLK, 3, 3), L)
    count = np.zeros(NBLK)
    Dl = D.astype(L).reshape(nc, 5, 3, 5, 3)
    for c in range(nc):
        w = np.einsum("r,risj->isj", N[:, a[c]].astype(L), Dl[c])
        blk = np.einsum("isj,sb->bij", w, N[:, :nen].astype(L))
        for b in range(nen):
            ref[tgt[c, b]] += blk[b]
            count[tgt[c, b]] += 1
    E = np.frexp(np.abs(D).reshape(nc, 5, 3, 5, 3).max(axis=(0, 1, 3)))[1]
    unit = np.ldexp(L(1), (E + grow - 31).astype(int)) / L(10) ** 8
    ex = np.abs(kx.astype(L) - ref)
    # and the final rounding to double, half an ulp
    assert (ex <= 8 * unit * count[:, None, None] + np.abs(ref) * L(2) ** -53).all()
    # every entry relative to its pair's size
    e = [float(np.sqrt((((k.astype(L) - ref) / (scale * pair)) ** 2).sum())) for k in (kx, kd)]
    print(f"table {table} error {e[0]:.3g}, double chain {e[1]:.3g}")
    assert nc < 24 or shared or e[0] <= e[1], e
