"""The fixed-point row at the edge of the rule that keeps a row in integers
(fx.cuh, kFxSpread): one stiff element, 23 softer by 2^-4.  Over the blocks that
hold soft elements only, each row's error against extended precision must be no
larger than the double chain's, in the sum over six rows of 24 contributions.

Expected: a contribution's roundings are 2^-57.8 of the row's unit E together
(half a unit of K, 2.26 half units of w), uniform, so an rms of some 2^-58.8 of E,
or 2^-54.8 of the soft elements; the chain's 30 roundings of 2^-53 of growing
values leave it near 2^-52.2 of the result.  Two binades further apart the
integers would be the worse."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from biofem.gpu import basis_tables

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
NBLK, NC, L = 36, 24, np.longdouble


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if NVCC is None:
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("fx") / "fx_host"
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    str(ROOT / "tests" / "fx_host.cu"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("table,ints", [(0, 1), (5, 0), (10, 0)])
def test_soft_elements_beside_a_stiff_one(driver, tmp_path, table, ints):
    N = basis_tables()[table]
    nen = 12 if table == 0 else table + 6
    err = np.zeros(2)
    for seed in range(6):
        rng = np.random.default_rng(1000 * table + seed)
        D = rng.uniform(0.5, 1.0, (NC, 15, 15)) * rng.choice([-1.0, 1.0], (NC, 15, 15))
        D[1:] *= 2.0 ** -4
        a = rng.integers(0, nen, NC).astype(np.int32)
        tgt = np.array([rng.permutation(NBLK)[:16] for _ in range(NC)], np.int32)
        inp, out = tmp_path / "in.bin", tmp_path / "out.bin"
        with open(inp, "wb") as f:
            for x in (np.array([NC, nen, NBLK, ints], np.int32), a, tgt, D, N):
                f.write(np.ascontiguousarray(x).tobytes())
        subprocess.run([str(driver), str(inp), str(out)], check=True)
        k = np.fromfile(out)[1:].reshape(2, NBLK, 3, 3).astype(L)
        ref, soft = np.zeros((NBLK, 3, 3), L), np.ones(NBLK, bool)
        for c in range(NC):
            w = np.einsum("r,risj->isj", N[:, a[c]].astype(L), D[c].astype(L).reshape(5, 3, 5, 3))
            np.add.at(ref, tgt[c, :nen], np.einsum("isj,sb->bij", w, N[:, :nen].astype(L)))
        soft[tgt[0, :nen]] = False
        err += [float(((x - ref)[soft] ** 2).sum()) for x in k]
    assert 0 < err[0] <= err[1], np.sqrt(err)
