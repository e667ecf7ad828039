"""The fixed-point row's functions (fx.cuh) as the FP64 row assembly uses them,
run on the host against extended precision: every subdivision table of both kinds
and the flat cap triangle's, with the follower-pressure blocks, in the row's unit
and with every element in its own (fx_wide); and the rule that decides between them.

Tolerances.  In the row's unit u = 2^(E-31) / den^2, E the row's exponent and the
growth bits: 8 u a contribution and slot (test_fx_host.py derives it), on the
integers themselves, over the entries that carry no load (a load's rounding there
is a double's, of v den^2).  With every element's own unit: 8 of its units a
contribution and slot, and a rounding of 2^-53 of the running sum's magnitude for
the conversion, for each addition and for the final scale."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from biofem.gpu import load_library

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
NBLK, L = 40, np.longdouble


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if NVCC is None:
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("fxrows") / "fx_rows_host"
    subprocess.run([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    str(ROOT / "tests" / "fx_rows_host.cu"), "-o", str(exe)], check=True)
    return exe


def tables(kind):
    out = np.zeros(11 * 80)
    assert load_library().GetGpuBasisTablesKind(kind, out.ctypes.data) == 0
    return out.reshape(11, 5, 16)


CAP = np.zeros((5, 16))                 # a1 = x2 - x1, a2 = x3 - x1
CAP[0, :2] = -1, 1
CAP[1, 0], CAP[1, 2] = -1, 1


@pytest.mark.parametrize("kind,table", [(k, t) for k in (0, 1) for t in (0, 3, 4, 5, 6, 7, 8, 9, 10, "cap")])
@pytest.mark.parametrize("nc,spread", [(1, 0.0), (24, 0.0), (24, 6.0)], ids=["one", "alike", "uneven"])
@pytest.mark.parametrize("load", [0.0, 1.0, 1e4])
def test_rows_against_extended_precision(driver, tmp_path, kind, table, nc, spread, load):
    N = CAP if table == "cap" else tables(kind)[table]
    nen = 3 if table == "cap" else 12 if table == 0 else table + 6
    den = 31 * 324 if kind else 10000
    rng = np.random.default_rng([kind, 99 if table == "cap" else table, nc, int(spread), int(load)])
    D = rng.uniform(0.5, 1, (nc, 15, 15)) * rng.choice([-1.0, 1.0], (nc, 15, 15)) * 1e-3
    D *= 10.0 ** rng.uniform(-spread, 0, (nc, 1, 1))
    a = rng.integers(0, nen, nc).astype(np.int32)
    a[0] = 1                                            # a corner's row
    tgt = np.array([rng.permutation(NBLK)[:16] for _ in range(nc)], np.int32)
    P = rng.uniform(-1, 1, (nc, 3, 3)) * 1e-3 * load
    inp, out = tmp_path / "in.bin", tmp_path / "out.bin"
    with open(inp, "wb") as f:
        for x in (np.array([nc, nen, NBLK, den], np.int32), a, tgt, D, N, P):
            f.write(np.ascontiguousarray(x).tobytes())
    subprocess.run([str(driver), str(inp), str(out)], check=True)
    res = np.fromfile(out)
    ints, grow, E = res[0], int(res[1]), res[2:11].reshape(3, 3).astype(int)
    hi, lo, kw = res[11:].reshape(3, NBLK, 3, 3).astype(L)
    ref, mag = np.zeros((NBLK, 3, 3), L), np.zeros((NBLK, 3, 3), L)
    count, loads, own = np.zeros((NBLK, 1, 1)), np.zeros((NBLK, 3, 3)), np.zeros((NBLK, 3, 3), L)
    for c in range(nc):
        w = np.einsum("r,risj->isj", N[:, a[c]].astype(L), D[c].astype(L).reshape(5, 3, 5, 3))
        blk = np.einsum("isj,sb->bij", w, N[:, :nen].astype(L))
        Ec = np.frexp(np.maximum(np.abs(D[c]).reshape(5, 3, 5, 3).max(axis=(0, 2)), 1e-300))[1]
        for b in range(nen):
            t = tgt[c, b]
            ref[t] += blk[b]
            mag[t] += np.abs(blk[b])
            count[t] += 1
            own[t] += 8 * np.ldexp(L(1), Ec - 31) / L(den) ** 2
        if a[c] < 3:
            for k in range(3):
                x, y, z = P[c, k].astype(L)
                m = np.array([[0, -z, y], [z, 0, -x], [-y, x, 0]], L)
                ref[tgt[c, k]] += m
                mag[tgt[c, k]] += np.abs(m)
                loads[tgt[c, k]] += np.abs(m) > 0
    unit = np.ldexp(L(1), E + grow - 31) / L(den) ** 2
    ulp = L(2) ** -53
    clear = loads == 0
    assert (np.abs(hi * L(2) ** 32 + lo - ref / unit) <= 8 * count)[clear].all()
    assert (np.abs(kw - ref) <= own + 2 * (count + loads + 2) * mag * ulp).all()
    # the rule: rows of like elements with a load of their size stay integer, uneven ones do not
    assert ints == float(spread == 0 and load <= 1.0)
