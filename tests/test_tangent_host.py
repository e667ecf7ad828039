"""The element algebra (element.cuh) on the host.

The analytic tangent against central differences of the element forces in long
double, relative step d = 1e-6: truncation d^2 times a ratio of third to first
derivatives of up to 1e3 (thickness corrections) and round-off 1e-19 / d leave
1e-9; a wrong or missing term is of order 1e-2 and more.  Bound 1e-8.

The double tangent against the long-double one: about 1e3 operations of 1e-16,
cancellation in the corrector's residual another 1e2.  Bound 1e-11.

FFAcc: nine products, each with an error of a few 2^-48 of its magnitude and
two-sums of the running sum's.  Bound 2^-44 of the sum of the magnitudes."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def tangent_host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("tangent") / "tangent_host"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                    str(ROOT / "tests" / "tangent_host.cu"), "-o", str(exe)], check=True)
    return exe


@pytest.mark.parametrize("nq,iters,tnormal", [(1, 1, 0), (1, 4, 1), (2, 3, 0), (3, 4, 0), (3, 1, 1), (6, 4, 1)])
def test_tangent_is_the_derivative_of_the_forces(tangent_host, nq, iters, tnormal):
    out = subprocess.run([str(tangent_host), str(nq), str(iters), str(tnormal)],
                         capture_output=True, text=True, check=True).stdout.split()
    e_fd, e_double, e_acc = map(float, out[:3])
    assert int(out[3]) == 0
    assert e_fd <= 1e-8
    assert e_double <= 1e-11
    assert e_acc <= 2.0 ** -44
