"""What a request takes from the device's memory pool (the pool's own count, before
and after) is what its handle reports, and stays below the estimate that admits
it, for two to six thickness points and both precisions."""
import ctypes
import dataclasses

import pytest

from biofem import configs

pytestmark = pytest.mark.gpu

USED_CURRENT = 7          # cudaMemPoolAttrUsedMemCurrent


def pool_used():
    import torch
    rt = next(lib for lib in map(_load, ("libcudart.so.13", "libcudart.so.12")) if lib)
    torch.cuda.synchronize()
    pool, used = ctypes.c_void_p(), ctypes.c_uint64()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert rt.cudaMemPoolGetAttribute(pool, USED_CURRENT, ctypes.byref(used)) == 0
    return used.value


def _load(name):
    try:
        return ctypes.CDLL(name)
    except OSError:
        return None


@pytest.mark.parametrize("q", [2, 3, 6])
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32_bulk"])
def test_estimate_covers_what_the_pool_gives(q, precision):
    import torch
    from biofem.gpu import GpuShell, MeshInfo, estimate_bytes
    torch.cuda.init()
    for nx, ny in ((16, 12), (96, 72), (150, 112)):
        w = configs.Workload("sheet", nx, ny, n_qp=q, z_sigma=1e-3, z_smooth=True, basis=int(q > 5), tnormal=int(q > 5))
        m = w.build_mesh()
        before = pool_used()
        sh = GpuShell(m, w, configs.MU, configs.BULK, configs.H0, precision=precision)
        sh.newton(w.initial_x(m, sh.topology()["xyz0_full"]), max_newton=1, gmres_max_it=5)
        taken = pool_used() - before
        info = MeshInfo()
        assert sh.lib.GetGpuMeshInfo(sh.handle, ctypes.byref(info)) == 0
        sh.close()
        assert taken == info.device_bytes
        assert taken <= estimate_bytes(m.n_v, m.n_elmt, m.n_ghosts, precision)
