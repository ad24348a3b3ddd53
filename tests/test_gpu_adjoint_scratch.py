"""Forces and their vector-Jacobian product on device arrays allocate nothing,
FP64 and FP32C (the driver's count of its stream-ordered pool and the free
memory), and FP64 gives the oracle's forces at ragged sizes."""
import ctypes

import numpy as np
import pytest

import oracle
from demon_simulation_code_gb300 import workloads as W

pytestmark = pytest.mark.gpu
USED_MEM_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_single_calls_allocate_nothing(oracle_lib, prec):
    torch = pytest.importorskip("torch")
    from demon_simulation_code_gb300.adjoint import AdjointKernels

    ns = [1, 33, 700]
    clouds = [W.disk_cloud(n, 2e-3, n) for n in ns]
    K = AdjointKernels(ns, precision=prec)
    K.set_params([c.shielding for c in clouds], [c.confine for c in clouds])
    cat = [torch.tensor(np.concatenate([getattr(c, k) for c in clouds]), device="cuda")
           for k in ("x", "y", "vx", "vy", "q", "m")]
    a = [torch.rand(sum(ns), dtype=torch.float64, device="cuda") for _ in range(2)]
    K.forces(*cat), K.vjp(*cat, *a)  # torch's own buffers are there
    torch.cuda.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")
    pool, high = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
    assert cu.cuMemPoolSetAttribute(pool, USED_MEM_HIGH, ctypes.byref(high)) == 0
    free = torch.cuda.mem_get_info()[0]
    fx, fy = K.forces(*cat)
    K.vjp(*cat, *a)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_HIGH, ctypes.byref(high)) == 0
    assert high.value == 0
    off = 0
    for c in clouds:
        rx, ry = oracle_lib.forces(c.x, c.y, c.vx, c.vy, c.q, c.m, oracle.make_params(**c.params()))
        gx, gy = (f[off:off + c.n].cpu().numpy() for f in (fx, fy))
        scale = max(np.sqrt((rx ** 2 + ry ** 2).sum()), 1e-300)
        assert np.sqrt(((gx - rx) ** 2 + (gy - ry) ** 2).sum()) <= (1e-13 if prec == "fp64" else 1e-6) * scale
        off += c.n
    K.close()
