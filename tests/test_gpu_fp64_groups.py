"""FP64 forces at the edges of their 32-particle groups and of the size above
which FP64 clouds are kept in Morton order (needs a GB300)."""
import numpy as np
import pytest

import oracle
from demon_simulation_code_gb300 import DeviceCloud
from demon_simulation_code_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 255, 256, 257, 1025, 4095, 4096, 4097]


@pytest.mark.parametrize("radius", [3e-4, 4e-3])  # every pair in reach; few
@pytest.mark.parametrize("n", SIZES)
def test_fp64_forces_match_the_oracle(gpu_ctx, oracle_lib, n, radius):
    c0 = W.disk_cloud(n, radius, n + 1, confine=1e2)
    rx, ry = oracle_lib.forces(c0.x, c0.y, c0.vx, c0.vy, c0.q, c0.m, oracle.make_params(**c0.params()))
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    fx, fy = c.eval_forces("fp64")
    # the library's FP64 force gate
    assert np.sqrt(np.sum((fx - rx) ** 2 + (fy - ry) ** 2)) <= 1e-12 * np.sqrt(np.sum(rx**2 + ry**2))
    c.close()

