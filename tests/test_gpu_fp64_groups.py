"""FP64 forces and diagnostics at the edges of their groups, tiles and size
rules (needs a GB300): 32-particle groups, the 256-particle diagnostics tile,
the size above which FP64 clouds are kept in Morton order."""
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


@pytest.mark.parametrize("radius", [3e-4, 4e-3])
@pytest.mark.parametrize("n", SIZES)
def test_diagnostics_match_plain_sums(gpu_ctx, n, radius):
    c0 = W.disk_cloud(n, radius, n + 1, confine=1e2)
    rng = np.random.default_rng(n)
    c0.vx, c0.vy = rng.normal(0, 1e-2, n), rng.normal(0, 1e-2, n)
    coulomb = 1.0 / (4.0 * np.pi * 8.8541878e-12)
    pe = 0.0
    for i in range(n - 1):
        r = np.sqrt((c0.x[i] - c0.x[i + 1:]) ** 2 + (c0.y[i] - c0.y[i + 1:]) ** 2)
        r = r[c0.shielding * r < 10.0]
        pe += np.sum(coulomb * c0.q[i] ** 2 * np.exp(-c0.shielding * r) / r)
    want = [np.sum(0.5 * c0.m * (c0.vx**2 + c0.vy**2)), pe,
            np.sum(-0.5 * c0.q * c0.confine * (c0.x**2 + c0.y**2)), np.sum(c0.m * c0.vx), np.sum(c0.m * c0.vy)]
    size = [want[0], pe, want[2], np.sum(np.abs(c0.m * c0.vx)), np.sum(np.abs(c0.m * c0.vy))]
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    got = c.diagnostics()
    # n^2 terms of one sign (momentum: of both) summed in another order: n eps
    for k in range(5):
        assert abs(got[k] - want[k]) <= max(n, 8) * 2.2e-16 * size[k], k
    c.close()
