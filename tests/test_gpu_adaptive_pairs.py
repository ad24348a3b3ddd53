"""The adaptive time step's distance test over exactly the reference's pairs
(Integrator.cpp:87-129) at sizes around the kernel's 32-block tiles, in the
caller's order whatever order the device keeps, with the closest pair planted
in turn in the first, the last and a diagonal block.  FP32, the same
operations: exact."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu

DIAGONAL = [(0, 1), (2, 3), (0, 3), (1, 2), (1, 3), (0, 2)]


def checked_min(x, y):
    fx, fy = x.astype(np.float32).reshape(-1, 4), y.astype(np.float32).reshape(-1, 4)
    best = np.float32(np.inf)
    for a, b in DIAGONAL:
        sx, sy = fx[:, a] - fx[:, b], fy[:, a] - fy[:, b]
        best = min(best, (sx * sx + sy * sy).min())
    nb = len(fx)
    o, p = np.triu_indices(nb, 1)
    for k in range(4):
        for d in range(3):
            m = (k - d) % 4
            if len(o):
                sx, sy = fx[o, k] - fx[p, m], fy[o, k] - fy[p, m]
                best = min(best, (sx * sx + sy * sy).min())
    return np.sqrt(best)


@pytest.mark.parametrize("n", [4, 8, 124, 128, 132, 256, 260, 1540])
def test_checked_pairs_minimum(gpu_ctx, n):
    rng = np.random.default_rng(n)
    for plant in ((0, 1), (n - 2, n - 1), (0, n - 1), (1, n - 4), (n // 2, n - 1), (3, n - 4)):
        c0 = W.disk_cloud(n, 2e-2, n)
        x, y = c0.x.copy(), c0.y.copy()
        i, j = plant
        if i != j:
            x[j], y[j] = x[i] + 3e-6, y[i] - 1e-6
        c = DeviceCloud.from_cloud(gpu_ctx, c0)
        c.eval_forces("fp32c")  # the device's own order
        c.upload(x, y, c0.vx, c0.vy)
        dmin, dt = c.modify_timestep(1e-4)
        want = checked_min(x, y)
        assert np.float32(dmin) == want
        dist, dt_want = np.float32(1e-4), 1e-4
        while want <= dist:
            dist, dt_want = np.float32(dist / np.float32(10.0)), dt_want / 10.0
        assert dt == dt_want
        c.close()
