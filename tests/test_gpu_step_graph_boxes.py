"""A captured block of steps starts by forming the super group boxes that its
first pass reads, whatever was valid when it was captured: with a re-sort
interval of 0, a force evaluation right before the capture leaves those boxes
valid, and every replay after the first meets moved particles (several group
widths a block).  The same bits as single steps."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 2])
def test_blocks_after_a_force_evaluation(gpu_ctx, order):
    n = 33003
    c0 = W.disk_cloud(n, 3e-2, 5)
    rng = np.random.default_rng(6)
    c0.vx, c0.vy = rng.normal(0.0, 5.0, n), rng.normal(0.0, 5.0, n)
    runs = []
    for blocks in (True, False):
        c = DeviceCloud.from_cloud(gpu_ctx, c0)
        c.set_integrator(order)
        c.set_kernel("fp32c<4,2,128,false,cull>", 1)
        c.set_reorder_interval(0)
        c.step(1, 1e-4, "fp32c")
        c.eval_forces("fp32c")
        if blocks:
            c.step(48, 1e-4, "fp32c")
        else:
            for _ in range(48):
                c.step(1, 1e-4, "fp32c")
        runs.append(c.download())
        c.close()
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
