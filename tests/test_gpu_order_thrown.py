"""Particles thrown far out of a sorted cloud, by the pairs swept in the steps
that follow against those of a new cloud (sorted afresh) in the same state.  A
re-sort interval that the caller set is kept: interval 1 sorts every step, also
where the default would leave the order (two particles thrown)."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceBatch, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu
DT = 1e-6


def throwing_cloud(n, thrown, seed):
    """A disk at disk16k's density; `thrown` of its particles move a metre a step."""
    c = W.disk_cloud(n, 2e-2 * np.sqrt(n / 16384), seed)
    rng = np.random.default_rng(seed + 1)
    i = rng.choice(n, thrown, replace=False)
    t = rng.uniform(0, 2 * np.pi, thrown)
    c.vx[i], c.vy[i] = 1e6 * np.cos(t), 1e6 * np.sin(t)
    return c


def at(c0, state):
    c = c0.copy()
    c.x, c.y, c.vx, c.vy = state
    return c


def swept(obj, *step):
    e = obj.evaluated_pairs()
    obj.step(*step)
    return obj.evaluated_pairs() - e


@pytest.mark.parametrize("n", [16384, 20000])
def test_interval_one_sorts_every_step(gpu_ctx, n):
    c0 = throwing_cloud(n, 2, 6)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    c.set_kernel("fp32c<4,2,128,false,cull>", 4)
    c.set_reorder_interval(1)
    c.step(1, DT, "fp32c")
    for _ in range(5):
        new = DeviceCloud.from_cloud(gpu_ctx, at(c0, c.download()))
        new.set_kernel("fp32c<4,2,128,false,cull>", 4)
        # particles that share a key may lie in either order
        assert swept(c, 1, DT, "fp32c") < 1.01 * swept(new, 1, DT, "fp32c")
        new.close()
    c.close()


@pytest.mark.parametrize("thrown", [20, 50, 400])
@pytest.mark.parametrize("n", [16384, 20000])
def test_cloud(gpu_ctx, n, thrown):
    c0 = throwing_cloud(n, thrown, 3)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    c.set_kernel("fp32c<4,2,128,false,cull>", 4)
    c.step(1, DT, "fp32c")
    for _ in range(5):
        new = DeviceCloud.from_cloud(gpu_ctx, at(c0, c.download()))
        new.set_kernel("fp32c<4,2,128,false,cull>", 4)
        assert swept(c, 1, DT, "fp32c") < 1.3 * swept(new, 1, DT, "fp32c")
        new.close()
    c.close()


@pytest.mark.parametrize("thrown", [6, 20, 100])
def test_batch(gpu_ctx, thrown):
    clouds = [throwing_cloud(4096, thrown, s) for s in (4, 5)]
    b = DeviceBatch(gpu_ctx, clouds)
    b.set_kernel("batch_fp32c<4,2,128,cull>")
    b.step(1, DT)
    for _ in range(5):
        parts = [b.split(a) for a in b.download()]
        new = DeviceBatch(gpu_ctx, [at(c, [p[k] for p in parts]) for k, c in enumerate(clouds)])
        new.set_kernel("batch_fp32c<4,2,128,cull>")
        assert swept(b, 1, DT) < 1.3 * swept(new, 1, DT)
        new.close()
    b.close()
