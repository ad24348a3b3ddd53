"""A re-sort that is due leaves a cloud alone whose order is still good (and
then only completes the next step's midpoint, if the time step changed).
With no forces the trajectory is the oracle's bit for bit whichever sorts
were skipped: velocities from far below a group's size per step (sorts
skipped) to many group sizes (every sort done), and time steps that change
between and within runs of skipped sorts."""
import numpy as np
import pytest

import oracle
from demon_simulation_code_gb300 import DeviceBatch, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu

RUNS = [(2, 1e-4), (3, 5e-5), (1, 2e-4), (18, 2e-4)]  # (steps, dt); 18: a captured block


def free_cloud(n, seed, speed):
    rng = np.random.default_rng(seed)
    x, y = W.uniform_disk(rng, n, 5e-3)
    return W.Cloud(x=x, y=y, vx=rng.normal(0.0, speed, n), vy=rng.normal(0.0, speed, n),
                   q=np.full(n, W.Q_DUST), m=np.full(n, W.M_DUST), flags=0)


def oracle_run(oracle_lib, c0):
    state = (c0.x, c0.y, c0.vx, c0.vy)
    p = oracle.make_params(**c0.params())
    for steps, dt in RUNS:
        state = oracle_lib.rk4_fixed(*state, c0.q, c0.m, p, dt, steps)[:4]
    return state


@pytest.mark.parametrize("speed", [1e-6, 5.0])
@pytest.mark.parametrize("n", [1, 33, 1025, 16384, 16385, 70001])
def test_cloud_trajectory_with_skipped_sorts(gpu_ctx, oracle_lib, n, speed):
    c0 = free_cloud(n, 40 + n, speed)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    for steps, dt in RUNS:
        c.step(steps, dt, "fp32c")
    got = c.download()
    c.close()
    for a, b in zip(got, oracle_run(oracle_lib, c0)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("speed", [1e-6, 5.0])
def test_batch_trajectory_with_skipped_sorts(gpu_ctx, oracle_lib, speed):
    clouds = [free_cloud(n, 60 + n, speed) for n in (1, 32, 33, 1000, 4096)]
    b = DeviceBatch(gpu_ctx, clouds)
    for steps, dt in RUNS:
        b.step(steps, dt)
    parts = [b.split(a) for a in b.download()]
    b.close()
    for k, c0 in enumerate(clouds):
        for comp, ref in enumerate(oracle_run(oracle_lib, c0)):
            assert np.array_equal(parts[comp][k], ref)


@pytest.mark.parametrize("n", [16384, 20000])
def test_round_trips_between_steps_keep_the_bits(gpu_ctx, n):
    """Uploading the state just downloaded changes nothing: the order, and
    with it every bit of the FP32C sums, stays that of a run without."""
    c0 = W.disk_cloud(n, 2e-2, 11)
    a, b = DeviceCloud.from_cloud(gpu_ctx, c0), DeviceCloud.from_cloud(gpu_ctx, c0)
    for c in (a, b):
        c.set_kernel("fp32c<4,2,128,false,cull>", 8)
    for _ in range(10):
        a.step(1, 1e-5, "fp32c")
        b.upload(*b.download())
        b.step(1, 1e-5, "fp32c")
    for u, v in zip(a.download(), b.download()):
        assert np.array_equal(u, v)
    a.close()
    b.close()
