"""Re-sorts of both precisions where they do sort (FP32C at every size, FP64
above 4096 particles): with no forces the trajectory is the oracle's bit for
bit; forces come back in the caller's order after steps that permuted the
cloud; and the interval at which the cloud is sorted changes results only by
the rounding of sums in another order (FP64 as gated for unsorted clouds, 1e-13;
FP32C forces are within 1e-6 of FP64, and a calm cloud's velocities over 40
steps follow them with no more than a tenfold growth)."""
import numpy as np
import pytest

import oracle
from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "fp32c": 1e-6}  # of the forces against the oracle


def calm(n, seed):
    return W.calm_cloud(n, 4e-4 * np.sqrt(n), seed)


@pytest.mark.parametrize("prec,n", [("fp32c", n) for n in (1, 2, 31, 33, 700, 2047, 2049, 16383, 16384, 16385)]
                         + [("fp64", n) for n in (4097, 5000)])
def test_resort_every_step_is_a_permutation(gpu_ctx, oracle_lib, prec, n):
    rng = np.random.default_rng(100 + n)
    x, y = W.uniform_disk(rng, n, 5e-3)
    c0 = W.Cloud(x=x, y=y, vx=rng.normal(0.0, 1e-1, n), vy=rng.normal(0.0, 1e-1, n), q=np.full(n, W.Q_DUST),
                 m=np.full(n, W.M_DUST), flags=0)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    c.set_reorder_interval(1)
    c.step(3, 1e-4, prec)
    p = oracle.make_params(**c0.params())
    for a, b in zip(c.download(), oracle_lib.rk4_fixed(c0.x, c0.y, c0.vx, c0.vy, c0.q, c0.m, p, 1e-4, 3)):
        assert np.array_equal(a, b)
    c.close()


@pytest.mark.parametrize("steps_in,n", [("fp32c", 700), ("fp64", 5000)])
@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
def test_forces_after_a_resort_are_in_caller_order(gpu_ctx, oracle_lib, steps_in, n, prec):
    c0 = calm(n, 3)
    c0.q = c0.q * np.linspace(0.5, 1.5, n)  # charges and masses move with their particles
    c0.m = c0.m * np.linspace(1.5, 0.5, n)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    c.step(3, 1e-4, steps_in)
    x, y, vx, vy = c.download()
    rx, ry = oracle_lib.forces(x, y, vx, vy, c0.q, c0.m, oracle.make_params(**c0.params()))
    for _ in range(2):
        fx, fy = c.eval_forces(prec)
        assert np.sqrt(((fx - rx) ** 2 + (fy - ry) ** 2).sum() / (rx ** 2 + ry ** 2).sum()) <= TOL[prec]
        c.upload(x, y, vx, vy)
    c.close()


@pytest.mark.parametrize("prec,n,tol", [("fp64", 4500, 1e-13), ("fp32c", 512, 1e-5), ("fp32c", 4500, 1e-5)])
def test_intervals_change_results_by_rounding_alone(gpu_ctx, prec, n, tol):
    c0 = calm(n, 4)
    outs = []
    for interval in (None, 0, 1, 4, 16):
        c = DeviceCloud.from_cloud(gpu_ctx, c0)
        if interval is not None:
            c.set_reorder_interval(interval)
        c.step(40, 1e-4, prec)
        outs.append(c.download())
        c.close()
    for o in outs[1:]:
        for a, b in zip(o, outs[0]):
            assert np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()) < tol
