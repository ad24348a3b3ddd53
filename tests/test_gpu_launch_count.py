"""The launch count of a replayed block of 16 steps is that of 16 single steps,
also where blocks of one cloud at two precisions, and of two batches of
different integrators, take turns."""
import pytest

from demon_simulation_code_gb300 import Context, DeviceBatch, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


def test_blocks_in_turn():
    ctx = Context(0)
    c = DeviceCloud.from_cloud(ctx, W.calm_cloud(512, 1e-2, 1))
    clouds = [W.calm_cloud(n, 1e-2, n) for n in (100, 512)]
    rk4, rk2 = DeviceBatch(ctx, clouds), DeviceBatch(ctx, clouds)
    rk2.set_integrator(2)
    steps = [lambda n: c.step(n, 1e-5, "fp32c"), lambda n: c.step(n, 1e-5, "fp64"),
             lambda n: rk4.step(n, 1e-5), lambda n: rk2.step(n, 1e-5)]
    c.autotune("fp64")
    for f in steps:  # sorted, and at a multiple of 16 steps, where blocks begin
        for _ in range(16):
            f(1)

    def counted(f, calls):
        n = ctx.launch_count()
        for k in calls:
            f(k)
        return ctx.launch_count() - n

    single = [counted(f, [1] * 16) for f in steps]
    assert len(set(single)) > 1
    for _ in range(3):
        assert [counted(f, [16]) for f in steps] == single
    for o in (c, rk4, rk2):
        o.close()
