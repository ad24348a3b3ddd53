"""Force parameters and the caller's stream capture.  The position sets carry
a filter bound that depends on kappa: a capture that recorded set_forces and
has not run leaves the bound of the old kappa, and a replay of steps recorded
with an old kappa brings it back.  Forces afterwards, FP64 (not re-sorted up
to 4096 particles) and FP32C, are those of a new cloud with the parameters
last set."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-13, "fp32c": 2e-6}  # the order of the sums may differ; FP32C is within 1e-6 of FP64


def same_forces(c, c0, params, prec, ctx):
    x, y, vx, vy = c.download()
    ref = DeviceCloud(ctx, x, y, vx, vy, c0.q, c0.m)
    ref.set_forces(params)
    want = ref.eval_forces(prec)
    got = c.eval_forces(prec)
    ref.close()
    scale = np.sqrt(sum((w ** 2).sum() for w in want))
    assert np.sqrt(sum(((g - w) ** 2).sum() for g, w in zip(got, want))) < TOL[prec] * scale


@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
@pytest.mark.parametrize("captured", ["set_forces", "step"])
def test_longer_screening_around_a_capture(gpu_ctx, prec, captured):
    torch = pytest.importorskip("torch")
    c0 = W.disk_cloud(500, 3e-3, 3, shielding=5e4)
    wide = dict(c0.params(), shielding=1e4)
    ctx = Context(0)
    c = DeviceCloud.from_cloud(ctx, c0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        c.step(1, 1e-6, prec)  # tuned
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            if captured == "set_forces":
                c.set_forces(wide)
            else:
                c.step(1, 1e-6, prec)
        if captured == "step":
            c.set_forces(wide)
            with torch.cuda.stream(stream):
                graph.replay()
        same_forces(c, c0, wide, prec, gpu_ctx)
    finally:
        ctx.synchronize()
        ctx.reset_stream()
        c.close()
