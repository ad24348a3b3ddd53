"""Steps recorded by the caller's own stream capture and replayed: between
replays the state may be uploaded, stepped with another time step or by
another integrator's parity, and the host library cannot know.  With no pair
force the trajectory is the same bits as without a capture, FP64 and FP32C,
RK4 and RK2 (one step: its slots and position sets change places)."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceBatch, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


def free_cloud(n, seed):
    rng = np.random.default_rng(seed)
    x, y = W.uniform_disk(rng, n, 5e-3)
    return W.Cloud(x=x, y=y, vx=rng.normal(0.0, 1e-3, n), vy=rng.normal(0.0, 1e-3, n),
                   q=np.full(n, W.Q_DUST), m=np.full(n, W.M_DUST), flags=W.CONFINEMENT | W.DRAG, heat=0.0)


@pytest.mark.parametrize("order", [4, 2])
@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
@pytest.mark.parametrize("steps", [1, 2, 17])
def test_replayed_steps(order, prec, steps):
    torch = pytest.importorskip("torch")
    c0 = free_cloud(500, 3)
    ctx, ref_ctx = Context(0), Context(0)
    c, ref = DeviceCloud.from_cloud(ctx, c0), DeviceCloud.from_cloud(ref_ctx, c0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    for k in (c, ref):
        k.set_integrator(order)
        k.step(1, 1e-4, prec)  # tuned
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        c.step(steps, 2e-5, prec)

    def replay(times):
        with torch.cuda.stream(stream):
            for _ in range(times):
                graph.replay()
        ref.step(times * steps, 2e-5, prec)

    c.step(1, 1e-4, prec)  # directly after a capture that did not run
    ref.step(1, 1e-4, prec)
    replay(3)
    c.step(1, 2e-5, prec)
    ref.step(1, 2e-5, prec)
    replay(1)
    c.step(1, 1e-4, prec)  # an odd number of steps between: RK2's slots and sets
    ref.step(1, 1e-4, prec)
    replay(2)
    s = free_cloud(500, 4)
    for k in (c, ref):
        k.upload(s.x, s.y, s.vx, s.vy)
    replay(2)
    c.step(3, 1e-4, prec)
    ref.step(3, 1e-4, prec)
    got, want = c.download(), ref.download()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert c.get_step_counter() == ref.get_step_counter()
    ctx.reset_stream()
    c.close()
    ref.close()


@pytest.mark.parametrize("order", [4, 2])
def test_replayed_batch_steps(order):
    torch = pytest.importorskip("torch")
    clouds = [free_cloud(n, 10 + n) for n in (1, 33, 700)]
    ctx, ref_ctx = Context(0), Context(0)
    b, ref = DeviceBatch(ctx, clouds), DeviceBatch(ref_ctx, clouds)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    for k in (b, ref):
        k.set_integrator(order)
        k.step(1, 1e-4)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        b.step(1, 2e-5)
    b.step(1, 1e-4)
    ref.step(1, 1e-4)
    with torch.cuda.stream(stream):
        for _ in range(3):
            graph.replay()
    ref.step(3, 2e-5)
    b.step(1, 1e-4)
    ref.step(1, 1e-4)
    for u, v in zip(b.download(), ref.download()):
        assert np.array_equal(u, v)
    ctx.reset_stream()
    b.close()
    ref.close()
