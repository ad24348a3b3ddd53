"""Steps recorded by the caller's stream capture keep the buffers they were
recorded with: a kernel with a larger j split, whose partial sums need a larger
buffer, is set (and used) between the capture and its replays.  The same bits
as the same sequence of kernels and steps without a capture."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu
SMALL, LARGE = ("fp32c<8,4,256,false,cull>", 2), ("fp32c<8,4,256,false,cull>", 8)


def test_replay_after_a_larger_split(gpu_ctx):
    torch = pytest.importorskip("torch")
    c0 = W.disk_cloud(5000, 1e-2, 3)
    ctx = Context(0)
    c, ref = DeviceCloud.from_cloud(ctx, c0), DeviceCloud.from_cloud(gpu_ctx, c0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        for k in (c, ref):
            k.set_reorder_interval(1)
            k.set_kernel(*SMALL)
            k.step(1, 1e-6, "fp32c")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            c.step(1, 1e-6, "fp32c")
        for k in (c, ref):
            k.set_kernel(*LARGE)
            k.step(1, 1e-6, "fp32c")
        fill = torch.full((1 << 22,), float("nan"), device="cuda")  # memory given back would be taken again
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
        ref.set_kernel(*SMALL)
        ref.step(2, 1e-6, "fp32c")
        for a, b in zip(c.download(), ref.download()):
            assert np.array_equal(a, b)
        del fill
    finally:
        ctx.synchronize()
        ctx.reset_stream()
        c.close()
        ref.close()
