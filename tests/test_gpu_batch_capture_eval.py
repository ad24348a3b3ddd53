"""A batch's force evaluation after steps that the caller's stream capture
recorded and that have not run: the group boxes they would have left are not
there (the memory may hold those of a batch that is gone, here a wider one).
Against a kernel that needs no boxes (FP32C: both within 1e-6 of the FP64
sum)."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceBatch, workloads as W

pytestmark = pytest.mark.gpu
SIZES = (700, 3000)


def pairs_only(c):
    c.flags = W.SHIELDED_COULOMB
    return c


def test_forces_before_the_first_replay():
    torch = pytest.importorskip("torch")
    ctx = Context(0)
    ctx.set_autotune(False)  # the first launch of the batch is the captured one
    gone = DeviceBatch(ctx, [W.disk_cloud(n, 0.5, n) for n in SIZES])
    gone.set_kernel("batch_fp32c<4,2,128,cull>")
    gone.step(2, 1e-5)
    gone.close()
    b = DeviceBatch(ctx, [pairs_only(W.calm_cloud(n, 4e-4 * np.sqrt(n), n)) for n in SIZES])
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        b.set_kernel("batch_fp32c<4,2,128,cull>")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            b.step(1, 1e-5)
        got = b.eval_forces()
        b.set_kernel("batch_fp32c<4,2,128>")
        want = b.eval_forces()
    finally:
        ctx.reset_stream()
        b.close()
    err = np.sqrt(sum(((g - w) ** 2).sum() for g, w in zip(got, want)) / sum((w ** 2).sum() for w in want))
    assert err < 2e-6
