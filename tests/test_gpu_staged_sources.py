"""Uploads of small states read their sources when the stream gets there, if a
source is memory that work queued on the stream may still write: one
page-locked array among pageable ones, filled by a copy still in flight."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", range(4))
def test_a_page_locked_source_still_being_written(which):
    torch = pytest.importorskip("torch")
    n = 1000
    ctx = Context(0)
    c = DeviceCloud.from_cloud(ctx, W.disk_cloud(n, 5e-3, 1))
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        rng = np.random.default_rng(2)
        state = [rng.normal(size=n) for _ in range(4)]
        c.upload(*state)  # the staging area is there
        want = rng.normal(size=n)
        src = torch.tensor(want, device="cuda")
        pinned = torch.zeros(n, dtype=torch.float64, pin_memory=True)
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(200_000_000)  # ~0.1 s
            pinned.copy_(src, non_blocking=True)
        state[which] = pinned.numpy()
        c.upload(*state)
        got = c.download()
        for k in range(4):
            assert np.array_equal(got[k], want if k == which else state[k])
    finally:
        ctx.synchronize()
        ctx.reset_stream()
        c.close()
