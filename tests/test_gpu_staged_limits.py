"""The page-locked staging of small pageable states at its limit (16,384
particles) and one above, where states go by DMA; when it grows for a larger
cloud while the upload of a smaller one may still be pending; and downloads
that leave arrays out.  Exact."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import Context, DeviceCloud, workloads as W
from demon_simulation_code_gb300._lib import addr

pytestmark = pytest.mark.gpu


def random_state(rng, n):
    return [rng.normal(size=n) for _ in range(4)]


@pytest.mark.parametrize("n", [16384, 16385])
def test_round_trips_at_the_limit(n):
    ctx = Context(0)
    rng = np.random.default_rng(n)
    c = DeviceCloud.from_cloud(ctx, W.disk_cloud(n, 2e-2, 1))
    c.step(1, 1e-4, "fp32c")
    for _ in range(2):
        s = random_state(rng, n)
        want = [a.copy() for a in s]
        c.upload(*s)
        for a in s:
            a[:] = np.nan
        for a, b in zip(c.download(), want):
            assert np.array_equal(a, b)
    c.close()


def test_growth_behind_a_pending_upload():
    torch = pytest.importorskip("torch")
    ctx = Context(0)
    rng = np.random.default_rng(5)
    sizes = (100, 5000, 16384)
    clouds = [DeviceCloud.from_cloud(ctx, W.disk_cloud(n, 2e-2, n)) for n in sizes]
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    try:
        with torch.cuda.stream(stream):
            torch.cuda._sleep(100_000_000)  # ~50 ms: the uploads below wait
        states = [random_state(rng, n) for n in sizes]
        for c, s in zip(clouds, states):
            c.upload(*s)
        for c, s in zip(clouds, states):
            for a, b in zip(c.download(), s):
                assert np.array_equal(a, b)
    finally:
        ctx.synchronize()
        ctx.reset_stream()
        for c in clouds:
            c.close()


def test_downloads_of_some_arrays():
    ctx = Context(0)
    n = 777
    c = DeviceCloud.from_cloud(ctx, W.disk_cloud(n, 2e-2, 1))
    s = random_state(np.random.default_rng(6), n)
    c.upload(*s)
    for chosen in ([0], [3], [1, 2], [0, 1, 2], []):
        out = [np.full(n, np.nan) if k in chosen else None for k in range(4)]
        assert ctx.lib.dm_cloud_download(c.h, *(None if a is None else addr(a) for a in out)) == 0
        for k in chosen:
            assert np.array_equal(out[k], s[k])
    c.close()
