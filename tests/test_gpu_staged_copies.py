"""States of small clouds in pageable memory cross through one page-locked
staging area of the context: back-to-back uploads of two clouds, sources
changed right after each call, and partial downloads, at the limit and around
it.  Exact."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 4096, 4097])
def test_uploads_and_downloads_share_the_staging(gpu_ctx, n):
    rng = np.random.default_rng(n)
    clouds = [DeviceCloud.from_cloud(gpu_ctx, W.disk_cloud(n, 2e-2, s)) for s in (1, 2)]
    clouds[0].step(1, 1e-4, "fp32c")  # an internal order of its own
    for _ in range(3):
        states = []
        for c in clouds:
            s = [rng.normal(size=n) for _ in range(4)]
            states.append([a.copy() for a in s])
            c.upload(*s)
            for a in s:
                a[:] = np.nan
        for c, want in zip(clouds, states):
            for a, b in zip(c.download(), want):
                assert np.array_equal(a, b)
    for c in clouds:
        c.close()
