"""When a cloud is re-sorted depends on its state and on the steps since the
last sort, not on how many steps the object has taken: the same upload and the
same steps give the same bits however often they are repeated, and a block of
steps the same bits as single ones (FP32C, and FP64 above the size up to which
it is not sorted).  The clouds are jittered lattices: no two particles share a
sort key, so a sort's result does not depend on the order before it."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


def lattice_cloud(n, seed):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(np.sqrt(n)))
    i, j = np.divmod(rng.permutation(m * m)[:n], m)
    c = W.disk_cloud(n, 1e-2, seed)
    c.x = 3e-4 * (i - m / 2 + rng.uniform(-0.1, 0.1, n))
    c.y = 3e-4 * (j - m / 2 + rng.uniform(-0.1, 0.1, n))
    # slow enough that orders are kept, fast enough that a sort would change them
    c.vx, c.vy = rng.normal(0.0, 0.1, n), rng.normal(0.0, 0.1, n)
    return c


SIZES = [("fp32c", 4096), ("fp32c", 16384), ("fp32c", 20000), ("fp64", 5000)]


@pytest.mark.parametrize("prec,n", SIZES)
def test_repeated_intervals(gpu_ctx, prec, n):
    c0 = lattice_cloud(n, 7)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    first = None
    for _ in range(6):
        c.upload(c0.x, c0.y, c0.vx, c0.vy)
        c.step(3, 1e-4, prec)
        got = c.download()
        first = first or got
        for a, b in zip(got, first):
            assert np.array_equal(a, b)
    c.close()


@pytest.mark.parametrize("prec,n", SIZES)
def test_blocks_and_single_steps(gpu_ctx, prec, n):
    c0 = lattice_cloud(n, 8)
    runs = []
    for steps in ([40], [1] * 40, [3, 17, 20]):
        c = DeviceCloud.from_cloud(gpu_ctx, c0)
        for s in steps:
            c.step(s, 1e-4, prec)
        runs.append(c.download())
        c.close()
    for r in runs[1:]:
        for a, b in zip(r, runs[0]):
            assert np.array_equal(a, b)
