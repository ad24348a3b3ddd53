"""Clouds of 32,768 particles and more skip 32 groups at a time by the boxes of
super groups: forces of the culling kernels against a kernel that tests every
pair (FP32C: both within 1e-6 of the FP64 sum, so 2e-6 of each other; FP64: the
culled kernel against FP32C, 1e-6), with a partial last group and super group,
at the start and after steps (boxes left by the epilogue)."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import DeviceCloud, workloads as W

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.sqrt(sum(((u - v) ** 2).sum() for u, v in zip(a, b)) / sum((v ** 2).sum() for v in b))


@pytest.mark.parametrize("n", [32767, 32768, 33003])
def test_super_group_boxes_keep_every_pair(gpu_ctx, n):
    c = DeviceCloud.from_cloud(gpu_ctx, W.disk_cloud(n, 3e-2, 5))
    for steps in (0, 2):
        c.set_kernel("fp32c<4,2,128,false,cull>", 1)
        c.step(steps, 1e-6, "fp32c")
        got = [c.eval_forces("fp32c")]
        for kernel, split in (("fp32c<4,2,128,false,cull>", 4), ("fp32c<8,4,256,true,cull>", 2)):
            c.set_kernel(kernel, split)
            got.append(c.eval_forces("fp32c"))
        c.set_kernel("fp32c<8,4,256,false>", 8)
        every = c.eval_forces("fp32c")
        for f in got:
            assert rel(f, every) < 2e-6
        c.set_kernel("fp64<4,near>", 1)
        assert rel(every, c.eval_forces("fp64")) < 1e-6
    c.close()
