"""Lanes past a cloud's last particle (index -1) take part in the sweep's direct
chunks: the slow path for pairs on the cutoff circle must not read their
positions.  Compiled for the host with reads checked (tests/border_check.cu);
and, on the GPU, dense clouds whose sizes leave such lanes, with particles on
the cutoff circle about the origin, where those lanes sit, give the forces of
the FP64 kernel."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from demon_simulation_code_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_no_position_is_read_for_a_lane_without_a_particle(tmp_path):
    nvcc = B.nvcc()
    if not shutil.which(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "border_check")
    subprocess.run([nvcc, *B.ARCH, "-std=c++17", "-O1", "-I" + os.path.join(B.ROOT, "include"), "-I" + B.CSRC,
                    os.path.join(HERE, "border_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65, 129, 1001])
def test_particles_on_the_cutoff_circle_about_the_origin(gpu_ctx, n):
    from demon_simulation_code_gb300 import DeviceCloud, workloads as W

    c0 = W.disk_cloud(n, 3e-4, n)
    t = 2 * np.pi * np.arange(n // 2) / (n // 2)
    c0.x[: n // 2] = 5e-4 * (1 + 1e-7 * (np.arange(n // 2) % 5 - 2)) * np.cos(t)
    c0.y[: n // 2] = 5e-4 * (1 + 1e-7 * (np.arange(n // 2) % 5 - 2)) * np.sin(t)
    c = DeviceCloud.from_cloud(gpu_ctx, c0)
    want = c.eval_forces("fp64")
    scale = np.sqrt(sum((w ** 2).sum() for w in want))
    for kernel in ("fp32c<8,4,256,false,cull>", "fp32c<8,4,256,true>", "fp32c<4,2,128,false,cull>"):
        c.set_kernel(kernel, 1)
        got = c.eval_forces("fp32c")
        # FP32C forces are within 1e-6 of the FP64 sum
        assert np.sqrt(sum(((g - w) ** 2).sum() for g, w in zip(got, want))) < 1e-6 * scale
    c.close()
