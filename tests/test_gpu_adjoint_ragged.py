"""Fused rollout step and its adjoint at cloud sizes that end inside a warp,
inside a block or inside a staged tile: the FP32C kernels against the FP64
ones (needs a GB300)."""
import numpy as np
import pytest

from demon_simulation_code_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

DT = 1e-4
# FP32C pair sums are within 1e-6 of the FP64 ones norm-wise (the library's
# force gate); a step is linear in them, and its adjoint evaluates the same
# pairs with one more derivative: ten times that
FORCE_TOL, ADJOINT_TOL = 1e-6, 1e-5


def rel(a, b):
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


@pytest.mark.parametrize("kappa", [5e3, 2e4])  # nearly all pairs in reach; few
@pytest.mark.parametrize("ns", [[1, 2, 31], [33, 64, 65], [127, 129, 255], [257, 5, 300]])
def test_fp32c_step_and_adjoint_match_fp64(ns, kappa):
    from demon_simulation_code_gb300.adjoint import AdjointKernels

    rng = np.random.default_rng(sum(ns))
    xy = [W.uniform_disk_minsep(rng, n, 1.2e-3, 5e-5) for n in ns]
    total = sum(ns)
    cuda = dict(dtype=torch.float64, device="cuda")
    start = [torch.tensor(np.concatenate([p[k] for p in xy]), **cuda) for k in (0, 1)]
    start += [torch.tensor(rng.normal(0, 1e-4, total), **cuda) for _ in range(2)]
    q, m = torch.full((total,), W.Q_DUST, **cuda), torch.full((total,), W.M_DUST, **cuda)
    lam0 = [torch.tensor(rng.normal(0, 1, total), **cuda) for _ in range(4)]
    out = {}
    for prec in ("fp64", "fp32c"):
        K = AdjointKernels(ns, flags=W.SHIELDED_COULOMB, precision=prec)
        K.set_params(np.full(len(ns), kappa), np.zeros(len(ns)))
        s = tuple(v.clone() for v in start)
        stages = torch.empty((16, total), **cuda)
        K.rk4_step(s, q, m, DT, stages=stages)
        if prec == "fp64":
            kept = stages.clone()  # both adjoints from the same stage inputs
        lam = tuple(v.clone() for v in lam0)
        g = [torch.zeros(total, **cuda) for _ in range(3)]
        K.rk4_step_vjp(kept, q, m, DT, lam, *g)
        torch.cuda.synchronize()
        out[prec] = ([a - b for a, b in zip(s, start)], [a - b for a, b in zip(lam, lam0)], g[:2])
    moved, lam, g = zip(*(out[p] for p in ("fp32c", "fp64")))
    for k in (2, 3):  # velocity increments: the pair force alone
        assert rel(moved[0][k], moved[1][k]) <= FORCE_TOL
    for k in range(4):
        assert rel(lam[0][k], lam[1][k]) <= ADJOINT_TOL
    for k in range(2):
        assert rel(g[0][k], g[1][k]) <= ADJOINT_TOL
