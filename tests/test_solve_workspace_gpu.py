"""The solvers' work vectors stay with the plan: whatever was solved on a plan
before -- the other solver, a longer restart that made the workspace grow, one
too large to be kept -- a solve gives, bit for bit, what it gives on a new plan.
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import HMatrix, Plan

pytestmark = pytest.mark.gpu


def _blocks(nd, block=32, seed=0):
    """Diagonal blocks, each near the identity: both solvers converge in a few steps."""
    rng = np.random.default_rng(seed)
    n = nd // block
    a = 0.02 * rng.uniform(-1, 1, (n, block, block)) + np.eye(block)
    first = np.arange(n) * block + 1
    a1 = np.arange(n, dtype=np.int64) * block * block
    return HMatrix.from_arrays(nd, 1, [2] * n, [0] * n, [block] * n, [block] * n, first, first, a1, [0] * n, a.ravel())


def _solve(plan, b, solver, restart, max_steps):
    import torch

    u = torch.zeros_like(b)
    if solver == "bicgstab":
        steps, rel = plan.bicgstab(b, u, eps=1e-10, max_steps=max_steps)
    else:
        steps, rel = plan.gcrm(b, u, eps=1e-10, max_steps=max_steps, restart=restart)
    return u.cpu(), steps, rel


SEQUENCE = [("bicgstab", 0, 100), ("gcrm", 3, 100), ("bicgstab", 0, 1), ("gcrm", 40, 100), ("bicgstab", 0, 100),
            ("gcrm", 2, 5), ("bicgstab", 0, 0), ("gcrm", 40, 100)]


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
def test_solves_in_turn(gpu, prec):
    import torch

    hm = _blocks(4000 // 32 * 32)
    dt = torch.float32 if prec == "fp32" else torch.float64
    rhs = [torch.from_numpy(np.random.default_rng(i).uniform(-1, 1, hm.nd)).to(dt).cuda() for i in range(2)]
    with Plan(hm, prec) as plan:
        for i, case in enumerate(SEQUENCE):
            b = rhs[i % 2]
            with Plan(hm, prec) as fresh:
                want = _solve(fresh, b, *case)
            got = _solve(plan, b, *case)
            assert torch.equal(got[0], want[0]) and got[1:] == want[1:], (i, case)


def test_workspace_too_large_to_keep(gpu):
    """130 vectors of N = 70,016 take 73 MB: allocated for the call and given back."""
    import torch

    hm = _blocks(70016)
    b = torch.from_numpy(np.random.default_rng(5).uniform(-1, 1, hm.nd)).cuda()
    with Plan(hm, "fp64") as plan:
        first = _solve(plan, b, "bicgstab", 0, 100)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        large = _solve(plan, b, "gcrm", 64, 100)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free
        again = _solve(plan, b, "bicgstab", 0, 100)
        assert torch.equal(first[0], again[0]) and first[1:] == again[1:]
    with Plan(hm, "fp64") as fresh:
        want = _solve(fresh, b, "gcrm", 64, 100)
    assert torch.equal(large[0], want[0]) and large[1:] == want[1:]
    assert large[2] < 1e-10
