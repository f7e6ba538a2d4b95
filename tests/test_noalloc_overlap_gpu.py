"""hmvm_b200_apply_noalloc beside hmvm_b200_apply and replay of the same plan on
another stream: the two calls share no buffer, so each gives, bit for bit, what
it gives alone.  (Calls of apply_noalloc among themselves share the library's
array and are ordered here.)
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import HMatrix, Plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("replayed", [False, True], ids=["apply", "replay"])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
def test_overlapping_calls_keep_their_inputs(gpu, prec, replayed):
    import torch

    hm = HMatrix.generate(20000, "sphere", eps=1e-4, seed=4)
    dt = torch.float32 if prec == "fp32" else torch.float64
    x = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, (2, hm.nd))).to(dt).cuda()
    with Plan(hm, prec) as plan:
        alone = torch.empty_like(x)
        for i in range(2):
            plan.apply(x[i], alone[i])
        y = torch.full_like(x, float("nan"))
        plan.apply_noalloc(x[1], y[1])
        torch.cuda.synchronize()
        assert torch.equal(y[1], alone[1])
        if replayed:
            plan.capture(x[0], y[0])
        s = [torch.cuda.Stream(), torch.cuda.Stream()]
        for _ in range(20):
            y.fill_(float("nan"))
            torch.cuda.synchronize()
            for _ in range(10):
                if replayed:
                    plan.replay(stream=s[0])
                else:
                    plan.apply(x[0], y[0], stream=s[0])
                plan.apply_noalloc(x[1], y[1], stream=s[1])
            torch.cuda.synchronize()
            assert torch.equal(y, alone)
        plan.status()
