"""What hmvm_b200_apply_noalloc counts against its 16 MiB array: t and the partial
sums, each rounded up to 256 bytes, and nothing else (a mixed plan's rounded x
lies in the plan).
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import HMatrix, Plan, _lib

pytestmark = pytest.mark.gpu


def _tall_ranks(nd, ranks):
    """One 1 x 1 low-rank leaf of each rank down the diagonal: long t, short x."""
    k = len(ranks)
    r = np.array(ranks, np.int64)
    a1 = np.concatenate([[0], np.cumsum(2 * r)[:-1]])
    rows = np.arange(1, k + 1) * (nd // k)
    return HMatrix.from_arrays(nd, int(r.max()), [1] * k, r, [1] * k, [1] * k, rows, rows, a1, a1 + r,
                               np.full(int(2 * r.sum()), 0.5))


@pytest.mark.parametrize("nd,fits", [(1_000_000, True), (1_000_000, False)])
def test_mixed_plan_counts_t_and_partial_sums(gpu, nd, fits):
    import torch

    limit = _lib.HMVM_NOALLOC_SCRATCH_BYTES
    hm = _tall_ranks(nd, [1000] * (3500 if fits else 4300))
    x = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, nd)).cuda()
    y, yn = torch.zeros_like(x), torch.zeros_like(x)
    with Plan(hm, "mixed") as plan:
        t_bytes = plan.info()["t_len"] * 4
        plan.apply(x, y)
        if fits:
            assert t_bytes < limit < t_bytes + 4 * nd  # t fits, t and one rounded x would not
            plan.apply_noalloc(x, yn)
            torch.cuda.synchronize()
            assert torch.equal(y, yn)
        else:
            assert t_bytes > limit
            with pytest.raises(_lib.HMVMError) as e:
                plan.apply_noalloc(x, yn)
            assert e.value.status == _lib.HMVM_ERANGE
        plan.status()
