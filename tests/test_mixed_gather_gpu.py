"""Inputs of the mixed single-vector kernel: segments of x that start at every
residue of a 16-byte group, of every short length, with values beside them that
no leaf reads not finite (they must not reach y); more than one FP64 segment per
tile.  Against the FP64 oracle with the mixed bar (1e-4 relative 2-norm error).
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import HMatrix, Plan
from helpers import oracle_hmvm, relerr

pytestmark = pytest.mark.gpu


def _apply(plan, x):
    import torch

    xd = torch.from_numpy(x).cuda()
    yd = torch.full_like(xd, float("nan"))
    plan.apply(xd, yd)
    torch.cuda.synchronize()
    plan.status()
    return yd.cpu().numpy()


def _leaves(nd, dense, lowrank, seed):
    """dense: (row, column, rows, columns); lowrank: the same and the rank, 0-based."""
    rng = np.random.default_rng(seed)
    lt, kt, ndl, ndt, sl, st, a1, a2, rm, off = [], [], [], [], [], [], [], [], [], 0
    for r, c, m, n, *k in list(dense) + list(lowrank):
        lt.append(1 if k else 2)
        kt.append(k[0] if k else 0)
        ndl.append(m), ndt.append(n), sl.append(r + 1), st.append(c + 1), a1.append(off)
        first = k[0] * n if k else m * n
        a2.append(off + first if k else 0)
        total = first + (k[0] * m if k else 0)
        rm.append(rng.uniform(-1, 1, total))
        off += total
    return HMatrix.from_arrays(nd, max(kt + [1]), lt, kt, ndl, ndt, sl, st, a1, a2, np.concatenate(rm))


@pytest.mark.parametrize("fmt", ["fp16", "bf16"])
@pytest.mark.parametrize("cols", [1, 2, 3, 4, 5, 9])
def test_segment_starts_and_lengths(gpu, fmt, cols):
    step = cols + 2  # every residue of the start, a gap before the next segment
    starts = [step * j + 1 for j in range(28)]
    dense = [(16 * i, c, 16, cols) for i in range(3) for c in starts]
    lowrank = [(64 + 8 * j, c, 8, cols, 3) for j, c in enumerate(starts)]
    hm = _leaves(400, dense, lowrank, cols)
    x = np.random.default_rng(cols).uniform(-1, 1, hm.nd)
    yo = oracle_hmvm(hm, x)
    used = np.zeros(hm.nd, bool)
    for c in starts:
        used[c:c + cols] = True
    x[~used] = np.nan
    with Plan(hm, "mixed", mixed_lr_format=fmt) as plan:
        y = _apply(plan, x)
    assert relerr(y, yo) <= 1e-4


@pytest.mark.parametrize("width", [4, 7, 8, 33, 511, 512, 513])
def test_wide_panels_and_diagonal_blocks(gpu, width):
    """V panels wider than an input buffer from an odd column, FP64 diagonal blocks beside FP32 and t segments."""
    nd = 1200
    dense = [(8 * i, 8 * i, 8, 8) for i in range(12)] + [(0, 300 + 11 * j, 8, 5) for j in range(9)]
    lowrank = [(8 * i, 601, 8, width, 5) for i in range(12)]
    hm = _leaves(nd, dense, lowrank, width)
    x = np.random.default_rng(width).uniform(-1, 1, nd)
    yo = oracle_hmvm(hm, x)
    with Plan(hm, "mixed") as plan:
        assert relerr(_apply(plan, x), yo) <= 1e-4
