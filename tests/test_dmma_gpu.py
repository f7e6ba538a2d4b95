"""The multi-RHS kernel on the FP64 matrix instruction (hmvm_dmma_kernel) at the
edges of its tiles: blocks of 8 rows, steps of 4 columns, batches of 8 vectors,
pages of inputs, groups of 32 segments, pass widths 2 / 4 / 8 with ragged last
passes.  Against the FP64 oracle per column; the bars are those of the
single-vector kernels (FP64 1e-12, FP32 1e-5).
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import HMatrix, Plan
from helpers import oracle_hmvm, relerr

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-12, "fp32": 1e-5}
PRECISIONS = ["fp64", "fp32"]


def _apply(plan, X):
    import torch

    dt = torch.float32 if plan.dtype == np.float32 else torch.float64
    xd = torch.from_numpy(X.astype(plan.dtype)).cuda()
    yd = torch.full_like(xd, float("nan"))
    plan.apply_multi(xd, yd)
    torch.cuda.synchronize()
    plan.status()
    assert yd.dtype == dt
    return yd.cpu().numpy().astype(np.float64)


def _dense_leaves(nd, blocks, seed=0):
    """An H-matrix of dense leaves (row, column, rows, columns), 0-based."""
    rng = np.random.default_rng(seed)
    a1, rm, off = [], [], 0
    for _, _, m, n in blocks:
        a1.append(off)
        rm.append(rng.uniform(-1, 1, m * n))
        off += m * n
    b = np.array(blocks)
    k = len(blocks)
    return HMatrix.from_arrays(nd, 1, [2] * k, [0] * k, b[:, 2], b[:, 3], b[:, 0] + 1, b[:, 1] + 1, a1, [0] * k,
                               np.concatenate(rm))


@pytest.mark.parametrize("prec", PRECISIONS)
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 17, 24, 32])
def test_tile_rows_and_pass_widths(gpu, prec, rows):
    hm = HMatrix.generate(900, "cube", leaf_size=20, eta=2.0, eps=1e-6, seed=rows)
    X = np.random.default_rng(rows).uniform(-1, 1, (13, hm.nd))
    Yo = [oracle_hmvm(hm, x) for x in X]
    for nrhs_max in (2, 3, 4, 8):
        with Plan(hm, prec, nrhs_max=nrhs_max, max_tile_rows=rows) as plan:
            for nrhs in (1, 2, 3, 5, 8, 13):
                Y = _apply(plan, X[:nrhs])
                for r in range(nrhs):
                    assert relerr(Y[r], Yo[r]) <= TOL[prec], (nrhs_max, nrhs, r)


@pytest.mark.parametrize("prec", PRECISIONS)
@pytest.mark.parametrize("width", [1, 2, 3, 15, 16, 17, 63, 64, 65, 127, 128, 129, 1000])
def test_column_counts(gpu, prec, width):
    """One dense leaf of `width` columns over 29 rows: steps, batches, pages and items."""
    hm = _dense_leaves(1003, [(2, 3, 29, width)], seed=width)
    X = np.random.default_rng(width).uniform(-1, 1, (8, hm.nd))
    with Plan(hm, prec, nrhs_max=8) as plan:
        Y = _apply(plan, X)
    for r in range(8):
        yo = oracle_hmvm(hm, X[r])
        assert relerr(Y[r], yo) <= TOL[prec]
        assert np.all(Y[r][yo == 0] == 0)


@pytest.mark.parametrize("prec", PRECISIONS)
@pytest.mark.parametrize("cols", [1, 3, 4])
def test_many_segments_and_values_beside_them(gpu, prec, cols):
    """Tiles of 70 separate segments, and inputs that no leaf reads (between the
    segments, next to their padding) not finite: they must not reach y."""
    blocks = [(8 * i, 7 * j, 8, cols) for i in range(5) for j in range(70)]
    hm = _dense_leaves(500, blocks, seed=cols)
    X = np.random.default_rng(1).uniform(-1, 1, (8, hm.nd))
    used = np.zeros(hm.nd, bool)
    for j in range(70):
        used[7 * j:7 * j + cols] = True
    Yo = [oracle_hmvm(hm, x) for x in X]
    X[:, ~used] = np.nan
    X[3, ~used] = np.inf
    with Plan(hm, prec, nrhs_max=8) as plan:
        Y = _apply(plan, X)
    for r in range(8):
        assert relerr(Y[r], Yo[r]) <= TOL[prec]
