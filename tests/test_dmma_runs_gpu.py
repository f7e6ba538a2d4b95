"""hmvm_dmma_kernel on long runs: many pages of inputs and several groups of 32
segments in one run, asserted from the layout, with values beside the segments
that no leaf reads not finite.  Against the FP64 oracle per column.

FP64: the bar of the single-vector kernels, 1e-12 (2-norm).  FP32: dense leaves
have FP64 products and sums of FP32 values, rounded to FP32 where a run's share
of a row is stored (one rounding), added to the others' (one each) and written;
with u = 2^-24, 8 shares of like size and roundings of rms u / sqrt(3) that is
about 1.2 u of the row; the bar is 3e-7 = 5 u, an FP32 sum of the 1,300 products
would be some 20 u off.  Low-rank leaves also round t to FP32, 50 values per row:
1e-6.
"""
import numpy as np
import pytest

from hacapk_hmvm_b200 import Batch, HMatrix, Plan, _lib
from helpers import layout_for, oracle_hmvm, relerr
from test_layout_multi import multi_view

pytestmark = pytest.mark.gpu

NSEG = 1300
PRECISIONS = [("fp64", 0), ("fp32", 1)]


def _float(hm, prec):
    return hm.to_float() if prec == "fp32" else hm


def _scattered(cols, tiles=256, rows=32):
    """`tiles` row tiles, each of NSEG dense leaves of `cols` columns with gaps of 2 between them."""
    rng = np.random.default_rng(cols)
    nd = max(tiles * rows, NSEG * (cols + 2) + 1)
    i, j = np.divmod(np.arange(tiles * NSEG), NSEG)
    k = len(i)
    a1 = np.arange(k, dtype=np.int64) * rows * cols
    a = rng.uniform(-1, 1, k * rows * cols).astype(np.float32).astype(np.float64)
    hm = HMatrix.from_arrays(nd, 1, np.full(k, 2), np.zeros(k, int), np.full(k, rows), np.full(k, cols),
                             i * rows + 1, j * (cols + 2) + 2, a1, np.zeros(k, int), a)
    used = np.zeros(nd, bool)
    for c in range(cols):
        used[np.arange(NSEG) * (cols + 2) + 1 + c] = True
    return hm, used


def _vectors(nd, nrhs, seed=0):
    return np.random.default_rng(seed).uniform(-1, 1, (nrhs, nd)).astype(np.float32).astype(np.float64)


def _device(X, prec):
    import torch

    return torch.from_numpy(X.astype(np.float32 if prec == "fp32" else np.float64)).cuda()


def _runs(hm, code, width, stage):
    """The stage's multi-RHS items on 148 SMs: (most segments, most vectors, fewest vectors of a full tile)."""
    h, v = layout_for(hm, precision=code, nrhs_max=width)
    try:
        m = multi_view(h, v)
        tiles = np.ctypeslib.as_array((_lib.TileDesc * m.n_tiles).from_address(m.tiles)).copy()
    finally:
        _lib.hmvm_lib().hmvm_b200_layout_destroy(h)
    t = tiles[:m.stage1_tiles] if stage == 1 else tiles[m.stage1_tiles:]
    return int(t["nseg"].max()), int(t["nvec"].max())


def _page_vectors(prec, width):
    return 4096 // (16 * (max(width, 4) if prec == "fp32" else width))


@pytest.mark.parametrize("cols", [1, 3])
@pytest.mark.parametrize("width", [2, 3, 8])
@pytest.mark.parametrize("prec,code", PRECISIONS)
def test_many_segments_and_pages(gpu, prec, code, width, cols):
    import torch

    hm, used = _scattered(cols)
    hf = _float(hm, prec)
    w = 2 if width == 3 and prec == "fp64" else width  # the pass that runs
    segs, vecs = _runs(hf, code, width, 2)
    assert segs > 64 and vecs > 1.4 * _page_vectors(prec, w)
    X = _vectors(hm.nd, 5)
    Yo = [oracle_hmvm(hm, x) for x in X]
    X[:, ~used] = np.nan
    X[1, ~used] = np.inf
    xd = _device(X, prec)
    with Plan(hf, prec, nrhs_max=width) as plan:
        yd = torch.full_like(xd, float("nan"))
        plan.apply_multi(xd, yd)
        plan.status()
        y1 = torch.full_like(xd[0], float("nan"))
        plan.apply(xd[0], y1)  # the same items, single-vector kernel
        plan.status()
    Y = yd.cpu().numpy().astype(np.float64)
    for r in range(5):
        assert relerr(Y[r], Yo[r]) <= (1e-12 if prec == "fp64" else 3e-7), r
    assert relerr(y1.cpu().numpy(), Yo[0]) <= (1e-12 if prec == "fp64" else 1e-5)


@pytest.mark.parametrize("prec,code", PRECISIONS)
def test_long_runs_in_a_batch(gpu, prec, code):
    """The same through the batch's kernel, whose width is a run-time value."""
    import torch

    mats, xs, yo = [], [], []
    for cols, nrhs in ((1, 8), (3, 3)):
        hm, used = _scattered(cols, tiles=128)
        X = _vectors(hm.nd, nrhs, cols)
        yo.append([oracle_hmvm(hm, x) for x in X])
        X[:, ~used] = np.nan
        mats.append(_float(hm, prec))
        xs.append(_device(X, prec))
    ys = [torch.full_like(x, float("nan")) for x in xs]
    with Batch(mats, prec, nrhs=[8, 3]) as batch:
        batch.apply(xs, ys)
        torch.cuda.synchronize()
        batch.status()
    for y, want in zip(ys, yo):
        for r, w in enumerate(want):
            assert relerr(y[r].cpu().numpy(), w) <= (1e-12 if prec == "fp64" else 3e-7), r


@pytest.mark.parametrize("width", [2, 8])
@pytest.mark.parametrize("prec,code", PRECISIONS)
def test_wide_panels(gpu, prec, code, width):
    """V panels of 8,191 columns: runs of many pages over one segment, and their partial sums."""
    import torch

    nd, k, rank, rows = 8192, 128, 33, 64
    rng = np.random.default_rng(7)
    size = rank * (rows + nd - 1)
    a1 = np.arange(k, dtype=np.int64) * size
    a = rng.uniform(-1, 1, k * size).astype(np.float32).astype(np.float64)
    hm = HMatrix.from_arrays(nd, rank, np.full(k, 1), np.full(k, rank), np.full(k, rows), np.full(k, nd - 1),
                             np.arange(k) * rows + 1, np.full(k, 2), a1, a1 + rank * (nd - 1), a)
    hf = _float(hm, prec)
    assert _runs(hf, code, width, 1)[1] > 2 * _page_vectors(prec, width)
    X = _vectors(nd, 3)
    Yo = [oracle_hmvm(hm, x) for x in X]
    X[:, 0] = np.nan  # the column that no leaf reads
    xd = _device(X, prec)
    yd = torch.full_like(xd, float("nan"))
    with Plan(hf, prec, nrhs_max=width) as plan:
        plan.apply_multi(xd, yd)
        plan.status()
    for r in range(3):
        assert relerr(yd[r].cpu().numpy(), Yo[r]) <= (1e-12 if prec == "fp64" else 1e-6), r
