"""The items that the multi-RHS kernel of FP64 and FP32 plans runs (runs of the
consecutive parts of a tile, their segments, team ranges and reductions), on the
CPU: walked like the kernel walks them they reproduce the oracle, every index
stays inside its buffer, and hmvm_b200_layout_validate rejects a set with one
entry changed.  Few SMs give long runs and tiles that several teams share, many
give one part per run."""
import ctypes as C
import os
import subprocess
from types import SimpleNamespace

import numpy as np
import pytest
from hypothesis import HealthCheck, given, settings

from hacapk_hmvm_b200 import HMatrix, _lib
from helpers import ROOT, emulate_layout, layout_for, oracle_hmvm
from layout_checks import check_layout_bounds
from test_layout_random import _abs_bound, leaf_tables


def multi_view(h, v):
    """The layout's view with the multi-RHS items in the place of its own."""
    m = _lib.LayoutMultiView()
    _lib.check(_lib.hmvm_lib().hmvm_b200_layout_multi_view(h, C.byref(m)), "multi view")
    fields = {f: getattr(v, f) for f, _ in v._fields_}
    fields.update({f: getattr(m, f) for f, _ in m._fields_ if f != "_pad0"})
    return SimpleNamespace(**fields)


def _arrays(m):
    return (np.ctypeslib.as_array((_lib.TileDesc * m.n_tiles).from_address(m.tiles)),
            np.ctypeslib.as_array((_lib.SegDesc * m.n_segs).from_address(m.segs)),
            np.ctypeslib.as_array(m.seg_first, (m.n_segs,)))


def _validate(h):
    rc = _lib.hmvm_lib().hmvm_b200_layout_validate(h)
    return rc, _lib.hmvm_lib().hmvm_b200_last_error().decode(errors="replace")


def _check(hm, x, prec, tol, **opts):
    h, v = layout_for(hm, precision=prec, **opts)
    try:
        rc, msg = _validate(h)
        assert rc == _lib.HMVM_OK, (opts, msg)
        m = multi_view(h, v)
        if m.n_segs:
            check_layout_bounds(m)
            y = emulate_layout(m, x)
            yo, bound = oracle_hmvm(hm, x), tol * _abs_bound(hm, x)
            assert np.all(np.abs(y - yo) <= bound), opts
            tiles, segs, first = _arrays(m)
            for td in tiles:
                s0, s1 = int(td["seg_begin"]), int(td["seg_begin"]) + int(td["nseg"])
                padded = -(-segs["ncols"][s0:s1] // v.vec) * v.vec
                assert np.array_equal(first[s0:s1], np.cumsum(padded) - padded)
        return m, h, v
    finally:
        _lib.hmvm_lib().hmvm_b200_layout_destroy(h)


OPTS = [dict(nrhs_max=8), dict(nrhs_max=2, num_sms=1), dict(nrhs_max=3, num_sms=2, max_tile_rows=5),
        dict(nrhs_max=8, num_sms=3, split_cols=4), dict(nrhs_max=8, num_sms=1, kernel=0)]


@settings(max_examples=30, deadline=None, derandomize=True, suppress_health_check=[HealthCheck.too_slow])
@given(leaf_tables())
def test_random_tables(table):
    hm, x = table
    for opts in OPTS:
        _check(hm, x, 0, 1e-13, **opts)
    _check(hm.to_float(), x, 1, 1e-5, **OPTS[1])


@pytest.mark.parametrize("prec,tol", [(0, 1e-13), (1, 1e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("num_sms", [1, 3, 20, 148])
def test_generated(prec, tol, num_sms):
    hm = HMatrix.generate(3000, "sphere", eta=2.0, eps=1e-5, leaf_size=24, seed=9)
    hm = hm.to_float() if prec else hm
    x = np.random.default_rng(1).uniform(-1, 1, hm.nd)
    for width in (2, 4, 8):
        m, _, _ = _check(hm, x, prec, tol, nrhs_max=width, num_sms=num_sms)
        assert m.n_tiles > 0 and m.n_red2 > 0  # some tile is shared by two teams


def test_other_layouts_have_none():
    hm = HMatrix.generate(500, "cube", seed=2)
    for opts in (dict(precision=0), dict(precision=2, nrhs_max=8), dict(precision=1, nrhs_max=64)):
        h, v = layout_for(hm, **opts)
        try:
            assert multi_view(h, v).n_tiles == 0
        finally:
            _lib.hmvm_lib().hmvm_b200_layout_destroy(h)


def test_changed_entries_are_rejected():
    """One entry of each table moved outside its buffer, or onto another's outputs."""
    hm = HMatrix.generate(3000, "sphere", eta=2.0, eps=1e-5, leaf_size=24, seed=9)
    h, v = layout_for(hm, precision=0, nrhs_max=8, num_sms=3)
    try:
        m = multi_view(h, v)
        tiles, segs, first = _arrays(m)
        tb2 = np.ctypeslib.as_array(m.team_begin2, (m.stage2_teams + 1,))
        red2 = np.ctypeslib.as_array(m.red2, (4 * m.n_red2,))
        own_tb2 = np.ctypeslib.as_array(v.team_begin2, (v.stage2_teams + 1,))
        row = m.stage1_tiles  # the first row-stage item
        whole = next(k for k in range(row, m.n_tiles) if tiles[k]["mode"] == 0)
        shared = next(k for k in range(row, m.n_tiles) if tiles[k]["mode"] == 2)
        long = next(k for k in range(row, m.n_tiles) if tiles[k]["nseg"] > 1)
        xseg = next(j for j in range(m.n_segs) if segs[j]["src"] >= 0)
        assert _validate(h)[0] == _lib.HMVM_OK
        for arr, idx, field, value, phrase in [
            (tiles, row, "data_off", v.data_vectors, "leave the data stream"),
            (tiles, row + 1, "data_off", int(tiles[row]["data_off"]), "does not follow"),
            (tiles, row, "seg_begin", m.n_segs, "segment descriptors"),
            (tiles, row, "nrows", 33, "rows are outside"),
            (tiles, row, "nvec", int(tiles[row]["nvec"]) + 1, "leave the data stream"),
            (tiles, whole, "out_base", v.nd, "output rows"),
            (tiles, whole, "out_base", (int(tiles[whole]["out_base"]) + 32) % (v.nd - 32), "another item writes"),
            (tiles, shared, "out_base", v.p_len, "output rows"),
            (tiles, shared, "out_base", int(tiles[shared]["out_base"]) + 1, "another item writes"),
            (segs, xseg, "src", v.nd, "columns leave x or t"),
            (first, int(tiles[long]["seg_begin"]) + 1, None, 0, "first column"),
            (red2, 0, None, int(red2[4]), "written already"),
            (red2, 1, None, int(red2[1]) + 1, "not its own"),
            (red2, 2, None, 1 << 20, "reduction entry"),
            (tb2, m.stage2_teams, None, int(tb2[m.stage2_teams]) - 1, "team ranges"),
            (own_tb2, 0, None, int(own_tb2[0]) + 1, "team ranges"),
        ]:
            old = arr[idx][field] if field else arr[idx]
            if field:
                arr[idx][field] = value
            else:
                arr[idx] = value
            rc, msg = _validate(h)
            if field:
                arr[idx][field] = old
            else:
                arr[idx] = old
            assert rc == _lib.HMVM_ERANGE and phrase in msg, (idx, field, value, phrase, rc, msg)
            assert ("multi-RHS" in msg) == (arr is not own_tb2)
            assert _validate(h)[0] == _lib.HMVM_OK
    finally:
        _lib.hmvm_lib().hmvm_b200_layout_destroy(h)


def test_view_struct_matches_the_header(tmp_path):
    py = _lib.LayoutMultiView
    lines = ['#include <stdio.h>', '#include <stddef.h>', '#include "hmvm_b200.h"', "int main(void) {",
             '  printf("%zu", sizeof(hmvm_layout_multi_view));']
    lines += [f'  printf(" %zu", offsetof(hmvm_layout_multi_view, {f}));' for f, _ in py._fields_]
    src, exe = tmp_path / "view.c", tmp_path / "view"
    src.write_text("\n".join(lines + ["  return 0; }"]))
    subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    assert [int(o) for o in out] == [C.sizeof(py)] + [getattr(py, f).offset for f, _ in py._fields_]
