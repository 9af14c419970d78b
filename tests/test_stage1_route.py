"""owm_stage1 on the window grid only where the grid can hold the job: windows
whose sub-cells cannot be numbered, parameters whose windows do not rise, and a
scratch that cannot grow go by the tree walk."""
import ctypes as C

import numpy as np
import pytest


def _route(owm, p, n, leaf=32):
    f = owm.lib().owm_stage1_route_host
    f.argtypes = [C.POINTER(type(p)), C.c_int64, C.c_int32]
    return f(C.byref(p), n, -(-n // leaf))


def _params(owm, side=2000.0, W=10, Ov=0.8, n=2_000_000):
    return owm.params(owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side), n, W, Ov, 20)


@pytest.mark.parametrize("ncols,nrows,grid", [(1009, 1009, 1), (32767, 16383, 1), (32768, 32767, 0), (65535, 65535, 0)])
def test_sub_cells_that_cannot_be_numbered_walk(owm, ncols, nrows, grid):
    p = _params(owm)
    p.ncols, p.nrows, p.ncells = ncols, nrows, ncols * nrows
    assert _route(owm, p, 2_000_000) == grid


@pytest.mark.parametrize("change", [lambda p: setattr(p, "displace", 0.0), lambda p: setattr(p, "displace", -2.0),
                                    lambda p: setattr(p, "displace", float("nan")),
                                    lambda p: setattr(p.bbox, "max_x", p.bbox.min_x),
                                    lambda p: setattr(p.bbox, "max_y", float("nan")),
                                    lambda p: setattr(p.bbox, "max_y", float("inf"))])
def test_windows_that_do_not_rise_and_boxes_without_an_area_walk(owm, change):
    p = _params(owm)
    assert _route(owm, p, 2_000_000) == 1
    change(p)
    assert _route(owm, p, 2_000_000) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [4096, 1 << 20])
def test_walks_when_the_scratch_cannot_grow(owm, oracle, limit):
    ctx = owm.Context(0)
    rng = np.random.default_rng(4)
    n, side = 80_000, 90.0
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, np.round(rng.random(n) * 9, 2)])
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    p = owm.params(bb, n, 10, 0.8, 20)
    p0 = oracle.params(bb, n, 10, 0.8, 20)
    assert _route(owm, p, n) == 1
    cloud = ctx.cloud(xyz, bb)
    tree = ctx.tree(cloud)
    other = owm.Context(0)  # its scratch holds nothing yet
    owm.lib().owm_ctx_limit_scratch(other.handle, C.c_int64(limit))
    want = oracle.stage1(xyz, p0)
    np.testing.assert_array_equal(other.stage1(tree, p), want)
    np.testing.assert_array_equal(ctx.stage1(tree, p), want)
    tree.close()
    cloud.close()
    other.close()
    ctx.close()
