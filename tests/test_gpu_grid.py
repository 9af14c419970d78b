"""The whole path on the window grid against the oracle where it can go wrong:
warps that are not full, one cloud in several orders (runs of points in one
sub-cell and none), coordinates on the window and cell edges, axes without the
linear form, cells kept apart from the windows' sub-cells, -0 heights, points
outside the box, and heights at the sentinel's.  Ids: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(rng, n, x0, y0, side, quantum=0.0):
    xy = rng.random((n, 2)) * side
    if quantum:
        xy = np.round(xy / quantum) * quantum
    z = np.round(50 + 3 * np.sin(xy[:, 0] / 9) + rng.random(n) * 4, 2)
    return np.column_stack([x0 + xy[:, 0], y0 + xy[:, 1], z])


def _order(xyz, how):
    if how == "scan":
        return xyz[np.lexsort((xyz[:, 0], np.floor(xyz[:, 1] * 2)))]
    if how == "same":  # long runs in one sub-cell
        return xyz[np.lexsort((np.floor(xyz[:, 0] / 7), np.floor(xyz[:, 1] / 7)))]
    return xyz


def _check(owm, oracle, ctx, xyz, bb, W, Ov, B):
    cloud = ctx.cloud(xyz, bb)
    got = ctx.run(cloud, owm.run_cfg(W, Ov, B, 32))
    host = ctx.run_host(xyz, bb, owm.run_cfg(W, Ov, B, 32))
    cloud.close()
    want, _ = oracle.run(xyz, bb, W, Ov, B)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(host, want)
    return want


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 257, 4099])
def test_sizes(owm, oracle, ctx, n):
    xyz = _cloud(np.random.default_rng(n), n, 500000.0, 4700000.0, 23.0)
    _check(owm, oracle, ctx, xyz, owm.Bbox(500000.0, 4700000.0, 500023.0, 4700023.0), 6, 0.5, 5)


@pytest.mark.parametrize("how", ["shuffled", "scan", "same"])
@pytest.mark.parametrize("x0,y0,quantum", [(500000.0, 4700000.0, 0.01), (500000.0, 4700000.0, 0.5), (-31.0, 1000.0, 0.01),
                                           (524250.0, 4194280.0, 0.0)])
@pytest.mark.parametrize("W,Ov,B", [(10, 0.8, 20), (10, 0.5, 15), (9, 0.3, 4), (8, 0.0, 6)])
def test_orders_edges_axes(owm, oracle, ctx, how, x0, y0, quantum, W, Ov, B):
    xyz = _order(_cloud(np.random.default_rng(3), 30_000, x0, y0, 60.0, quantum), how)
    bb = owm.Bbox(x0, y0, x0 + 60.0, y0 + 60.0)
    assert len(_check(owm, oracle, ctx, xyz, bb, W, Ov, B)) > 0


@pytest.mark.parametrize("W,Ov", [(40, 0.0), (40, 0.5), (31, 0.2)])
def test_cells_apart(owm, oracle, ctx, W, Ov):
    """Few wide windows and many small cells: the cells' edges would multiply
    the sub-cells, so they get a table of their own."""
    xyz = _cloud(np.random.default_rng(5), 200_000, 500000.0, 4700000.0, 1200.0, 0.25)
    bb = owm.Bbox(500000.0, 4700000.0, 501200.0, 4701200.0)
    assert len(_check(owm, oracle, ctx, xyz, bb, W, Ov, 2)) > 100_000


def test_zero_and_sentinel_heights_outside_points(owm, oracle, ctx):
    rng = np.random.default_rng(9)
    xyz = _cloud(rng, 20_000, 100000.0, 200000.0, 40.0, 0.01)
    xyz[:, 2] = rng.choice([0.0, -0.0, 1.0, -1.0, 5e-324], xyz.shape[0])
    bb = owm.Bbox(100003.3, 200001.7, 100037.0, 200035.5)  # the header's, inside the data
    _check(owm, oracle, ctx, xyz, bb, 7, 0.5, 6)
    xyz[:, 2] = np.finfo(np.float64).max  # as high as the sentinel: never below it
    cloud = ctx.cloud(xyz, bb)
    a = ctx.run(cloud, owm.run_cfg(7, 0.5, 6, 32))
    b = ctx.run(cloud, owm.run_cfg(7, 0.5, 6, 32, stage1_walk=True))
    cloud.close()
    np.testing.assert_array_equal(a, b)
    xyz[19_999, 0] = np.inf
    with pytest.raises(owm.OwmError):
        ctx.run_host(xyz, bb, owm.run_cfg(7, 0.5, 6, 32))


@pytest.mark.parametrize("W,Ov,policy", [(10, 0.8, 1), (9, 0.3, 1), (10, 0.5, 0), (60, 0.0, 1)])
@pytest.mark.parametrize("x0", [500000.0, -40.0])
def test_stage1_of_a_tree(owm, oracle, x0, W, Ov, policy):
    """owm_stage1 folds the tree's sorted points into a window grid or walks the
    tree, by the number of windows; a walk limit above every walk's steps gives
    the walk's answer."""
    ctx = owm.Context(0)
    xyz = _cloud(np.random.default_rng(8), 60_000, x0, 1000.0, 80.0, 0.01)
    bb = owm.Bbox(x0, 1000.0, x0 + 80.0, 1080.0)
    cloud = ctx.cloud(xyz, bb)
    tree = ctx.tree(cloud, policy, 32, 0.5)
    p = owm.params(bb, xyz.shape[0], W, Ov, 20)
    got = ctx.stage1(tree, p)
    ctx.set_walk_limit(1 << 30)
    np.testing.assert_array_equal(ctx.stage1(tree, p), got)
    np.testing.assert_array_equal(got, oracle.stage1(xyz, oracle.params(bb, xyz.shape[0], W, Ov, 20)))
    ctx.close()


@pytest.mark.parametrize("n", [7, 1025, 8192, 8193, 32767, 32768])
@pytest.mark.parametrize("x0,quantum,W,Ov,B,fits", [(500000.0, 0.01, 10, 0.8, 20, True), (500000.0, 0.5, 10, 0.5, 15, True),
                                                    (-31.0, 0.01, 9, 0.6, 6, True), (500000.0, 0.0, 8, 0.8, 0, False),
                                                    (500000.0, 0.01, 6, 0.0, 5, False)])
def test_one_launch(owm, oracle, x0, quantum, W, Ov, B, fits, n):
    """Small clouds by one launch (up to 32767 points whose tables fit a block's
    shared memory, overlap above 0), at the ends of its blocks' shares, and the
    first that goes by the chain; the same seeds again in the context's used
    scratch."""
    ctx = owm.Context(0)
    side = 60.0
    xyz = _cloud(np.random.default_rng(n), n, x0, 4700000.0, side, quantum)
    bb = owm.Bbox(x0, 4700000.0, x0 + side, 4700000.0 + side)
    want = _check(owm, oracle, ctx, xyz, bb, W, Ov, B)
    cloud = ctx.cloud(xyz, bb)
    l0 = ctx.launches
    np.testing.assert_array_equal(ctx.run(cloud, owm.run_cfg(W, Ov, B, 32)), want)
    assert (ctx.launches - l0 == 1) == (n < 32768 and fits)
    xyz[n // 2, 1] = np.nan
    with pytest.raises(owm.OwmError):
        ctx.run_host(xyz, bb, owm.run_cfg(W, Ov, B, 32))
    cloud.close()
    ctx.close()


@pytest.mark.parametrize("n", [40_960, 40_961, 622_593])
@pytest.mark.parametrize("heights", ["tied", "falling"])
@pytest.mark.parametrize("x0,side,W,Ov,B,quantum", [(500000.0, 90.0, 16, 0.5, 20, 0.5), (500000.0, 90.0, 16, 0.5, 25, 0.01),
                                                    (-31.0, 60.0, 15, 0.6, 0, 0.01), (500000.0, 1200.0, 200, 0.5, 2, 0.25)])
def test_few_sub_cells(owm, oracle, ctx, x0, side, W, Ov, B, quantum, heights, n):
    """Many points on few sub-cells: blocks fold into tables in shared memory,
    some in more than one group of points; equal heights keep the lowest id,
    and heights that fall with the id replace the entry in every group."""
    rng = np.random.default_rng(n)
    xyz = _cloud(rng, n, x0, 4700000.0, side, quantum)
    xyz[:, 2] = np.round(xyz[:, 2]) if heights == "tied" else 500.0 - np.arange(n) * 1e-4
    bb = owm.Bbox(x0, 4700000.0, x0 + side, 4700000.0 + side)
    _check(owm, oracle, ctx, xyz, bb, W, Ov, B)
    cloud = ctx.cloud(xyz, bb)
    tree = ctx.tree(cloud, 1, 32)
    p = owm.params(bb, n, W, Ov, B)
    np.testing.assert_array_equal(ctx.stage1(tree, p), oracle.stage1(xyz, oracle.params(bb, n, W, Ov, B)))
    tree.close()
    cloud.close()
    xyz[n - 1, 2] = np.inf
    with pytest.raises(owm.OwmError):
        ctx.run_host(xyz, bb, owm.run_cfg(W, Ov, B, 32))
