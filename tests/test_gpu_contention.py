"""Many updates of one address: results as the oracle's, and the kernels' times
within a factor of the same work spread over many addresses (they queued in L2 and
took 30 times as long)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel_us(owm, ctx, fn, reps=5, cap=128):
    """Median microseconds by kernel name of one call of fn."""
    got = {}
    fn()
    for _ in range(reps):
        owm.lib().owm_ctx_set_profiling(ctx.handle, 1)
        fn()
        names, ms, calls, n = (C.c_char * 64 * cap)(), (C.c_double * cap)(), (C.c_int64 * cap)(), C.c_int32()
        owm.lib().owm_ctx_kernel_times(ctx.handle, cap, names, ms, calls, C.byref(n))
        owm.lib().owm_ctx_set_profiling(ctx.handle, 0)
        for k in range(n.value):
            got.setdefault(names[k].value.decode(), []).append(1e3 * ms[k])
    return {k: float(np.median(v)) for k, v in got.items()}


def _want(w):
    ids, counts = np.unique(w[w >= 0], return_counts=True)
    return ids[counts > 1]


@pytest.mark.parametrize("ids", [1, 33, 1000])
def test_few_ids_in_many_windows(owm, ids):
    ctx = owm.Context(0)
    n = 3_000_000
    rng = np.random.default_rng(ids)
    few = rng.integers(0, ids, n)
    few[rng.random(n) < 0.1] = -1
    few[:2] = [ids + 5, ids + 70]  # once each
    spread = np.repeat(rng.permutation(20_000_000)[: n // 7 + 1], 7)[:n]
    for w in (few, spread):
        np.testing.assert_array_equal(ctx.stage2(w.copy(), 0.8), _want(w))
    slow = _kernel_us(owm, ctx, lambda: ctx.stage2(few.copy(), 0.8))["k_s2_mark"]
    fast = _kernel_us(owm, ctx, lambda: ctx.stage2(spread.copy(), 0.8))["k_s2_mark"]
    assert slow < 15 * fast, (slow, fast)
    ctx.close()


def test_sparse_cloud_under_many_windows(owm, oracle):
    ctx = owm.Context(0)
    n, side = 2_000, 2000.0
    rng = np.random.default_rng(2)
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, np.round(rng.random(n) * 9, 2)])
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    cfg = owm.run_cfg(10, 0.8, 20, 32)
    cloud = ctx.cloud(xyz, bb)
    np.testing.assert_array_equal(ctx.run(cloud, cfg), oracle.run(xyz, bb, 10, 0.8, 20)[0])
    us = _kernel_us(owm, ctx, lambda: ctx.run(cloud, cfg))
    assert us["k_grid_windows"] < 20 * us["k_grid_rows"], us
    ctx.close()


def _crowded(n, side, part, spots, seed, order):
    """part of the points within half a metre of some places, in no order or by places."""
    rng = np.random.default_rng(seed)
    xy = rng.random((n, 2)) * side
    m = int(n * part)
    if spots:
        at = (0.1 + 0.8 * rng.random((spots, 2))) * side
        xy[:m] = at[rng.integers(0, spots, m)] + rng.random((m, 2)) - 0.5
    else:  # as seen from one place: density falls with the square of the distance
        r, a = np.exp(rng.uniform(np.log(0.5), np.log(side / 2), n)), rng.uniform(0, 2 * np.pi, n)
        xy = side / 2 + np.column_stack([r * np.cos(a), r * np.sin(a)])
    xy = xy[rng.permutation(n)] if order == "none" else xy[np.lexsort((xy[:, 0], np.floor(xy[:, 1] * 2)))]
    xyz = np.column_stack([500000.0 + xy[:, 0], 4700000.0 + xy[:, 1], np.round(50 + 4 * rng.random(n), 2)])
    return xyz, (500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)


@pytest.mark.parametrize("n", [40_001, 300_007])
@pytest.mark.parametrize("part,spots,heights", [(0.9, 1, "rough"), (0.5, 3, "rough"), (0.0, 0, "rough"), (0.9, 1, "flat"),
                                                (0.9, 2, "falling"), (0.9, 2, "close")])
@pytest.mark.parametrize("x0", [500000.0, -31.0])
def test_crowded_clouds(owm, oracle, ctx, n, part, spots, heights, x0):
    """Lanes of one sub-cell that are not neighbours, at the ends of warps, with
    equal heights, heights that fall with the id and heights that differ in their
    lower bits alone."""
    xyz, box = _crowded(n, 120.0, part, spots, n, "none")
    rng = np.random.default_rng(n)
    if heights == "flat":
        xyz[:, 2] = 7.25
    elif heights == "falling":
        xyz[:, 2] = 500.0 - np.arange(n) * 1e-6
    elif heights == "close":
        xyz[:, 2] = 500.0 + rng.integers(0, 1000, n) * 1e-9
    xyz[:, 0] += x0 - 500000.0
    bb = owm.Bbox(x0, box[1], x0 + 120.0, box[3])
    cfg = owm.run_cfg(10, 0.8, 6, 32)
    want, _ = oracle.run(xyz, bb, 10, 0.8, 6)
    cloud = ctx.cloud(xyz, bb)
    np.testing.assert_array_equal(ctx.run(cloud, cfg), want)
    cloud.close()
    np.testing.assert_array_equal(ctx.run_host(xyz, bb, cfg), want)
    b = owm.Batch(ctx)
    for got in b.run([(xyz, bb, cfg), (xyz[: n // 3], bb, cfg), (xyz, bb, cfg)])[::2]:
        np.testing.assert_array_equal(got, want)
    b.close()


def test_crowded_cloud_in_no_order_takes_about_as_long_as_its_scan(owm):
    """Nine points of ten in one sub-cell: the adds of a warp go as one."""
    ctx = owm.Context(0)
    n, side, cfg = 5_000_000, 300.0, owm.run_cfg(10, 0.5, 2, 32)
    rng = np.random.default_rng(3)
    xy = rng.random((n, 2)) * side
    xy[: n // 10 * 9] = 150.5 + rng.random((n // 10 * 9, 2))  # window edges at 150 and 155, cell edges at 150 and 152
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    us = {}
    for order, at in (("scan", np.lexsort((xy[:, 0], np.floor(xy[:, 1] * 2)))), ("none", rng.permutation(n))):
        xyz = np.column_stack([500000.0 + xy[at, 0], 4700000.0 + xy[at, 1], np.round(50 + 4 * rng.random(n), 2)])
        cloud = ctx.cloud(xyz, bb)
        us[order] = _kernel_us(owm, ctx, lambda: ctx.run(cloud, cfg))["k_grid_fold"]
        cloud.close()
    assert us["none"] < 2 * us["scan"], us
    ctx.close()


def test_points_on_edges_in_no_order(owm, oracle):
    """Coordinates in whole metres, most of them on window edges: the words that
    say so are stored once, not by every warp."""
    ctx = owm.Context(0)
    n, side, cfg = 300_000, 500.0, owm.run_cfg(10, 0.8, 20, 32)
    rng = np.random.default_rng(6)
    xy = rng.random((n, 2)) * side
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    us = {}
    for step in (0.0, 2.0):
        p = np.round(xy / step) * step if step else xy
        xyz = np.column_stack([500000.0 + p[:, 0], 4700000.0 + p[:, 1], np.round(50 + 4 * rng.random(n), 2)])
        cloud = ctx.cloud(xyz, bb)
        np.testing.assert_array_equal(ctx.run(cloud, cfg), oracle.run(xyz, bb, 10, 0.8, 20)[0])
        us[step] = _kernel_us(owm, ctx, lambda: ctx.run(cloud, cfg))["k_grid_fold"]
        cloud.close()
    assert us[2.0] < 3 * us[0.0], us
    ctx.close()


@pytest.mark.parametrize("density", [0.6, 2.9, 5.9, 6.1, 30.0])
@pytest.mark.parametrize("heights", ["rough", "flat", "falling", "close"])
@pytest.mark.parametrize("W,Ov,B", [(10, 0.8, 20), (9, 0.3, 4)])
def test_scan_order_by_density(owm, oracle, ctx, density, heights, W, Ov, B):
    """Runs of neighbours in a sub-cell, short and long, on both sides of the
    density from which on they are reduced another way; two tiles of a batch on
    different sides."""
    n = 40_003
    side = float(np.ceil(np.sqrt(n / density)))
    rng = np.random.default_rng(int(10 * density))
    xy = rng.random((n, 2)) * side
    xy = xy[np.lexsort((xy[:, 0], np.floor(xy[:, 1] * 2)))]
    z = {"rough": np.round(50 + 4 * rng.random(n), 2), "flat": np.full(n, 7.25), "falling": 500.0 - np.arange(n) * 1e-6,
         "close": 500.0 + rng.integers(0, 1000, n) * 1e-9}[heights]
    xyz = np.column_stack([500000.0 + xy[:, 0], 4700000.0 + xy[:, 1], z])
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    cfg = owm.run_cfg(W, Ov, B, 32)
    want, _ = oracle.run(xyz, bb, W, Ov, B)
    cloud = ctx.cloud(xyz, bb)
    np.testing.assert_array_equal(ctx.run(cloud, cfg), want)
    tree = ctx.tree(cloud)
    p = owm.params(bb, n, W, Ov, B)
    np.testing.assert_array_equal(ctx.stage1(tree, p), oracle.stage1(xyz, oracle.params(bb, n, W, Ov, B)))
    tree.close()
    cloud.close()
    dense = xyz * [0.1, 0.1, 1.0] + [450000.0, 4230000.0, 0.0]
    db = owm.Bbox(500000.0, 4700000.0, 500000.0 + side / 10 + 1, 4700000.0 + side / 10 + 1)
    b = owm.Batch(ctx)
    got = b.run([(xyz, bb, cfg), (dense, db, cfg)])
    np.testing.assert_array_equal(got[0], want)
    np.testing.assert_array_equal(got[1], oracle.run(dense, db, W, Ov, B)[0])
    b.close()
