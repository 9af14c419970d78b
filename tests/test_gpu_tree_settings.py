"""The tree path's settings act on the tree path: leaf classes leave a batch's
graph on the window grid alone, the tuners time runs that build the tree, and
runs by the walk give the oracle's seeds for every leaf size and policy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n=60_000, side=60.0, x0=500000.0, seed=3):
    rng = np.random.default_rng(seed)
    xyz = np.column_stack([x0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, np.round(50 + 4 * rng.random(n), 2)])
    return xyz, (x0, 4700000.0, x0 + side, 4700000.0 + side)


@pytest.mark.parametrize("walk", [False, True])
def test_leaf_classes_and_the_graph(owm, walk):
    ctx = owm.Context(0)
    tiles = []
    for k in range(3):
        xyz, box = _cloud(20_000 + 5_000 * k, seed=k)
        tiles.append((xyz, owm.Bbox(*box), owm.run_cfg(10, 0.8, 15, 32, stage1_walk=walk)))
    b = owm.Batch(ctx)
    b.set_graphs(True)
    want = b.run(tiles)
    for leaf in (16, 128):
        b.set_leaf_classes([1 << 40], [leaf])
        l0 = ctx.launches
        got = b.run(tiles)
        assert (ctx.launches - l0 == 1) == (not walk)  # replayed; the trees of other leaves are captured anew
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    l0 = ctx.launches
    b.run(tiles)
    assert ctx.launches - l0 == 1
    b.close()
    ctx.close()


def _kernels(owm, ctx, fn, cap=128):
    owm.lib().owm_ctx_set_profiling(ctx.handle, 1)
    fn()
    names, ms, calls, n = (C.c_char * 64 * cap)(), (C.c_double * cap)(), (C.c_int64 * cap)(), C.c_int32()
    owm.lib().owm_ctx_kernel_times(ctx.handle, cap, names, ms, calls, C.byref(n))
    owm.lib().owm_ctx_set_profiling(ctx.handle, 0)
    return {names[k].value.decode(): calls[k] for k in range(n.value)}


def test_tuners_time_the_tree_path(owm):
    from fastowm_gb300 import autotune

    ctx = owm.Context(0)
    xyz, box = _cloud()
    cloud = ctx.cloud(xyz, owm.Bbox(*box))
    leaves = (32, 128)
    runs = {"leaf": lambda: autotune.tune_leaf_single(ctx, cloud, lambda leaf: owm.run_cfg(10, 0.8, 15, leaf), leaves, reps=1),
            "shapes": lambda: autotune.tune_shapes_single(ctx, cloud, owm.run_cfg(10, 0.8, 15, 32), reps=1),
            "classes": lambda: autotune.tune_leaf_classes(ctx, bounds=(200_000,), leaves=leaves, tiles_per_class=1, reps=1)}
    for name, tune in runs.items():
        seen = _kernels(owm, ctx, tune)
        assert any("gather" in k for k in seen) and not any("grid" in k for k in seen), (name, seen)
    cloud.close()
    ctx.close()


@pytest.mark.parametrize("leaf,policy,radius", [(1, 1, 0.1), (7, 1, 0.1), (32, 1, 0.1), (256, 1, 0.1), (1000, 1, 0.1), (32, 0, 0.5),
                                                (32, 0, 4.0)])
@pytest.mark.parametrize("x0,W,Ov,B", [(500000.0, 10, 0.8, 6), (-31.0, 9, 0.3, 4), (500000.0, 8, 0.0, 5)])
def test_runs_by_the_walk(owm, oracle, ctx, leaf, policy, radius, x0, W, Ov, B):
    xyz, box = _cloud(30_000, 45.0, x0)
    bb = owm.Bbox(*box)
    cloud = ctx.cloud(xyz, bb)
    got = ctx.run(cloud, owm.run_cfg(W, Ov, B, leaf, policy, radius, stage1_walk=True))
    cloud.close()
    np.testing.assert_array_equal(got, oracle.run(xyz, bb, W, Ov, B)[0])
