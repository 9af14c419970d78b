"""A batch whose window-grid tables cannot be numbered, do not fit or are over a
server's budget runs on its tiles' trees, where those take less."""
import ctypes as C

import numpy as np
import pytest

OWM_ENOMEM, OWM_ERANGE = -2, -6


def _sparse(owm, seed=1, n=2_000, side=2000.0, B=4):
    """Few points on a large area: the grid's tables are the larger."""
    rng = np.random.default_rng(seed)
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, rng.random(n) * 9.0])
    return xyz, owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side), owm.run_cfg(10, 0.8, B, 32)


def _route(owm, tiles, most=1 << 60):
    descs, keep, _ = owm.tile_descs(tiles)
    grid, size = C.c_int32(), C.c_int64()
    f = owm.lib().owm_batch_route_host
    f.argtypes = [C.c_void_p, C.c_int32, C.c_int64, C.POINTER(C.c_int32), C.POINTER(C.c_int64)]
    rc = f(descs, len(tiles), most, C.byref(grid), C.byref(size))
    return rc, grid.value, size.value


def _sizes(owm, tiles):
    """Bytes on the grid and on the trees."""
    rc, grid, by_grid = _route(owm, tiles)
    assert (rc, grid) == (0, 1)
    walk = [(x, b, owm.run_cfg(c.wsize, c.overlap, c.bsize, 32, stage1_walk=True)) for x, b, c in tiles]
    rc, grid, by_trees = _route(owm, walk)
    assert (rc, grid) == (0, 0)
    return by_grid, by_trees


@pytest.mark.parametrize("k", [1, 3])
def test_route_by_bytes(owm, k):
    tiles = [_sparse(owm, s) for s in range(k)]
    by_grid, by_trees = _sizes(owm, tiles)
    assert by_trees < by_grid
    assert _route(owm, tiles, by_grid) == (0, 1, by_grid)
    assert _route(owm, tiles, by_grid - 1) == (0, 0, by_trees)
    assert _route(owm, tiles, by_trees) == (0, 0, by_trees)
    assert _route(owm, tiles, by_trees - 1) == (0, 1, by_grid)  # over it either way


def test_sub_cells_that_cannot_be_numbered(owm):
    xyz, bb, cfg = _sparse(owm)
    big = (xyz, owm.Bbox(0.0, 0.0, 60000.0, 60000.0), owm.run_cfg(1, 0.0, 0, 32))  # 3.6 G windows
    assert owm.params(big[1], len(xyz), 1, 0.0, 0).ncells == 60001 * 60001
    rc, grid, size = _route(owm, [big])
    assert (rc, grid) == (0, 0) and size > 0
    assert _route(owm, [(xyz, bb, owm.run_cfg(10, 0.8, 4, 0))])[0] == -1  # a bad tile stays one


@pytest.mark.gpu
def test_batch_and_server_with_room_for_the_trees_alone(owm, oracle):
    ctx = owm.Context(0)
    tiles = [_sparse(owm, s) for s in range(3)]
    want = [oracle.run(x, b, c.wsize, c.overlap, c.bsize)[0] for x, b, c in tiles]
    by_grid, by_trees = _sizes(owm, tiles)
    b = owm.Batch(ctx)
    owm.lib().owm_batch_limit_memory(b.handle, C.c_int64((by_grid + by_trees) // 2))
    for got in (b.run(tiles), b.run(tiles)):
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)
    owm.lib().owm_batch_limit_memory(b.handle, C.c_int64(1 << 20))
    b.close()
    c = owm.Batch(ctx)
    owm.lib().owm_batch_limit_memory(c.handle, C.c_int64(by_trees // 2))
    with pytest.raises(owm.OwmError) as e:
        c.run(tiles)
    assert e.value.status == OWM_ENOMEM
    c.close()
    one_grid, one_trees = _sizes(owm, tiles[:1])
    srv = owm.Server(0, hbm_budget_bytes=(one_grid + one_trees) // 2, max_tiles_per_batch=1, max_inflight_batches=1)
    for (x, bb, cfg), w in zip(tiles, want):
        p = owm.params(bb, len(x), cfg.wsize, cfg.overlap, cfg.bsize)
        seeds, _ = srv.wait(srv.submit(x, bb, cfg), p.ncells + p.ngrid + 1, 20000.0)
        np.testing.assert_array_equal(seeds, w)
    srv.close()
    ctx.close()
