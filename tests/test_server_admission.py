"""What a server admits as one batch: tiles that cannot go together go in
smaller batches, sums that would wrap are over the budget, and a burst that is
over the budget as a whole still completes."""
import ctypes as C

import numpy as np
import pytest


def _tile(owm, n, seed=1, side=300.0):
    rng = np.random.default_rng(seed)
    m = min(n, 40_000)
    xyz = np.column_stack([500000.0 + rng.random(m) * side, 4700000.0 + rng.random(m) * side, rng.random(m) * 9.0])
    return xyz, owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side), owm.run_cfg(10, 0.8, 20, 32)


def _admitted(owm, tiles, budget, n=None):
    descs, keep, _ = owm.tile_descs(tiles)
    for d in descs:
        d.n = n or d.n  # sizes alone: the points are not read
    size, rc = C.c_int64(), C.c_int32()
    f = owm.lib().owm_server_admissible_host
    f.argtypes = [C.c_void_p, C.c_int32, C.c_int64, C.POINTER(C.c_int64), C.POINTER(C.c_int32)]
    k = f(descs, len(tiles), budget, C.byref(size), C.byref(rc))
    return k, size.value, rc.value


def test_batches_that_cannot_be_laid_out_are_split(owm):
    """2^32 points and more in one batch, and (tile, id) keys above 32 bits."""
    tiles = [_tile(owm, 1000, s) for s in range(4)]
    budget = 1 << 50
    k, size, rc = _admitted(owm, tiles, budget, 1_200_000_000)
    assert (k, rc) == (2, 0) and 0 < size < budget
    k, size, rc = _admitted(owm, tiles, budget, 2_000_000_000)
    assert (k, rc) == (2, 0) and 0 < size < budget


def test_batches_over_the_budget_are_split(owm):
    # tiles that ask for the tree walk: a batch of theirs has one size
    tiles = [(x, b, owm.run_cfg(10, 0.8, 20, 32, stage1_walk=True)) for x, b, _ in (_tile(owm, 40_000, s) for s in range(8))]
    whole = _admitted(owm, tiles, 1 << 40)
    one = _admitted(owm, tiles[:1], 1 << 40)
    assert whole[0] == 8 and one[0] == 1 and whole[1] > 4 * one[1]
    assert _admitted(owm, tiles, whole[1])[0] == 8
    assert _admitted(owm, tiles, whole[1] - 1)[0] == 4
    assert _admitted(owm, tiles, one[1])[0] == 1
    assert _admitted(owm, tiles, one[1] // 4) == (0, _admitted(owm, tiles[:1], one[1] // 4)[1], -2)


def test_sums_do_not_wrap(owm):
    f = owm.lib().owm_server_within_host
    f.argtypes = [C.c_uint64] * 3
    top = (1 << 64) - 1
    assert f(10, 20, 30) == 1 and f(10, 21, 30) == 0
    assert f(1 << 33, top - 1, 1 << 37) == 0 and f(31, 0, 30) == 0


@pytest.mark.gpu
def test_a_burst_over_the_budget_completes(owm):
    ctx = owm.Context(0)
    tiles = [_tile(owm, 40_000, s) for s in range(12)]
    want = [ctx.run_host(*t) for t in tiles]
    one = _admitted(owm, tiles[:1], 1 << 40)[1]
    srv = owm.Server(0, hbm_budget_bytes=2 * one, max_tiles_per_batch=64, max_inflight_batches=1)
    tickets = [srv.submit(*t) for t in tiles]
    for t, ticket, w in zip(tiles, tickets, want):
        p = owm.params(t[1], len(t[0]), t[2].wsize, t[2].overlap, t[2].bsize)
        seeds, _ = srv.wait(ticket, p.ncells + p.ngrid + 1, 10000.0)
        np.testing.assert_array_equal(seeds, w)
    srv.close()
    ctx.close()
