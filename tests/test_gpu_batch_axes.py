"""Batches of tiles where the batched fold can go wrong, against the oracle: axes
across zero and across a power of two (no fast form), cells with a table of their
own, points outside the tile's box, coordinates on edges, crowded tiles, overlap 0
beside others, and points around a chunk's end.  Ids: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tile(owm, n, x0, y0, side, W, Ov, B, seed, quantum=0.0, order="none", out=0.0, crowd=0.0):
    rng = np.random.default_rng(seed)
    xy = rng.random((n, 2)) * side
    m = int(crowd * n)
    xy[:m] = 0.4 * side + rng.random((m, 2))
    if quantum:
        xy = np.round(xy / quantum) * quantum
    xy = xy[np.lexsort((xy[:, 0], np.floor(xy[:, 1] * 2)))] if order == "scan" else xy[rng.permutation(n)]
    z = np.round(50 + 3 * np.sin(xy[:, 0] / 9) + rng.random(n) * 4, 2)
    z[:: max(1, n // 7)] = -0.0
    bb = owm.Bbox(x0 + out, y0 + out, x0 + side - out, y0 + side - out)
    return np.column_stack([x0 + xy[:, 0], y0 + xy[:, 1], z]), bb, owm.run_cfg(W, Ov, B, 32)


KINDS = {
    "across zero": dict(n=30_001, x0=-31.0, y0=-17.5, side=60.0, W=10, Ov=0.8, B=6),
    "across zero, scan": dict(n=30_001, x0=-31.0, y0=1000.0, side=60.0, W=9, Ov=0.3, B=4, quantum=0.01, order="scan"),
    "negative": dict(n=20_000, x0=-500000.0, y0=-4700000.0, side=50.0, W=10, Ov=0.5, B=15, quantum=0.5),
    "power of two": dict(n=30_000, x0=524250.0, y0=4194280.0, side=60.0, W=10, Ov=0.8, B=20, quantum=0.01),
    "own cells": dict(n=50_000, x0=500000.0, y0=4700000.0, side=1200.0, W=40, Ov=0.5, B=2, quantum=0.25),
    "own cells, scan": dict(n=50_000, x0=-600.0, y0=4700000.0, side=1200.0, W=31, Ov=0.2, B=2, order="scan"),
    "outside": dict(n=25_000, x0=100000.0, y0=200000.0, side=40.0, W=7, Ov=0.5, B=6, out=3.7),
    "edges": dict(n=40_000, x0=500000.0, y0=4700000.0, side=80.0, W=10, Ov=0.8, B=20, quantum=1.0),
    "crowded": dict(n=60_000, x0=500000.0, y0=4700000.0, side=80.0, W=10, Ov=0.8, B=5, crowd=0.8),
    "no cells": dict(n=15_000, x0=500000.0, y0=4700000.0, side=40.0, W=9, Ov=0.6, B=0),
    "few windows": dict(n=70_000, x0=500000.0, y0=4700000.0, side=40.0, W=30, Ov=0.5, B=20),
}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("zero", [False, True])
def test_kinds(owm, oracle, ctx, kind, zero):
    """Two tiles of a kind with an ordinary one between them, and (zero) one of
    overlap 0, which sorts stage 2 of all."""
    plain = dict(n=20_000, x0=501000.0, y0=4701000.0, side=45.0, W=10, Ov=0.8, B=20)
    specs = [KINDS[kind], plain, dict(KINDS[kind], n=KINDS[kind]["n"] // 3)]
    if zero:
        specs.append(dict(plain, Ov=0.0, W=8))
    tiles = [_tile(owm, seed=k + 1, **s) for k, s in enumerate(specs)]
    want = [oracle.run(x, bb, c.wsize, c.overlap, c.bsize)[0] for x, bb, c in tiles]
    b = owm.Batch(ctx)
    for graphs in (False, True, True):
        b.set_graphs(graphs)
        for k, (g, w) in enumerate(zip(b.run(tiles), want)):
            np.testing.assert_array_equal(g, w, err_msg=f"tile {k}")
    b.close()


@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 4095, 4096, 4097, 8193])
def test_ends_of_chunks(owm, oracle, ctx, n):
    specs = [dict(n=n, x0=-9.0 if k == 1 else 500000.0, y0=4700000.0, side=23.0, W=6, Ov=0.5, B=5) for k in range(3)]
    tiles = [_tile(owm, seed=n + k, **s) for k, s in enumerate(specs)]
    b = owm.Batch(ctx)
    for g, (x, bb, c) in zip(b.run(tiles), tiles):
        np.testing.assert_array_equal(g, oracle.run(x, bb, c.wsize, c.overlap, c.bsize)[0])
    tiles[1][0][n // 2, 1] = np.nan
    with pytest.raises(owm.OwmError):
        b.run(tiles)
    b.close()
