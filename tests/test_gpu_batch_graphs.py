"""A batch's captured graph across changes of the buffers that it names."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tiles(owm, sizes, seed, walk=False):
    out = []
    for k, n in enumerate(sizes):
        rng = np.random.default_rng(seed + k)
        side = 60.0
        x0 = 500000.0 + 100.0 * k
        xyz = np.column_stack([x0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, rng.random(n) * 9.0])
        out.append((xyz, owm.Bbox(x0, 4700000.0, x0 + side, 4700000.0 + side), owm.run_cfg(10, 0.8, 15, 32, stage1_walk=walk)))
    return out


def _launches(ctx, batch, tiles):
    l0 = ctx.launches
    return batch.run(tiles), ctx.launches - l0


@pytest.mark.parametrize("walk", [False, True])
def test_more_tiles_between_two_replays(owm, walk):
    """The pinned offsets grow with the number of tiles while the device buffer
    stays: the graph that writes to the old ones is captured anew."""
    ctx = owm.Context(0)
    few, many = _tiles(owm, [300_000, 500_000, 400_000], 1, walk), _tiles(owm, [1_500] * 40, 9, walk)
    want_few, want_many = [], []
    for tiles, want in ((few, want_few), (many, want_many)):
        for xyz, bb, cfg in tiles:
            want.append(ctx.run_host(xyz, bb, cfg))
    b = owm.Batch(ctx)
    b.set_graphs(True)
    b.run(few)
    again, replayed = _launches(ctx, b, few)
    assert replayed == 1
    b.set_graphs(False)  # the graph stays
    for g, w in zip(b.run(many), want_many):
        np.testing.assert_array_equal(g, w)
    b.set_graphs(True)
    for k in range(2):
        got, n = _launches(ctx, b, few)
        assert (n == 1) == (k == 1)
        for g, a, w in zip(got, again, want_few):
            np.testing.assert_array_equal(g, w)
            np.testing.assert_array_equal(a, w)
    b.close()
    ctx.close()
