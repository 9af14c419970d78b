"""owm_stage2 on lists whose highest id lies at the ends of its bitmaps' chunks
and beyond all of them (sorted instead): the ids that occur at least twice,
ascending.  Ids: equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 257, 70_001])
@pytest.mark.parametrize("top", [0, 1, 32767, 32768, 1_000_003, (1 << 27) - 1, 1 << 27, (1 << 30) - 1, 1 << 30,
                                 (1 << 32) - 2, None])
def test_repeated_ids(owm, ctx, n, top):
    rng = np.random.default_rng(n)
    if top is None:  # no window holds a point
        win = np.full(n, -1, np.int64)
    else:
        win = top - rng.integers(0, min(top, 3 * n) + 1, n, dtype=np.int64)
        win[rng.random(n) < 0.2] = -1
        win[: min(n, 2)] = top
    ids, count = np.unique(win[win >= 0], return_counts=True)
    np.testing.assert_array_equal(ctx.stage2(win.copy(), 0.5), ids[count >= 2])
    every = np.sort(win[win >= 0])
    np.testing.assert_array_equal(ctx.stage2(win.copy(), 0.0), every)
