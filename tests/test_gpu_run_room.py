"""owm_run where the window grid's tables do not fit: the tree path, the same seeds."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ov,B", [(0.8, 4), (0.0, 6), (0.5, 0)])
@pytest.mark.parametrize("policy", [0, 1])
def test_run_with_room_for_the_tree_alone(owm, oracle, Ov, B, policy):
    ctx = owm.Context(0)
    n, side = 3_000, 1500.0
    rng = np.random.default_rng(5)
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, np.round(rng.random(n) * 9, 2)])
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    cfg = owm.run_cfg(5, Ov, B, 32, policy, 4.0)
    want, _ = oracle.run(xyz, bb, 5, Ov, B)
    cloud = ctx.cloud(xyz, bb)
    owm.lib().owm_ctx_limit_scratch(ctx.handle, C.c_int64(10 << 20))
    l0 = ctx.launches
    np.testing.assert_array_equal(ctx.run(cloud, cfg), want)
    assert ctx.launches - l0 > 12  # the grid takes eight
    np.testing.assert_array_equal(ctx.run_host(xyz, bb, cfg), want)
    np.testing.assert_array_equal(ctx.run_wait(ctx.run_submit(cloud, cfg)), want)
    bad = xyz.copy()
    bad[5, 2] = np.nan
    with pytest.raises(owm.OwmError) as e:
        ctx.run_host(bad, bb, cfg)
    assert e.value.status == -1
    owm.lib().owm_ctx_limit_scratch(ctx.handle, C.c_int64(4096))
    small = owm.Context(0)
    owm.lib().owm_ctx_limit_scratch(small.handle, C.c_int64(4096))
    with pytest.raises(owm.OwmError) as e:
        small.run_host(xyz, bb, cfg)
    assert e.value.status == -2
    small.close()
    ctx.close()
