"""The context's device status word after whole-path runs: it tells of the last
run alone, whichever form that run took (one launch, the chain of kernels, shared
tables), through every entry point."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OWM_EINVAL = -1
OWM_ETIMEOUT = -4
NON_FINITE_BIT = 1
WALK_BOUND_BIT = 2


def _cloud(n, side):
    rng = np.random.default_rng(n)
    return np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, rng.random(n) * 9.0])


def _runs(ctx, owm, xyz, bb, cfg):
    """The whole path by every entry point of a context."""
    cloud = ctx.cloud(xyz, bb)
    return {"run": lambda: ctx.run(cloud, cfg), "run_host": lambda: ctx.run_host(xyz, bb, cfg),
            "host_submit": lambda: ctx.run_host_wait(ctx.run_host_submit(xyz, bb, cfg)),
            "submit": lambda: ctx.run_wait(ctx.run_submit(cloud, cfg))}


@pytest.mark.parametrize("n,side,W,Ov", [(1_000, 20.0, 10, 0.8), (32_767, 40.0, 10, 0.8), (1_000, 20.0, 10, 0.0),
                                         (150_000, 80.0, 10, 0.8), (60_000, 40.0, 30, 0.5)])
@pytest.mark.parametrize("entry", ["run", "run_host", "host_submit", "submit"])
def test_status_is_the_last_runs(owm, n, side, W, Ov, entry):
    ctx = owm.Context(0)
    xyz = _cloud(n, side)
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    bad = xyz.copy()
    bad[n // 3, 2] = np.nan
    cfg, walk = owm.run_cfg(W, Ov, 20, 32), owm.run_cfg(W, Ov, 20, 32, stage1_walk=True)
    good, nan = _runs(ctx, owm, xyz, bb, cfg)[entry], _runs(ctx, owm, bad, bb, cfg)[entry]
    gives_up = _runs(ctx, owm, xyz, bb, walk)[entry]
    good()
    assert ctx.device_status() == 0
    with pytest.raises(owm.OwmError) as e:
        nan()
    assert e.value.status == OWM_EINVAL
    assert ctx.device_status() == NON_FINITE_BIT
    good()
    assert ctx.device_status() == 0
    ctx.set_walk_limit(1)
    with pytest.raises(owm.OwmError) as e:
        gives_up()
    assert e.value.status == OWM_ETIMEOUT
    assert ctx.device_status() == WALK_BOUND_BIT
    ctx.set_walk_limit(0)
    good()
    assert ctx.device_status() == 0
    ctx.close()
