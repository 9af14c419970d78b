"""A walk limit acts on the walks that a call makes and on nothing else: owm_run
walks the tree for its cells alone, stage1_walk for its windows too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OWM_ETIMEOUT = -4


def _cloud(n=150_000, w=70.0, h=80.0):
    rng = np.random.default_rng(12)
    z = np.round(50 + rng.random(n) * 4, 2)
    return np.column_stack([500000.0 + rng.random(n) * w, 4700000.0 + rng.random(n) * h, z])


@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("Ov,B", [(0.8, 3), (0.0, 3), (0.5, 0)])
def test_limit_above_the_cells_and_below_the_windows(owm, oracle, Ov, B, policy):
    ctx = owm.Context(0)
    xyz = _cloud()
    bb = owm.Bbox(500000.0, 4700000.0, 500070.0, 4700080.0)
    cloud = ctx.cloud(xyz, bb)
    tree = ctx.tree(cloud, policy, 32, 0.5)
    p, p0 = owm.params(bb, len(xyz), 10, Ov, B), oracle.params(bb, len(xyz), 10, Ov, B)
    want, _ = oracle.run(xyz, bb, 10, Ov, B)
    llp = oracle.stage2(oracle.stage1(xyz, p0), Ov)
    cfg = owm.run_cfg(10, Ov, B, 32, policy, 0.5)
    walk = owm.run_cfg(10, Ov, B, 32, policy, 0.5, stage1_walk=True)
    ctx.set_walk_limit(40)
    if B:
        np.testing.assert_array_equal(ctx.stage3(tree, p, llp), oracle.stage3(xyz, p0, llp))
    with pytest.raises(owm.OwmError) as e:
        ctx.stage1(tree, p)
    assert e.value.status == OWM_ETIMEOUT
    with pytest.raises(owm.OwmError) as e:
        ctx.run(cloud, walk)
    assert e.value.status == OWM_ETIMEOUT
    info = owm.RunInfo()
    np.testing.assert_array_equal(ctx.run(cloud, cfg, info), want)
    assert info.n_seeds == len(want) and min(info.ms_tree, info.ms_stage1, info.ms_stage2, info.ms_total) > 0
    np.testing.assert_array_equal(ctx.run_host(xyz, bb, cfg), want)
    np.testing.assert_array_equal(ctx.run_wait(ctx.run_submit(cloud, cfg)), want)
    assert ctx.device_status() == 0
    if B:  # the cell walk's bound acts inside a run
        ctx.set_walk_limit(1)
        with pytest.raises(owm.OwmError) as e:
            ctx.run(cloud, cfg)
        assert e.value.status == OWM_ETIMEOUT
    bad = xyz.copy()
    bad[7, 0] = np.inf
    with pytest.raises(owm.OwmError) as e:
        ctx.run_host(bad, bb, cfg)
    assert e.value.status == -1
    ctx.set_walk_limit(0)
    np.testing.assert_array_equal(ctx.run(cloud, cfg), want)
    np.testing.assert_array_equal(ctx.run(cloud, walk), want)
    ctx.close()
