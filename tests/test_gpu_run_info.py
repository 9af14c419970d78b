"""owm_run's device times: the total ends when the seeds are with the caller, and
does not fall short of its phases."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,B", [(5_000_000, 3000.0, 2), (200_000, 100.0, 20)])
@pytest.mark.parametrize("walk", [False, True])
def test_total_covers_the_copy_of_the_seeds(owm, n, side, B, walk):
    ctx = owm.Context(0)
    rng = np.random.default_rng(1)
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, rng.random(n) * 9.0])
    cloud = ctx.cloud(xyz, owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side))
    cfg = owm.run_cfg(10, 0.8, B, 32, stage1_walk=walk)
    ctx.run(cloud, cfg)
    info = owm.RunInfo()
    seeds = ctx.run(cloud, cfg, info)
    phases = info.ms_tree + info.ms_stage1 + info.ms_stage2 + info.ms_stage3
    copy = 8 * len(seeds) / 250e9 * 1e3  # faster than the link can
    assert info.n_seeds == len(seeds) and phases > 0 and (B != 2 or len(seeds) > 1_500_000)
    assert info.ms_total > phases + (copy if B == 2 else -0.02), (info.ms_total, phases, copy)
    ctx.close()
