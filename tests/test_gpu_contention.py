"""Many updates of one address: results as the oracle's, and the kernels' times
within a factor of the same work spread over many addresses (they queued in L2 and
took 30 times as long)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernel_us(owm, ctx, fn, reps=5, cap=128):
    """Median microseconds by kernel name of one call of fn."""
    got = {}
    fn()
    for _ in range(reps):
        owm.lib().owm_ctx_set_profiling(ctx.handle, 1)
        fn()
        names, ms, calls, n = (C.c_char * 64 * cap)(), (C.c_double * cap)(), (C.c_int64 * cap)(), C.c_int32()
        owm.lib().owm_ctx_kernel_times(ctx.handle, cap, names, ms, calls, C.byref(n))
        owm.lib().owm_ctx_set_profiling(ctx.handle, 0)
        for k in range(n.value):
            got.setdefault(names[k].value.decode(), []).append(1e3 * ms[k])
    return {k: float(np.median(v)) for k, v in got.items()}


def _want(w):
    ids, counts = np.unique(w[w >= 0], return_counts=True)
    return ids[counts > 1]


@pytest.mark.parametrize("ids", [1, 33, 1000])
def test_few_ids_in_many_windows(owm, ids):
    ctx = owm.Context(0)
    n = 3_000_000
    rng = np.random.default_rng(ids)
    few = rng.integers(0, ids, n)
    few[rng.random(n) < 0.1] = -1
    few[:2] = [ids + 5, ids + 70]  # once each
    spread = np.repeat(rng.permutation(20_000_000)[: n // 7 + 1], 7)[:n]
    for w in (few, spread):
        np.testing.assert_array_equal(ctx.stage2(w.copy(), 0.8), _want(w))
    slow = _kernel_us(owm, ctx, lambda: ctx.stage2(few.copy(), 0.8))["k_s2_mark"]
    fast = _kernel_us(owm, ctx, lambda: ctx.stage2(spread.copy(), 0.8))["k_s2_mark"]
    assert slow < 15 * fast, (slow, fast)
    ctx.close()


def test_sparse_cloud_under_many_windows(owm, oracle):
    ctx = owm.Context(0)
    n, side = 2_000, 2000.0
    rng = np.random.default_rng(2)
    xyz = np.column_stack([500000.0 + rng.random(n) * side, 4700000.0 + rng.random(n) * side, np.round(rng.random(n) * 9, 2)])
    bb = owm.Bbox(500000.0, 4700000.0, 500000.0 + side, 4700000.0 + side)
    cfg = owm.run_cfg(10, 0.8, 20, 32)
    cloud = ctx.cloud(xyz, bb)
    np.testing.assert_array_equal(ctx.run(cloud, cfg), oracle.run(xyz, bb, 10, 0.8, 20)[0])
    us = _kernel_us(owm, ctx, lambda: ctx.run(cloud, cfg))
    assert us["k_grid_windows"] < 20 * us["k_grid_rows"], us
    ctx.close()
