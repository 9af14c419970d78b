"""The window grid's per-axis classification on the CPU: the edge counts that
its fixed-point form gives (owm_grid_classify_host, the code the kernels run)
against a search of the same edges, over every kind of axis: positive
coordinates of one binade and axes that cross a power of two or zero, windows
and cells that tile the axis in whole steps and ones that do not, coordinates
on the edges, one ulp beside them, near them, in whole centimetres, outside
the box and at the ends of the range.  Counts are integers: equal."""
import ctypes as C

import numpy as np
import pytest

AXES = [
    (500000.0, 502000.0), (500000.0, 500200.37), (4700000.01, 4700100.0), (1.0, 1.5),  # one binade
    (1000.0, 1100.0), (523000.0, 525000.0), (4194000.0, 4194900.5),                    # across a power of two
    (-20.0, 20.0), (-7.25, -0.125), (0.0, 7.0), (-5.0e6, -4.99e6), (1e-3, 90.0),       # zero, negative, many binades
]
STEPS = [(12, 0.8, 20), (10, 0.5, 15), (9, 0.3, 11), (2, 0.9, 5), (16, 0.0, 1), (1, 0.5, 2), (40, 0.95, 0), (5, 0.6, 3)]


def _d(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _i(a):
    return a.ctypes.data_as(C.POINTER(C.c_int32))


@pytest.mark.parametrize("lo,hi", AXES)
@pytest.mark.parametrize("W,Ov,B", STEPS)
def test_counts_equal_a_search(owm, lo, hi, W, Ov, B):
    f = owm.lib().owm_grid_classify_host
    p = owm.params((lo, lo, hi, hi), 1000, W, Ov, B)
    n, nc = p.ncols, p.ncols_grid
    if n <= 0:
        pytest.skip("no windows")

    def classify(x):
        edges, counts, mode = np.zeros(2 * n + 2 * nc), np.zeros((x.size, 4), np.int32), np.zeros(4, np.int32)
        rc = f(C.c_double(lo), C.c_double(hi), C.c_double(p.displace), W, n, B, nc, _d(x), C.c_int64(x.size), _d(edges),
               _i(counts), _i(mode))
        assert rc == 0  # the single-place form agrees wherever it settles a coordinate
        return edges, counts, mode

    edges, _, _ = classify(np.zeros(1))
    rng = np.random.default_rng(7)
    e = edges[rng.integers(0, edges.size, 400)]
    x = lo + rng.random(2000) * (hi - lo)
    x = np.concatenate([x, np.round(x * 100) / 100, e, np.nextafter(e, np.inf), np.nextafter(e, -np.inf),
                        e + (hi - lo) * rng.normal(size=400) * 2.0 ** -rng.integers(8, 50, 400),
                        lo - (hi - lo) + rng.random(300) * 3 * (hi - lo), rng.normal(size=50) * 1e9,
                        [lo, hi, 0.0, -0.0, 5e-324, 1.7e308, -1.7e308]])
    edges, counts, mode = classify(x)
    L, R, A, Z = edges[:n], edges[n:2 * n], edges[2 * n:2 * n + nc], edges[2 * n + nc:]
    want = np.stack([np.searchsorted(L, x, "left"), np.searchsorted(R, x, "right"),
                     np.searchsorted(A, x, "left"), np.searchsorted(Z, x, "right")], 1)
    np.testing.assert_array_equal(counts, want)
    assert mode[0] == 1 and mode[3] > 500  # the fixed-point form was in use


@pytest.mark.parametrize("W,Ov,B", STEPS)
def test_edges_are_the_references(owm, W, Ov, B):
    """Window and cell edges by the reference's formulas (optim3_func.cpp:
    310-324, 544-555, 630-651) in numpy's separately rounded doubles."""
    lo, hi = 600000.03, 600431.77
    p = owm.params((lo, lo, hi, hi), 1000, W, Ov, B)
    n, nc = p.ncols, p.ncols_grid
    edges, counts, mode, x = np.zeros(2 * n + 2 * nc), np.zeros((1, 4), np.int32), np.zeros(4, np.int32), np.zeros(1)
    owm.lib().owm_grid_classify_host(C.c_double(lo), C.c_double(hi), C.c_double(p.displace), W, n, B, nc, _d(x),
                                     C.c_int64(1), _d(edges), _i(counts), _i(mode))
    j, i = np.arange(n, dtype=np.float64), np.arange(nc, dtype=np.float64)
    c = ((lo - W // 2) + p.displace) + j * p.displace
    d = (lo + B // 2) + i * B
    want = np.concatenate([c - W // 2, c + W // 2, d - B // 2, d + B // 2])
    np.testing.assert_array_equal(edges, want)
