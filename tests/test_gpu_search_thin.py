"""The lane-a-cell search on grids one to three cells wide in two directions, whose
tiles cannot take 32 cells along every axis: bit-identical to the selection by exact
ranks over every candidate, and its time that of the same cells in another
direction (a tile of one cell took five times as long)."""
import numpy as np
import pytest

import helpers as H
from geo_bsd import hpgl_wrap as W
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu


def _wl(dims, rad, k=32):
    rng = np.random.default_rng(3)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, n // 20, replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    cov = WL.CovSpec(WL.EXPONENTIAL, tuple(float(r) for r in rad), (0.0, 0.0, 0.0), 1.0, 0.05)
    return WL.Workload("thin", dims, data, mask, cov, rad, k)


@pytest.mark.parametrize("dims,rad", [((1, 1, 9000), (1, 1, 300)), ((1, 9000, 1), (1, 300, 1)), ((9000, 1, 1), (300, 1, 1)),
                                      ((1, 90, 100), (1, 12, 12)), ((90, 1, 100), (12, 1, 12)), ((90, 100, 1), (12, 12, 1)),
                                      ((2, 3, 1500), (9, 9, 60)), ((3, 1500, 2), (2, 60, 9)), ((1500, 2, 3), (60, 1, 3))])
def test_equals_exact_selection(dims, rad):
    wl = _wl(dims, rad)
    a = H.engine_cont(0, wl, precision=0)
    b = H.engine_cont(0, wl, precision=0, flags=W.FLAG_EXACT_SEARCH)
    assert a["stats"]["prefilter_active"] == 1.0
    for key in ("status", "est", "var", "data", "mask"):
        np.testing.assert_array_equal(a[key], b[key])


def test_a_column_takes_no_longer_than_a_row():
    def ms(dims, rad):
        wl = _wl(dims, rad)
        H.engine_cont(0, wl)
        return float(np.median([H.engine_cont(0, wl)["stats"]["search_kernel_ms"] for _ in range(7)]))
    n, r = 400000, 300
    row, column = ms((n, 1, 1), (r, 1, 1)), ms((1, 1, n), (1, 1, r))
    assert column <= 2.0 * row
