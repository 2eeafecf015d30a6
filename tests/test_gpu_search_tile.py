"""The one-cell-a-lane neighbour search, whose neighbours stand in candidate
order: bit-identical estimates, variances and statuses to the selection by exact
ranks over every candidate (the same order), and against the CPU oracle where the
template has more offsets than 16-bit positions (rank keys, ties by the template
scan; there the exact run scans the template, so only rounding may differ: 1e-10
normwise, condition numbers below 64 sill / nugget).

Tiles cut at the grid's and the bins' ends, neighbour limits from 1 to 64, bins
beyond the candidates of the first launch, empty bins and sparse data."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import hpgl_wrap as W
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu


def _wl(dims, idx, cov, rad, k, seed=3):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    return WL.Workload("tile", dims, data, mask, cov, rad, k)


def _uniform(dims, points, seed=5):
    return np.random.default_rng(seed).choice(dims[0] * dims[1] * dims[2], points, replace=False)


def _same_as_exact(wl, kind):
    a = H.engine_cont(kind, wl, precision=0)
    b = H.engine_cont(kind, wl, precision=0, flags=W.FLAG_EXACT_SEARCH)
    assert a["stats"]["prefilter_active"] == 1.0 and b["stats"]["prefilter_active"] == 0.0
    for key in ("status", "est", "var", "data", "mask"):
        np.testing.assert_array_equal(a[key], b[key])
    assert a["stats"]["tie_cells"] == b["stats"]["tie_cells"]
    return a


EXP = WL.CovSpec(WL.EXPONENTIAL, (9.0, 7.0, 4.0), (25.0, 0.0, 0.0), 1.0, 0.05)


@pytest.mark.parametrize("k", [1, 4, 12, 20, 32, 33, 64])
@pytest.mark.parametrize("dims,points", [((41, 33, 13), 500), ((41, 33, 13), 30), ((5, 3, 200), 90), ((200, 2, 3), 60)])
def test_equals_exact_selection(dims, points, k):
    _same_as_exact(_wl(dims, _uniform(dims, points), EXP, (9, 7, 4), k), 0)
    _same_as_exact(_wl(dims, _uniform(dims, points), EXP, (9, 7, 4), k), 1)


@pytest.mark.parametrize("rad", [(1, 1, 1), (2, 1, 3), (3, 9, 1)])
def test_small_bins(rad):
    cov = WL.CovSpec(WL.EXPONENTIAL, (30.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    _same_as_exact(_wl((23, 17, 9), _uniform((23, 17, 9), 900), cov, rad, 16), 0)


def test_clustered_points_and_empty_bins():
    """A ball of points beside an empty half: candidate counts from 0 to thousands."""
    dims = (64, 40, 24)
    rng = np.random.default_rng(8)
    p = np.rint(rng.normal((20, 20, 12), 5.0, (2600, 3))).astype(int)
    p = np.unique(p[((p >= 0) & (p < dims)).all(1)], axis=0)
    idx = p[:, 0] + dims[0] * (p[:, 1] + dims[1] * p[:, 2])
    cov = WL.CovSpec(WL.EXPONENTIAL, (12.0, 12.0, 12.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    for k in (8, 40):
        _same_as_exact(_wl(dims, idx, cov, (12, 12, 12), k), 0)


@pytest.mark.parametrize("kind", [0, 1])
def test_templates_past_16_bit_positions(kind):
    """(45, 45, 9) radiuses: more than 65,534 template offsets; one overfull bin
    sends the cells around it to the template path."""
    dims = (60, 56, 20)
    rng = np.random.default_rng(11)
    p = np.rint(rng.normal((20, 20, 9), (9.0, 9.0, 4.0), (1800, 3))).astype(int)
    p = np.unique(p[((p >= 0) & (p < dims)).all(1)], axis=0)
    idx = p[:, 0] + dims[0] * (p[:, 1] + dims[1] * p[:, 2])
    cov = WL.CovSpec(WL.EXPONENTIAL, (45.0, 45.0, 9.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    wl = _wl(dims, idx, cov, (45, 45, 9), 24)
    od, om, oest, ovar, ost = O.cont_grid(kind, wl.dims, wl.data, wl.mask, wl.cov, wl.radiuses, wl.max_neighbours)
    e = H.engine_cont(kind, wl, precision=0)
    assert e["stats"]["template_cells"] > 0
    unk = wl.mask == 0
    np.testing.assert_array_equal(e["status"][unk], ost[unk].astype(np.int8))
    ok = unk & (ost == 0)
    assert H.rel_err(e["est"][ok], oest[ok]) <= 1e-10
    assert H.rel_err(e["var"][ok], ovar[ok]) <= 1e-10
