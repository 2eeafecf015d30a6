"""The FP64 solves that share one factorisation between neighbouring cells
(17 to 64 neighbours), and the one-system kernel for the cells that cannot
share, against the CPU oracle: statuses identical, estimates and variances
within 1e-10 (normwise; the systems' condition numbers stay below 64 sill /
nugget = 1,280, so FP64 rounding in any order of elimination stays below 1e-12).

Neighbour limits at every edge of the 8x8 blocks, grids one cell thick in each
direction or cut off inside a tile, radiuses so small that the pair table
limits the tile, data so sparse or so dense that groups split, and the FP32-
refined option, whose larger buckets run the same solves."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import hpgl_wrap as W
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu

EXP = WL.CovSpec(WL.EXPONENTIAL, (12.0, 9.0, 7.0), (30.0, 0.0, 0.0), 1.0, 0.05)
SPH = WL.CovSpec(WL.SPHERICAL, (9.0, 9.0, 9.0), (0.0, 0.0, 0.0), 2.0, 0.2)


def _wl(dims, points, cov, rad, k, seed=7):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, points, replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(points).astype(np.float32)
    mask[idx] = 1
    return WL.Workload("share", dims, data, mask, cov, rad, k)


def _check(wl, kind, precision=0, tol=1e-10):
    od, om, oest, ovar, ost = O.cont_grid(kind, wl.dims, wl.data, wl.mask, wl.cov, wl.radiuses, wl.max_neighbours)
    e = H.engine_cont(kind, wl, precision=precision)
    unk = wl.mask == 0
    np.testing.assert_array_equal(e["status"][unk], ost[unk].astype(np.int8))
    np.testing.assert_array_equal(e["mask"], om)
    ok = unk & (ost == 0)
    assert H.rel_err(e["est"][ok], oest[ok]) <= tol
    assert H.rel_err(e["var"][ok], ovar[ok]) <= tol
    return e["stats"]


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("k", [17, 24, 25, 31, 32, 33, 40, 41, 48, 56, 57, 64])
def test_neighbour_limits(kind, k):
    s = _check(_wl((37, 31, 13), 750, EXP, (12, 9, 7), k), kind)
    assert s["bucket_items_%d" % (2 if k <= 32 else 3)] > 64 * 148  # below that, no sharing
    _check(_wl((13, 11, 7), 50, EXP, (12, 9, 7), k), kind)


@pytest.mark.parametrize("dims,points,rad", [
    ((15001, 1, 1), 1500, (200, 3, 3)), ((1, 15001, 1), 1500, (3, 200, 3)), ((1, 1, 15001), 1500, (3, 3, 200)),
    ((3, 2003, 2), 900, (4, 60, 2)), ((1301, 3, 3), 900, (60, 3, 3)), ((9, 7, 201), 900, (6, 6, 12)),
])
@pytest.mark.parametrize("kind", [0, 1])
def test_thin_and_ragged_grids(kind, dims, points, rad):
    cov = WL.CovSpec(WL.EXPONENTIAL, tuple(float(v) for v in rad), (0.0, 0.0, 0.0), 1.0, 0.05)
    for k in (19, 32, 50):
        _check(_wl(dims, points, cov, rad, k), kind)


@pytest.mark.parametrize("rad", [(1, 1, 1), (2, 1, 3), (2, 2, 2), (3, 1, 1)])
@pytest.mark.parametrize("kind", [0, 1])
def test_small_radiuses(kind, rad):
    """The pair table of a small radius limits how far apart grouped cells may be."""
    cov = WL.CovSpec(WL.EXPONENTIAL, (30.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    _check(_wl((37, 30, 19), 14000, cov, rad, 27), kind)


@pytest.mark.parametrize("points", [300, 9000])
def test_sparse_and_dense_data(points):
    """Neighbour counts that vary from cell to cell; neighbourhoods of a few
    cells, of which the next cell has hardly any."""
    _check(_wl((51, 47, 17), points, SPH, (9, 9, 9), 32), 0)
    _check(_wl((51, 47, 17), points, SPH, (9, 9, 9), 60), 1)


@pytest.mark.parametrize("np_,k", [(32, 32), (64, 50)])
def test_refined_option_runs_the_shared_solve(np_, k):
    wl = _wl((37, 31, 13), 750, EXP, (12, 9, 7), k)
    prev = W.solve_variant(np_, wl.cov.cov_type, W.FP32_REFINED, W.VARIANT_SHARE)
    try:
        s = _check(wl, 0, precision=W.FP32_REFINED, tol=1e-10)
        assert s["escalated_cells"] == 0
    finally:
        W.solve_variant(np_, wl.cov.cov_type, W.FP32_REFINED, prev)
    with pytest.raises(ValueError):
        W.solve_variant(16, 1, W.FP32_REFINED, W.VARIANT_SHARE)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("k", [17, 24, 25, 31, 32, 33, 40, 41, 48, 56, 57, 64])
def test_neighbour_limits_shared(kind, k):
    """Enough systems for the sharing kernel whatever k (fewer go one by one)."""
    s = _check(_wl((53, 47, 19), 2400, EXP, (12, 9, 7), k), kind)
    assert s["bucket_items_%d" % (2 if k <= 32 else 3)] >= 256 * 148


@pytest.mark.parametrize("dims,points,rad", [
    ((45001, 1, 1), 4500, (200, 3, 3)), ((1, 45001, 1), 4500, (3, 200, 3)), ((1, 1, 45001), 4500, (3, 3, 200)),
    ((3, 7003, 2), 2900, (4, 60, 2)), ((4501, 3, 3), 2900, (60, 3, 3)), ((9, 7, 701), 2900, (6, 6, 12)),
    ((47, 40, 23), 40000, (1, 1, 1)), ((47, 43, 23), 44000, (2, 1, 3)),
])
@pytest.mark.parametrize("kind", [0, 1])
def test_thin_and_ragged_grids_shared(kind, dims, points, rad):
    cov = WL.CovSpec(WL.EXPONENTIAL, tuple(10.0 * v for v in rad), (0.0, 0.0, 0.0), 1.0, 0.05)
    for k in (19, 32, 50):
        _check(_wl(dims, min(points, dims[0] * dims[1] * dims[2] // 10), cov, rad, k), kind)
