"""The solves that share one factorisation between neighbouring cells, at sizes
that reach them: a bucket shares from 256 systems a multiprocessor (17 to 32
neighbours) or 128 (33 to 64), which every test asserts.

Against the CPU oracle: statuses identical, estimates and variances within 1e-10
(normwise; condition numbers stay below 64 sill / nugget = 1,280, so FP64 rounding
in any order of elimination stays below 1e-12)."""
import numpy as np
import pytest
import torch

import helpers as H
import oracle as O
from geo_bsd import hpgl_wrap as W
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu


def _wl(dims, informed, cov, rad, k, seed=7):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, int(n * informed), replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    return WL.Workload("groups", dims, data, mask, cov, rad, k)


def _shares(stats, bucket):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert stats["bucket_items_%d" % bucket] >= (256 if bucket == 2 else 128) * sms


def _check(wl, kind, precision=0, tol=1e-10):
    _, om, oest, ovar, ost = O.cont_grid(kind, wl.dims, wl.data, wl.mask, wl.cov, wl.radiuses, wl.max_neighbours)
    e = H.engine_cont(kind, wl, precision=precision)
    unk = wl.mask == 0
    np.testing.assert_array_equal(e["status"][unk], ost[unk].astype(np.int8))
    np.testing.assert_array_equal(e["mask"], om)
    ok = unk & (ost == 0)
    assert H.rel_err(e["est"][ok], oest[ok]) <= tol
    assert H.rel_err(e["var"][ok], ovar[ok]) <= tol
    return e["stats"]


def _tile_groups(wl, kind, tiles):
    """Common neighbours of the uninformed cells of 2x2x2 tiles: per tile, of all of
    them and of the first half, against the number that a group has to share."""
    nx, ny, nz = wl.dims
    out = []
    for t in tiles:
        x0, y0, z0 = 2 * (t % (nx // 2)), 2 * (t // (nx // 2) % (ny // 2)), 2 * (t // (nx // 2) // (ny // 2))
        cells = [x0 + x + nx * (y0 + y + ny * (z0 + z)) for z in (0, 1) for y in (0, 1) for x in (0, 1)]
        cells = [c for c in cells if not wl.mask[c]]
        if len(cells) < 4:
            continue
        r = O.krige_nodes("port", kind, wl.dims, wl.data, wl.mask, wl.cov, wl.radiuses, wl.max_neighbours,
                          nodes=np.array(cells, np.int32))
        sets = [set(row[:c]) for row, c in zip(r["idx"], r["count"])]
        if min(r["count"]) <= 16 or max(r["count"]) > 32:
            continue

        def fits(g):
            return len(set.intersection(*sets[:g])) >= 8 * ((max(r["count"][:g]) + 7) // 8 - 1)
        out.append((fits(len(cells)), fits((len(cells) + 1) // 2)))
    return out


@pytest.mark.parametrize("kind", [0, 1])
def test_groups_that_fail_and_are_halved(kind):
    """Few common neighbours: most tiles' cells have too few of them all together, some
    enough by halves, others not even then."""
    cov = WL.CovSpec(WL.EXPONENTIAL, (12.0, 12.0, 12.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    wl = _wl((52, 48, 30), 0.03, cov, (6, 6, 6), 28)
    groups = _tile_groups(wl, kind, range(0, 26 * 24 * 15, 31))
    assert sum(not whole and half for whole, half in groups) >= 10
    assert sum(not half for _, half in groups) >= 10
    _shares(_check(wl, kind), 2)


@pytest.mark.parametrize("dims,rad", [((96, 80, 60), (1, 1, 1)), ((60, 60, 40), (2, 1, 3))])
@pytest.mark.parametrize("kind", [0, 1])
def test_small_radiuses_shared(kind, dims, rad):
    """The pair table of a small radius limits how far apart grouped cells may be: two
    thirds of the cells informed, so that its few cells hold 17 neighbours."""
    cov = WL.CovSpec(WL.EXPONENTIAL, (30.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    _shares(_check(_wl(dims, 0.66, cov, rad, 27), kind), 2)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("k", [19, 32, 50])
def test_long_thin_grid_shared(kind, k):
    cov = WL.CovSpec(WL.EXPONENTIAL, (600.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    _shares(_check(_wl((5301, 3, 3), 0.07, cov, (60, 3, 3), k), kind), 2 if k <= 32 else 3)


@pytest.mark.parametrize("np_,k,informed", [(32, 32, 0.05), (64, 50, 0.05)])
@pytest.mark.parametrize("kind", [0, 1])
def test_refined_option_shared(kind, np_, k, informed):
    """FP32-refined keys set to SHARE: the FP64 solves, nothing escalated."""
    cov = WL.CovSpec(WL.EXPONENTIAL, (12.0, 9.0, 7.0), (30.0, 0.0, 0.0), 1.0, 0.05)
    wl = _wl((53, 47, 19), informed, cov, (12, 9, 7), k)
    prev = W.solve_variant(np_, cov.cov_type, W.FP32_REFINED, W.VARIANT_SHARE)
    try:
        s = _check(wl, kind, precision=W.FP32_REFINED)
    finally:
        W.solve_variant(np_, cov.cov_type, W.FP32_REFINED, prev)
    _shares(s, 2 if np_ == 32 else 3)
    assert s["escalated_cells"] == 0


@pytest.mark.parametrize("k,bucket,nugget", [(30, 2, 0.75), (52, 3, 0.82)])
def test_indefinite_systems_shared(k, bucket, nugget):
    """Simple kriging whose box cuts the covariance off at a fifth of its range: some
    systems are indefinite, and fail in any order of elimination; the others' solves
    go through. Cells whose smallest eigenvalue is within 1e-6 of zero are left out."""
    rad = (6, 6, 6)
    cov = WL.CovSpec(WL.GAUSSIAN, (30.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, nugget)
    wl = _wl((50, 46, 24), 0.05, cov, rad, k)
    nx, ny, _ = wl.dims
    nodes = np.flatnonzero(wl.mask == 0).astype(np.int32)
    r = O.krige_nodes("port", 1, wl.dims, wl.data, wl.mask, cov, rad, k, mean=0.0, nodes=nodes)
    e = H.engine_cont(1, wl, precision=0, mean=0.0)
    _shares(e["stats"], bucket)
    clear = np.zeros(len(nodes), bool)
    for n in np.unique(r["count"]):
        at = np.flatnonzero(r["count"] == n)
        if n == 0:
            clear[at] = True
            continue
        p = r["idx"][at, :n]
        xyz = np.stack([p % nx, p // nx % ny, p // (nx * ny)], -1)
        d = xyz[:, :, None, :] - xyz[:, None, :, :]
        A = (1 - nugget) * np.exp(-3 * (d * d).sum(-1) / 900.0) * (np.abs(d) <= np.array(rad)).all(-1)
        A += nugget * np.eye(n)
        clear[at] = np.abs(np.linalg.eigvalsh(A)).min(-1) > 1e-6
    failed = r["status"] == 2
    assert clear.mean() > 0.9 and (failed & clear).sum() > 1000 and (~failed & clear).sum() > 1000
    np.testing.assert_array_equal(e["status"][nodes][clear], r["status"][clear].astype(np.int8))
    ok = clear & (r["status"] == 0)
    assert H.rel_err(e["est"][nodes][ok], r["est"][ok]) <= 1e-8  # condition numbers below 10^8
