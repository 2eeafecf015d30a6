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
