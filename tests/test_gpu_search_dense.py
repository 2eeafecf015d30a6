"""Template-path bins that are scanned because their data are dense, beside bins that
the lane-a-cell search takes: estimates against the CPU oracle (1e-10, condition
numbers below 64 sill / nugget = 1,280), and dense data take no longer than data of a
third of the density, whose scans are longer."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu
EXP = WL.CovSpec(WL.EXPONENTIAL, (20.0, 20.0, 10.0), (0.0, 0.0, 0.0), 1.0, 0.05)


def _wl(dims, idx, rad, k):
    n = dims[0] * dims[1] * dims[2]
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = np.random.default_rng(2).standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    return WL.Workload("dense", dims, data, mask, EXP, rad, k)


def _uniform(dims, density):
    n = dims[0] * dims[1] * dims[2]
    return np.random.default_rng(3).choice(n, int(n * density), replace=False)


def _matches(wl, kind):
    _, om, oest, ovar, ost = O.cont_grid(kind, wl.dims, wl.data, wl.mask, wl.cov, wl.radiuses, wl.max_neighbours)
    e = H.engine_cont(kind, wl, precision=0)
    assert e["stats"]["template_cells"] > 0
    unk = wl.mask == 0
    np.testing.assert_array_equal(e["status"][unk], ost[unk].astype(np.int8))
    np.testing.assert_array_equal(e["mask"], om)
    ok = unk & (ost == 0)
    assert H.rel_err(e["est"][ok], oest[ok]) <= 1e-10
    assert H.rel_err(e["var"][ok], ovar[ok]) <= 1e-10


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("density,rad,k", [(0.3, (8, 8, 8), 16), (0.1, (12, 12, 6), 40), (0.5, (5, 5, 5), 8)])
def test_dense_data(kind, density, rad, k):
    dims = (47, 41, 26)
    _matches(_wl(dims, _uniform(dims, density), rad, k), kind)


@pytest.mark.parametrize("kind", [0, 1])
def test_dense_beside_sparse(kind):
    """A dense half (scanned), a sparse one (searched), bins of both around the border."""
    dims = (72, 40, 24)
    idx = _uniform(dims, 0.3)
    x = idx % dims[0]
    idx = idx[(x < 36) | (np.arange(len(idx)) % 40 == 0)]
    _matches(_wl(dims, idx, (8, 8, 8), 20), kind)


def test_dense_data_take_no_longer():
    def ms(density):
        wl = _wl((100, 100, 50), _uniform((100, 100, 50), density), (10, 10, 10), 16)
        H.engine_cont(0, wl)
        return float(np.median([H.engine_cont(0, wl)["stats"]["search_kernel_ms"] for _ in range(7)]))
    assert ms(0.4) <= 1.25 * ms(0.13)
