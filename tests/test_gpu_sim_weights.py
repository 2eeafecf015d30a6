"""The simulation and cokriging solves on the FP64 tensor instruction (weights
solved ahead of the levels, sim_weights.cu; a target a warp, cokriging.cu)
against the CPU oracle, at neighbour limits on every edge of the 8x8 blocks and
over more nodes than one chunk of weights holds. The bars are those of the
simulations and of cokriging: masks and statuses identical, SGS values
bit-identical on 99 % of the cells and within 1e-4 everywhere, SIS categories
identical, cokriging bit-identical on 99 % and within 1e-5."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu

EXP = WL.CovSpec(WL.EXPONENTIAL, (12.0, 9.0, 7.0), (30.0, 0.0, 0.0), 1.0, 0.05)


def _grid(dims, points, seed=4):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, points, replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(points).astype(np.float32)
    mask[idx] = 1
    return data, mask


def _sgs_matches(dims, data, mask, cov, rad, k, kind):
    od, om, ost = O.sgs(dims, data, mask, cov, rad, k, 77, kind=kind)
    e = H.engine_sgs(dims, data, mask, cov, rad, k, 77, kind=kind)
    np.testing.assert_array_equal(e["mask"], om)
    sim = ost >= 0
    np.testing.assert_array_equal(e["status"][sim], ost[sim].astype(np.int8))
    same = e["data"].view(np.uint32) == od.view(np.uint32)
    assert same.mean() >= 0.99
    assert np.abs(e["data"].astype(np.float64) - od).max() <= 1e-4 * max(1.0, float(np.abs(od).max()))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32])
def test_sgs_neighbour_limits(kind, k):
    dims = (17, 13, 9)
    data, mask = _grid(dims, 60)
    _sgs_matches(dims, data, mask, EXP, (12, 9, 7), k, kind)


def test_sgs_over_several_chunks():
    """1.18 M simulated nodes of 32 neighbours: more than the weights of one chunk."""
    dims = (120, 110, 90)
    data, mask = _grid(dims, 9000)
    cov = WL.CovSpec(WL.SPHERICAL, (9.0, 9.0, 5.0), (0.0, 0.0, 0.0), 1.0, 0.1)
    _sgs_matches(dims, data, mask, cov, (9, 9, 5), 32, 1)


@pytest.mark.parametrize("ks", [(32, 1, 8, 9, 17), (24, 24, 24, 24, 24), (7, 32), (16, 25, 31)])
@pytest.mark.parametrize("corr", [False, True])
def test_sis_neighbour_limits(ks, corr):
    dims = (19, 14, 8)
    m = len(ks)
    rng = np.random.default_rng(6)
    data, mask = _grid(dims, 90)
    cats = np.zeros(len(data), np.uint8)
    cats[mask == 1] = rng.integers(0, m, int(mask.sum()))
    covs = [WL.CovSpec(WL.SPHERICAL, (9.0 + c, 8.0, 5.0), (0.0, 0.0, 0.0), 1.0, 0.1) for c in range(m)]
    rads = [(9 + c, 8, 5) for c in range(m)]
    marg = [1.0 / m] * m
    means = [np.clip(0.2 + 0.05 * c + 0.1 * rng.random(len(data)), 0, 1).astype(np.float32) for c in range(m)]
    kw = dict(means=means if corr else None)
    od, om, ost = O.sis(dims, cats, mask, covs, rads, list(ks), marg, 9, correlogram=corr, **kw)
    e = H.engine_sis(dims, cats, mask, covs, rads, list(ks), marg, 9, corr=corr, **kw)
    np.testing.assert_array_equal(e["mask"], om)
    np.testing.assert_array_equal(e["data"], od)
    sim = ost >= 0
    np.testing.assert_array_equal(e["status"][sim], ost[sim].astype(np.int8))


@pytest.mark.parametrize("k", [1, 7, 8, 9, 16, 17, 24, 25, 31, 32])
def test_cokriging_neighbour_limits(k):
    import test_gpu_cokriging as T
    dims = (17, 13, 9)
    data, mask = _grid(dims, 60)
    rng = np.random.default_rng(3)
    second = (0.6 * np.where(mask == 1, data, 0) + rng.standard_normal(len(data))).astype(np.float32)
    x = {"dims": dims, "pdata": data, "pmask": mask, "sdata": second, "smask": (rng.random(len(data)) < 0.5).astype(np.uint8),
         "cov": EXP, "cov2": None, "rad": (12, 9, 7), "k": k, "pm": 0.1, "sm": -0.2, "sv": 1.3, "corr": 0.6}
    out, om, st = T._run_ex(x, 1)
    ref, rom, rst = T._oracle(x, 1)[:3]
    np.testing.assert_array_equal(om, rom)
    tgt = mask == 0
    np.testing.assert_array_equal(st[tgt], np.asarray(rst)[tgt].astype(np.int8))
    T._close(out, ref, k)
