"""Singular systems on every path: the covariance of a range of 10^20 cells is 1 at
every distance, so each system of two neighbours or more has the pivots 1 and
1 - 1 * 1 = 0, exactly, in any order of elimination. Statuses and what is written in
place of a solution equal the CPU oracle's; every cell ties with every other."""
import numpy as np
import pytest
import torch

import helpers as H
import oracle as O
from geo_bsd import loo as L
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu
ONES = WL.CovSpec(WL.EXPONENTIAL, (1e20, 1e20, 1e20), (0.0, 0.0, 0.0), 1.0, 0.0)


def _grid(dims, points, seed=4):
    rng = np.random.default_rng(seed)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, points, replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(points).astype(np.float32)
    mask[idx] = 1
    return data, mask


# few systems (one a warp) and enough to share
@pytest.mark.parametrize("dims,points", [((17, 13, 9), 60), ((60, 50, 20), 1800)])
@pytest.mark.parametrize("k", [8, 24, 32, 48])
@pytest.mark.parametrize("kind", [0, 1])
def test_kriging(kind, k, dims, points):
    data, mask = _grid(dims, points)
    wl = WL.Workload("ones", dims, data, mask, ONES, (9, 9, 7), k)
    od, om, _, _, ost = O.cont_grid(kind, dims, data, mask, ONES, wl.radiuses, k)
    e = H.engine_cont(kind, wl, precision=0)
    unk = mask == 0
    assert (ost[unk] == 2).mean() > 0.9
    np.testing.assert_array_equal(e["status"][unk], ost[unk].astype(np.int8))
    np.testing.assert_array_equal(e["mask"], om)
    np.testing.assert_array_equal(e["data"][ost == 2], od[ost == 2])


@pytest.mark.parametrize("k", [8, 24, 32])
@pytest.mark.parametrize("kind", [0, 1])
def test_sgs(kind, k):
    dims = (17, 13, 9)
    data, mask = _grid(dims, 60)
    od, om, ost = O.sgs(dims, data, mask, ONES, (6, 6, 5), k, 77, kind=kind)
    e = H.engine_sgs(dims, data, mask, ONES, (6, 6, 5), k, 77, kind=kind)
    sim = ost >= 0
    assert (ost[sim] == 2).mean() > 0.9
    np.testing.assert_array_equal(e["status"][sim], ost[sim].astype(np.int8))
    np.testing.assert_array_equal(e["mask"], om)
    assert np.abs(e["data"] - od).max() <= 1e-5  # draws from N(0, 1): one rounding to float


@pytest.mark.parametrize("ks", [(8, 24, 32), (16, 16)])
def test_sis(ks):
    dims = (17, 13, 9)
    m = len(ks)
    data, mask = _grid(dims, 60)
    cats = np.zeros(len(data), np.uint8)
    cats[mask == 1] = np.random.default_rng(6).integers(0, m, int(mask.sum()))
    args = (dims, cats, mask, [ONES] * m, [(6, 6, 5)] * m, list(ks), [1.0 / m] * m, 9)
    od, om, ost = O.sis(*args)
    e = H.engine_sis(*args)
    sim = ost >= 0
    assert (ost[sim] == 2).mean() > 0.9
    np.testing.assert_array_equal(e["status"][sim], ost[sim].astype(np.int8))
    np.testing.assert_array_equal(e["data"], od)
    np.testing.assert_array_equal(e["mask"], om)


@pytest.mark.parametrize("k", [8, 24, 32])
def test_cokriging(k):
    import test_gpu_cokriging as T
    dims = (17, 13, 9)
    data, mask = _grid(dims, 60)
    rng = np.random.default_rng(3)
    x = {"dims": dims, "pdata": data, "pmask": mask, "sdata": rng.standard_normal(len(data)).astype(np.float32),
         "smask": (rng.random(len(data)) < 0.5).astype(np.uint8), "cov": ONES, "cov2": None, "rad": (9, 9, 7), "k": k,
         "pm": 0.1, "sm": -0.2, "sv": 1.3, "corr": 0.6}
    out, om, st = T._run_ex(x, 1)
    ref, rom, rst = T._oracle(x, 1)[:3]
    tgt = mask == 0
    assert (np.asarray(rst)[tgt] == 2).mean() > 0.9
    np.testing.assert_array_equal(st[tgt], np.asarray(rst)[tgt].astype(np.int8))
    np.testing.assert_array_equal(om, rom)
    np.testing.assert_array_equal(out, ref)


def test_leave_one_out():
    xyz = torch.tensor([[x, y, 0] for x in range(6) for y in range(6)], dtype=torch.int32, device="cuda")
    nb = torch.stack([torch.tensor([j for j in range(36) if j != i][:32]) for i in range(36)]).int().cuda()
    cnt = torch.tensor([0, 1, 2, 8, 9, 24, 31, 32] + [17] * 28, dtype=torch.int32, device="cuda")
    values = torch.arange(36, dtype=torch.float64, device="cuda")
    geom = L.LooGeometry(xyz, values, torch.arange(36, dtype=torch.int32, device="cuda"), nb, cnt, k=32, cov_type=1,
                         nodes=None)
    par = [(torch.eye(3, dtype=torch.float64) * 1e-20).cuda().requires_grad_(True),
           torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True),
           torch.tensor(0.0, dtype=torch.float64, device="cuda", requires_grad=True)]
    z = values.clone().requires_grad_(True)
    zhat, status = L.LooKriging.apply(*par, z, geom, 1e20)
    assert status.cpu().tolist() == [1, 0] + [2] * 34
    assert zhat[2:].abs().max() == 0
    zhat.sum().backward()
    assert all(torch.isfinite(p.grad).all() for p in par + [z])
    assert z.grad.abs().sum() == 1  # the one kriged target's neighbour


def test_sis_over_several_chunks():
    """384,000 nodes of three categories, one with 32 neighbours: more than the
    weights of one chunk (256 MB of 96 weights a node)."""
    dims = (80, 80, 60)
    data, mask = _grid(dims, 4000)
    cats = np.zeros(len(data), np.uint8)
    cats[mask == 1] = np.random.default_rng(6).integers(0, 3, int(mask.sum()))
    cov = WL.CovSpec(WL.SPHERICAL, (9.0, 9.0, 5.0), (0.0, 0.0, 0.0), 1.0, 0.1)
    args = (dims, cats, mask, [cov] * 3, [(9, 9, 5)] * 3, [32, 6, 6], [0.5, 0.3, 0.2], 9)
    od, om, ost = O.sis(*args)
    e = H.engine_sis(*args)
    np.testing.assert_array_equal(e["mask"], om)
    sim = ost >= 0
    np.testing.assert_array_equal(e["status"][sim], ost[sim].astype(np.int8))
    assert (e["data"] == od).mean() >= 0.999  # a draw within rounding of a category's edge may fall beside it
