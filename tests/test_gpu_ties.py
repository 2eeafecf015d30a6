"""Ties at the k-th neighbour: the partitions of std::sort replayed by a warp pick
the members of a tie group that the CPU oracle's std::sort picks.

Points on lattices share most of their covariances, so nearly every cell ties. The
lists are shorter and longer than a partition's block of 32, than std::sort's last
16, and up to thousands; the neighbour counts lie at the front, in the middle and
at 64. Sets are whole numbers: they are equal or the replay is wrong."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 6, 20, 33, 64])
@pytest.mark.parametrize("step,rad,keep", [((3, 3, 4), (15, 15, 15), 1.0), ((3, 3, 4), (15, 15, 15), 0.6),
                                           ((4, 4, 4), (9, 9, 9), 1.0), ((6, 6, 4), (12, 8, 6), 0.8),
                                           ((9, 9, 2), (12, 12, 3), 0.5)])
def test_tied_sets_equal_the_oracles(step, rad, keep, k):
    dims = (48, 45, 24)
    rng = np.random.default_rng(17)
    xs, ys, zs = np.meshgrid(*[np.arange(0, d, s) for d, s in zip(dims, step)], indexing="ij")
    idx = (xs + dims[0] * (ys + dims[1] * zs)).ravel()
    idx = idx[rng.random(len(idx)) < keep]
    n = dims[0] * dims[1] * dims[2]
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    cov = WL.CovSpec(WL.EXPONENTIAL, (30.0, 30.0, 30.0), (0.0, 0.0, 0.0), 1.0, 0.05)
    wl = WL.Workload("ties", dims, data, mask, cov, rad, k)
    nodes = np.sort(rng.choice(np.flatnonzero(mask == 0), 200, replace=False))
    got, cnt, path = H.engine_neighbours(1, wl, nodes)
    want = O.krige_nodes("port", 1, dims, data, mask, cov, rad, k, nodes=nodes)
    np.testing.assert_array_equal(cnt, want["count"])
    np.testing.assert_array_equal(np.sort(got, 1), np.sort(want["idx"][:, :k], 1))
