"""Rounding of the FP64 solves: the errors of estimates and variances against the
oracle's solves in 80 bits, next to those of its solves in 64 (a Cholesky
substitution in the neighbours' order).

Fused operations leave less error than the oracle's separate ones, and another order
of the same operations gives another sample of the same errors, whose root mean
square over 2,000 cells is within a few per cent of the first's. What multiplies them
(an order of unknowns, or explicit inverses, whose blocks are ill conditioned) exceeds
it by its factor. The bound is 1.25 times the 64-bit solve's error; 1.5 times for
exponential models, whose errors are the last roundings of the result."""
import numpy as np
import pytest

import helpers as H
import oracle as O
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu


def _rms(a, b):
    return float(np.sqrt(np.mean((a - b) ** 2)))


@pytest.mark.parametrize("cov_type,ranges,azimuth,nugget,density,k", [
    (WL.GAUSSIAN, (20, 15, 6), 30.0, 0.05, 0.01, 12), (WL.GAUSSIAN, (20, 15, 6), 30.0, 0.01, 0.01, 16),
    # beyond 16 neighbours: the sharing solves
    (WL.GAUSSIAN, (20, 15, 6), 30.0, 0.05, 0.01, 32), (WL.GAUSSIAN, (18, 18, 6), 0.0, 0.05, 0.015, 24),
    (WL.GAUSSIAN, (20, 15, 6), 30.0, 0.2, 0.02, 40), (WL.SPHERICAL, (18, 18, 6), 0.0, 0.0, 0.015, 24),
    (WL.EXPONENTIAL, (30, 15, 6), 30.0, 0.0, 0.01, 32),
])
def test_error_is_that_of_a_substitution(cov_type, ranges, azimuth, nugget, density, k):
    dims = (72, 64, 48)
    n = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(3)
    idx = rng.choice(n, int(n * density), replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = np.exp(0.5 * rng.standard_normal(len(idx))).astype(np.float32)
    mask[idx] = 1
    cov = WL.CovSpec(cov_type, tuple(float(r) for r in ranges), (azimuth, 0.0, 0.0), 1.0, nugget)
    wl = WL.Workload("rounding", dims, data, mask, cov, ranges, k)
    nodes = np.sort(rng.choice(np.flatnonzero(mask == 0), 2000, replace=False)).astype(np.int32)
    # simple kriging: its covariances are the same host table on every side
    args = ("port", 1, dims, data, mask, cov, ranges, k)
    exact, plain = (O.krige_nodes(*args, mean=1.0, nodes=nodes, precision=p) for p in (1, 0))
    e = H.engine_cont(1, wl, precision=0, mean=1.0)
    ok = exact["status"] == 0
    assert ok.sum() >= 1900
    bound = 1.5 if cov_type == WL.EXPONENTIAL else 1.25
    for name in ("est", "var"):
        want = exact[name][ok]
        assert _rms(e[name][nodes][ok], want) <= bound * _rms(plain[name][ok], want), name
