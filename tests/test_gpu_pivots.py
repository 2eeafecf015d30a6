"""The FP64 solves' reciprocal of a pivot, against CUDA's correctly rounded one over
every exponent that the pivot check passes, and that check at its edges.

The iteration leaves e^3 < 2^-57 of the result beside the half place of its last
operation, so it gives the correctly rounded number or one next to it. The functions
are compiled from the header here; systems with pivots outside of the range go
through the library."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

import helpers as H
from geo_bsd import workloads as WL

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "mma64.cuh"
__global__ void k(int n, const double *d, double *own, double *rn, double *e0, unsigned char *fail)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double x0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x0) : "d"(d[i]));
    own[i] = hb::pivot_inverse(d[i]);
    rn[i] = __drcp_rn(d[i]);
    e0[i] = fma(-d[i], x0, 1.0);
    fail[i] = (hb::pivot_fails<false>(d[i]) ? 1 : 0) | (hb::pivot_fails<true>(d[i]) ? 2 : 0);
}
extern "C" int run(int n, const double *d, double *own, double *rn, double *e0, unsigned char *fail)
{
    k<<<(n + 255) / 256, 256>>>(n, d, own, rn, e0, fail);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc here")
    work = tmp_path_factory.mktemp("pivots")
    (work / "p.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-I", os.path.join(ROOT, "hpgl-reborn_b200", "csrc"), "-o", str(work / "p.so"),
                    str(work / "p.cu")], check=True)
    fn = C.CDLL(str(work / "p.so")).run
    fn.argtypes = [C.c_int] + [C.c_void_p] * 5

    def call(values):
        d = torch.from_numpy(np.ascontiguousarray(values)).cuda()
        own, rn, e0 = (torch.empty_like(d) for _ in range(3))
        fail = torch.empty(len(d), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert fn(len(d), *(t.data_ptr() for t in (d, own, rn, e0, fail))) == 0
        return [t.cpu().numpy() for t in (own, rn, e0, fail)]
    return call


def test_reciprocal_is_within_one_place_of_cudas(run):
    rng = np.random.default_rng(1)
    exponents = np.arange(-1022, 1022)
    m = np.concatenate([rng.integers(0, 1 << 52, (len(exponents), 500)),
                        np.tile([0, 1, 2, (1 << 52) - 1, (1 << 52) - 2, 1 << 51, (1 << 32) - 1, 1 << 32],
                                (len(exponents), 1))], axis=1)
    d = (((exponents + 1023).astype(np.int64) << 52)[:, None] + m).view(np.float64).ravel()
    own, rn, e0, fail = run(d)
    assert not (fail & 1).any()
    assert np.abs(e0).max() < 2.0 ** -19
    assert np.abs(own.view(np.int64) - rn.view(np.int64)).max() <= 1


def test_check_passes_the_reciprocals_domain(run):
    tiny, huge, eps = 2.0 ** -1022, 2.0 ** 1022, 2.0 ** -52
    below = np.nextafter(tiny, 0)
    d = np.array([0.0, -0.0, -1.0, -tiny, 5e-324, 2.0 ** -1042, below, tiny, np.nextafter(eps, 0), eps, 1.0,
                  np.nextafter(huge, 0), huge, np.finfo(float).max, np.inf, -np.inf, np.nan])
    _, _, _, fail = run(d)
    with np.errstate(invalid="ignore"):
        np.testing.assert_array_equal(fail & 1, ~((d >= tiny) & (d < huge)))
        np.testing.assert_array_equal(fail >> 1, ~((d >= eps) & (d < huge)))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("sill", [1e-310, 1e308, 1.0])
def test_extreme_sills_solve_or_fail(kind, sill):
    """No estimate that is not a number under a status that says kriged."""
    dims = (40, 36, 12)
    rng = np.random.default_rng(2)
    n = dims[0] * dims[1] * dims[2]
    idx = rng.choice(n, 900, replace=False)
    data = np.full(n, -99.0, np.float32)
    mask = np.zeros(n, np.uint8)
    data[idx] = rng.standard_normal(len(idx)).astype(np.float32)
    mask[idx] = 1
    cov = WL.CovSpec(WL.EXPONENTIAL, (12.0, 12.0, 9.0), (0.0, 0.0, 0.0), sill, 0.0)
    for k in (28, 50):
        e = H.engine_cont(kind, WL.Workload("sill", dims, data, mask, cov, (12, 12, 9), k), mean=0.0)
        ok = (mask == 0) & (e["status"] == 0)
        assert np.isfinite(e["est"][ok]).all() and np.isfinite(e["data"][ok]).all()
        if sill == 1.0:
            assert ok.sum() == (mask == 0).sum()
