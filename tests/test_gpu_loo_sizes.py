"""Leave-one-out estimates and gradients at every neighbour count of a block row's
edges, the variogram on the device and on the host: against the dense FP64
reference and autograd.

The factorisations are backward stable in FP64 and the systems' condition stays
below about 32 sill / nugget = 320: 1e-10 for estimates, 1e-8 for gradients
(whose sums over targets cancel by up to a hundred)."""
import pytest
import torch

import loo_reference as R
from geo_bsd import loo as L

pytestmark = pytest.mark.gpu


def _geometry(k, counts, t, seed):
    rng = torch.Generator().manual_seed(seed)
    node = torch.randperm(25 ** 3, generator=rng)[:400]  # no two points in a cell: those systems are singular
    xyz = torch.stack([node % 25, node // 25 % 25, node // 625], 1).int()
    nb = torch.stack([torch.randperm(399, generator=rng)[:k] + 1 for _ in range(t)]).int()
    cnt = torch.tensor([counts[i % len(counts)] for i in range(t)], dtype=torch.int32)
    return xyz, torch.randn(400, generator=rng, dtype=torch.float64), torch.zeros(t, dtype=torch.int32), nb, cnt


@pytest.mark.parametrize("on_device", [True, False])
@pytest.mark.parametrize("k,counts", [(1, [1]), (8, [7, 8, 1]), (16, [9, 16, 15, 3]), (24, [17, 24]), (32, [25, 31, 32, 2])])
@pytest.mark.parametrize("cov_type", [0, 1, 2])
def test_counts(cov_type, k, counts, on_device):
    cpu = _geometry(k, counts, 41, 10 * k + cov_type)
    dev = [x.cuda() for x in cpu]
    geom = L.LooGeometry(*dev, k=k, cov_type=cov_type, nodes=None)
    par = [torch.tensor(v, dtype=torch.float64, requires_grad=True)
           for v in ((9.0, 7.0, 5.0), (20.0, 10.0, -15.0), 1.0, 0.1)]
    ref = [p.detach().clone().requires_grad_(True) for p in par]
    vals, rvals = dev[1].clone().requires_grad_(True), cpu[1].clone().requires_grad_(True)
    M = L.transform_matrix(par[0], par[1])
    model = [x.cuda() for x in (M, par[2], par[3])] if on_device else [M, par[2], par[3]]
    zhat, status = L.LooKriging.apply(*model, vals, geom, 9.0)
    want = R.dense_loo(cpu[0], rvals, cpu[2], cpu[3], cpu[4], cov_type, ref[0], ref[1], ref[2], ref[3])
    assert (status == 0).all()
    assert float((zhat.detach().cpu() - want.detach()).abs().max() / want.detach().abs().max()) <= 1e-10
    if not on_device:
        return  # the gradients of a host variogram live on the host's side of autograd
    (zhat * zhat).sum().backward()
    (want * want).sum().backward()
    for a, b in zip(par + [vals], ref + [rvals]):
        a, b = a.grad.cpu(), b.grad
        assert float((a - b).abs().max()) <= 1e-8 * float(b.abs().max()) + 1e-12
