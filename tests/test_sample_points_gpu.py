"""GPU: Monte Carlo points by one kernel against the torch operations they
replace (u * (b - a) + a on the same draws), and the calls that stay with
torch operations."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

import torchquad_gb300 as tq
from torchquad_gb300.integration.rng import RNG

pytestmark = pytest.mark.gpu


def by_torch(N, domain, seed):
    u = RNG(seed=seed).uniform([N, domain.shape[0]], domain.dtype)
    start = domain[:, 0]
    return u * (domain[:, 1] - start) + start


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [1, 2, 3, 5, 7, 16])
def test_points_equal_torch_operations(dim, dtype, cuda):
    dom = torch.tensor([[-0.7 + 0.3 * k, 0.9 + 0.41 * k] for k in range(dim)], dtype=dtype, device=cuda)
    wide = torch.stack([dom, dom + 1.0], dim=2)[:, :, 0]  # the same bounds, strided
    assert not wide.is_contiguous()
    for N in (0, 1, 2, 3, 255, 1001):
        for d in (dom, wide):
            rng = RNG(seed=11)
            got = tq.MonteCarlo().calculate_sample_points(N, d, rng=rng)
            assert torch.equal(got, by_torch(N, dom, 11))
            assert rng.offset == RNG.blocks_for(N * dim, dtype)


def test_derivatives_stay_with_torch_operations(cuda):
    dom = torch.tensor([[0.0, 2.0], [1.0, 3.0]], dtype=torch.float64, device=cuda)
    leaf = dom.clone().requires_grad_()
    pts = tq.MonteCarlo().calculate_sample_points(9, leaf, seed=4)
    assert pts.requires_grad and torch.equal(pts.detach(), by_torch(9, dom, 4))
    with fwAD.dual_level():
        t = torch.ones_like(dom)
        pts = tq.MonteCarlo().calculate_sample_points(9, fwAD.make_dual(dom, t), seed=4)
        assert fwAD.unpack_dual(pts).tangent is not None
    half = tq.MonteCarlo().calculate_sample_points(9, dom.half(), seed=4)
    assert half.dtype == torch.float16
