"""GPU: VEGAS runs of built-in integrands that are infinite or undefined end
within their budget, with a result that is not finite or the error of a map
without finite edges (each cube keeps its two points: the variances that would
set their number are not numbers)."""
import math

import pytest
import torch

import torchquad_gb300 as tq
from torchquad_gb300.vegas_batch import VegasBatch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("c", [math.inf, math.nan])
@pytest.mark.parametrize("dim,N", [(1, 3000), (2, 20_000), (6, 5000)])  # 30, 14^2 and 1 cubes
def test_run_ends(dim, N, c, dtype, cuda):
    dom = torch.tensor([[0.0, 1.0]] * dim, dtype=dtype, device=cuda)
    f, good = tq.ExpSum(dim, c=c), tq.ExpSum(dim, a=0.5)
    v = tq.VEGAS()
    plain = {"use_grid_improve": False, "use_warmup": False}
    got = v.integrate(f, dim, N=N, integration_domain=dom, seed=1, **plain)
    assert not math.isfinite(got.item())
    assert 5 <= v.it <= 20 and 0 < v._nr_of_fevals <= 2 * N
    vb = VegasBatch([f, good, f], [N, N, N], dtype=dtype, **plain)
    res = [float(x) for x in vb.integrate(domains=[[[0.0, 1.0]] * dim] * 3, seeds=[1, 2, 3])]
    want = (2.0 * (math.exp(0.5) - 1.0)) ** dim
    assert not math.isfinite(res[0]) and not math.isfinite(res[2]) and abs(res[1] - want) < 0.1 * want
    with pytest.raises(RuntimeError, match="infinite edges"):
        v.integrate(f, dim, N=N, integration_domain=dom, seed=1)
