"""GPU: the batched adjoint with several integrals to a warp, of all families
and rules and beside node-by-node ones, against the numpy oracle."""
import numpy as np
import pytest
import torch

from oracle import grad as OGR
from torchquad_gb300 import batch as B

from .test_batch_adjoint_places_gpu import workload
from .test_separable_gpu import RULES, _assert_gradients

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,max_dim", [(9, 4), (2433, 4), (1217, 8)])
def test_rounds_match_oracle(n, max_dim, cuda):
    fs, rules, ns, doms = workload(n, max_dim)
    bg = B.BatchedGrid(dtype=torch.float64)
    plan = bg.plan(fs, rules, ns, doms)
    vals, gdom, gpar = (x.cpu().numpy() for x in bg.adjoint(plan, max_dim=max_dim))
    for i in sorted(set(np.linspace(0, n - 1, 150).astype(int).tolist())):
        d, f = plan.desc_np[i], fs[i]
        want = OGR.value_and_grad(f.family, f.params_numpy(), RULES[rules[i]][1], f.dim, int(d["n"]), doms[i])
        got = (vals[i], gdom[d["dom_off"]:d["dom_off"] + 2 * f.dim], gpar[d["par_off"]:d["par_off"] + 2 + 2 * f.dim])
        # the bound of the gradient tests; exponents up to 600 cost 600 roundings
        _assert_gradients(got, want, 1e-10, (i, rules[i], f.family, f.dim))
