"""Batched adjoint with more factored integrals than warps: an integral's
value and gradients do not depend on where in a batch it stands, beside
factored and node-by-node integrals of other families and dimensions."""
import numpy as np
import pytest
import torch

import torchquad_gb300 as tq
from torchquad_gb300 import batch as B

pytestmark = pytest.mark.gpu


def workload(n, max_dim):
    rng = np.random.default_rng(n + max_dim)
    fs, rules, ns, doms = [], [], [], []
    for i in range(n):
        d = 1 + int(rng.integers(max_dim))
        kind = int(rng.integers(5))
        a = rng.uniform(0.2, 2.0, d).tolist()
        if kind == 0:
            f = tq.ExpSum(d, a=a, b=0.1)
        elif kind == 1:
            f = tq.GaussianPeak(d, a=a, u=rng.uniform(0.0, 1.0, d).tolist())
        elif kind == 2:
            f = tq.Oscillatory(d, a=a, b=float(rng.uniform()))
        elif kind == 3:
            f = tq.SumSin(d, a=a)
        else:  # outside the factored form's range: node by node
            f = tq.ExpSum(d, a=[400.0 / d] * d, b=-600.0)  # at most e^0
        per = 5 if d > 3 else 9
        fs.append(f)
        rules.append(["trapezoid", "simpson", "boole", "gausslegendre"][int(rng.integers(4))])
        ns.append(per**d)
        doms.append([[0.0, float(rng.uniform(0.5, 1.5))] for _ in range(d)])
    return fs, rules, ns, doms


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,max_dim", [(1, 1), (9, 4), (305, 4), (2433, 4), (1217, 8)])
def test_integrals_do_not_depend_on_their_place(n, max_dim, dtype, cuda):
    fs, rules, ns, doms = workload(n, max_dim)
    bg = B.BatchedGrid(dtype=dtype)
    vals, gdom, gpar = bg.adjoint(bg.plan(fs, rules, ns, doms), max_dim=max_dim)
    doff = np.cumsum([0] + [2 * f.dim for f in fs])
    poff = np.cumsum([0] + [2 + 2 * f.dim for f in fs])
    some = sorted(set(np.linspace(0, n - 1, 25).astype(int).tolist()))
    for i in some:
        v, gd, gp = bg.adjoint(bg.plan(fs[i : i + 1], rules[i : i + 1], ns[i : i + 1], doms[i : i + 1]),
                               max_dim=max_dim)
        assert torch.equal(v[0], vals[i])
        assert torch.equal(gd, gdom[doff[i] : doff[i + 1]])
        assert torch.equal(gp, gpar[poff[i] : poff[i + 1]])
    assert torch.isfinite(vals).all() and torch.isfinite(gdom).all() and torch.isfinite(gpar).all()
