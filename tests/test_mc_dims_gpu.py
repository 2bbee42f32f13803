"""GPU: fused Monte Carlo of every dimension it is compiled for (and beyond),
at counts that end inside a thread's group of points, against the numpy
oracle on the same Philox draws."""
import numpy as np
import pytest
import torch

import torchquad_gb300 as tq
from oracle import integrands as OI
from oracle import mc as OM
from oracle import philox as OP

pytestmark = pytest.mark.gpu


def family(name, dim):
    a = [0.3 + 0.2 * k for k in range(dim)]
    return {"exp": tq.ExpSum(dim, a=[(-1.0) ** k * v for k, v in enumerate(a)], b=0.2, c=1.3),
            "gauss": tq.GaussianPeak(dim, a=a, u=[0.4 - 0.05 * k for k in range(dim)], c=0.7),
            "osc": tq.Oscillatory(dim, a=a, b=0.15, c=-1.1),
            "sumsin": tq.SumSin(dim, a=[1.0 + v for v in a], c=0.9)}[name]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("fam", ["exp", "gauss", "osc", "sumsin"])
def test_fused_dimensions_match_oracle(fam, dtype, cuda):
    """Within the rounding of one evaluation: a coordinate, its term and the
    running sum are rounded to 2^-24 (2^-53) each, and the outer function
    carries the sum's absolute error S into its value, S the largest sum of
    the magnitudes that enter it."""
    f32 = dtype == torch.float32
    nd = np.float32 if f32 else np.float64
    eps = 2.0**-24 if f32 else 2.0**-53
    for dim in range(1, 13):
        f = family(fam, dim)
        p = f.params_vector().numpy()
        a, u = p[2:2 + dim], p[2 + dim:]
        dom = [[-0.4 + 0.1 * k, 0.6 + 0.15 * k] for k in range(dim)]
        for n in (1, 2, 3, 4, 7, 255, 1025, 4099):
            got = tq.MonteCarlo().integrate(f, dim, N=n, integration_domain=torch.tensor(dom, dtype=dtype, device=cuda),
                                            seed=0x1_2345_6789 + n).item()
            r = OP.uniform(0x1_2345_6789 + n, 0, 0, n * dim, nd).reshape(n, dim)
            box = np.array(dom, dtype=nd)
            want = float(OM.integrate(lambda x: OI.evaluate(f.family, p, x), dim, n, box, r))
            x = np.abs(r * (box[:, 1] - box[:, 0]) + box[:, 0]).astype(np.float64) + 1.0
            S = float((np.abs(a) * (x + np.abs(u)) ** 2).sum(axis=1).max()) + 2.0
            top = float(np.abs(OI.evaluate(f.family, p, (r * (box[:, 1] - box[:, 0]) + box[:, 0]))).max())
            top = max(top, abs(float(p[0])) if f.family in (OI.OSCILLATORY, OI.SUM_SIN) else 0.0)
            tol = 8.0 * eps * (1.0 + S) * top * float(np.prod(box[:, 1] - box[:, 0]))
            assert abs(got - want) <= tol, (dim, n, got, want, tol)
