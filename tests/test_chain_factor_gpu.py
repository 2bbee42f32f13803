"""GPU: fp64 rows of one dimension with small factors c, whose nodes start far
below their largest: c joins the sum at its end, so that c times the first
node's value may be below the range of doubles."""
import numpy as np
import pytest
import torch

import torchquad_gb300 as tq
from oracle import grid as OG
from oracle import integrands as OI
from torchquad_gb300 import batch as B

pytestmark = pytest.mark.gpu

RULES = {"trapezoid": OG.TRAPEZOID, "simpson": OG.SIMPSON, "boole": OG.BOOLE}


@pytest.mark.parametrize("n", [125, 4001])
def test_small_factor(n, cuda):
    fs = [tq.ExpSum(1, a=1150.0, b=-575.0, c=1e-100), tq.ExpSum(1, a=-1150.0, b=575.0, c=-1e-90),
          tq.GaussianPeak(1, a=1600.0, u=0.5, c=1e-280), tq.GaussianPeak(1, a=1600.0, u=0.5, c=3e280)]
    cases = [(f, r) for f in fs for r in RULES]
    dom = [[0.0, 1.0]]
    got = B.integrate_batch([f for f, _ in cases], [r for _, r in cases], [n] * len(cases), [dom] * len(cases),
                            dtype=torch.float64).cpu().numpy()
    for g, (f, r) in zip(got, cases):
        want = OG.integrate(lambda x: OI.evaluate(f.family, f.params_numpy(), x), RULES[r], 1, n, np.asarray(dom))
        assert abs(g - want) <= 1e-12 * abs(want), (f.family, r, g, want)
