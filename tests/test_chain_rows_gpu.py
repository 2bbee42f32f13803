"""GPU: batches of one-dimensional fp64 rows around the lengths of their chains
(16 to 128 nodes), with all, some and none of the chains left to direct
evaluation, in tiles that cut rows, against the numpy oracle."""
import numpy as np
import pytest
import torch

import torchquad_gb300 as tq
from oracle import grid as OG
from oracle import integrands as OI
from torchquad_gb300 import batch as B

pytestmark = pytest.mark.gpu

RULES = {"trapezoid": OG.TRAPEZOID, "simpson": OG.SIMPSON, "boole": OG.BOOLE}


@pytest.mark.parametrize("tile,block", [(64, 256), (1000, 128), (32768, 256), (131072, 128)])
@pytest.mark.parametrize("n", [5, 17, 33, 129, 1001, 4097, 33_001])
def test_rows(n, tile, block, cuda):
    fs = [tq.GaussianPeak(1, a=40.0, u=0.3),            # every chain by its polynomial
          tq.GaussianPeak(1, a=2e4, u=0.5),             # the chains near the peak
          tq.GaussianPeak(1, a=2e9, u=0.25),            # none
          tq.GaussianPeak(1, a=-0.5, u=0.2),
          tq.ExpSum(1, a=1500.0, b=-1450.0, c=1.3),     # those of exponents within 600
          tq.Oscillatory(1, a=30.0, b=0.2), tq.SumSin(1, a=25.0, c=0.7)]
    cases = [(f, r) for f in fs for r in RULES]
    dom = [[0.0, 1.0]]
    bg = B.BatchedGrid(dtype=torch.float64, autotune=False, tile_points=tile, block=block)
    plan = bg.plan([f for f, _ in cases], [r for _, r in cases], [n] * len(cases), [dom] * len(cases))
    got = bg.run(plan).cpu().numpy()
    for g, (f, r) in zip(got, cases):
        ev = lambda x, f=f: OI.evaluate(f.family, f.params_numpy(), x)  # noqa: E731
        want = OG.integrate(ev, RULES[r], 1, n, np.asarray(dom))
        size = OG.integrate(lambda x: np.abs(ev(x)), RULES[r], 1, n, np.asarray(dom))
        # steep rows: an exponent's rounding, up to 1500 2^-53, is the values'
        assert abs(g - want) <= 1e-12 * size + 1e-300, (f.family, f.params_numpy(), r, g, want)
