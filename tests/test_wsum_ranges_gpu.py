"""GPU: one row of nodes (a one-dimensional grid) summed in many ranges, as a
materialise budget cuts it.  Against exact sums (math.fsum)."""
import numpy as np
import pytest
import torch

from torchquad_gb300 import _lib as L
from torchquad_gb300.integration import _kernels as K

from .test_wsum_shapes_gpu import check

pytestmark = pytest.mark.gpu

T, S, B, G = L.TQ_RULE_TRAPEZOID, L.TQ_RULE_SIMPSON, L.TQ_RULE_BOOLE, L.TQ_RULE_GAUSS


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("S_", [1, 3])
@pytest.mark.parametrize("rule,n", [(T, 100_000), (S, 2047), (S, 65_537), (B, 40_001), (G, 300)])
def test_row_in_many_ranges(rule, n, S_, dtype, cuda):
    cuts = np.unique(np.linspace(0, n, 41).astype(int))
    check(rule, 1, n, S_, dtype, n, [*cuts], cuda)
    ragged = [0, 1, 2, 5, 33, n // 3, n // 3 + 1, n // 3 + 130, n - 130, n - 1, n]
    check(rule, 1, n, S_, dtype, n, sorted(set(ragged)), cuda)


@pytest.mark.parametrize("S_,launches", [(1, 1), (3, 2)])
def test_launch_count(S_, launches, cuda):
    """Several values per node are summed and their partials combined."""
    d = torch.tensor([[0.0, 1.0]], dtype=torch.float64, device=cuda)
    acc = torch.zeros(2 * S_, dtype=torch.float64, device=cuda)
    before = L.launches[0]
    K.weighted_sum_into(acc, S, 1, 101, d, None, 0, torch.ones(101, S_, dtype=torch.float64, device=cuda))
    assert L.launches[0] - before == launches
