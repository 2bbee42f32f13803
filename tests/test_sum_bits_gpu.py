"""GPU: how many bits the sums keep, by inputs whose exact sum is known and
of which shorter sums lose a visible part."""
import pytest
import torch

from torchquad_gb300 import _lib as L
from torchquad_gb300.integration import _kernels as K

pytestmark = pytest.mark.gpu

T = L.TQ_RULE_TRAPEZOID


def total(rule, dim, n, values, cuda, width=1.0):
    dom = torch.tensor([[0.0, width]] * dim, dtype=torch.float64, device=cuda)
    return K.weighted_result(rule, dim, n, dom, None, 0, values, torch.float64).item()


def test_long_fp64_row(cuda):
    """2^30 intervals of a constant 1 + 2^-47: a lane's sums of up to 32 such
    values are exact, and what follows is compensated, so the result has no
    more than its last roundings (2^-51 for a few of them); a lane that adds
    its thousands of values without compensation drops the tail of each value
    beyond 2^12."""
    n = 2**30 + 1
    v = 1.0 + 2.0**-47
    got = total(T, 1, n, torch.full((n, 1), v, dtype=torch.float64, device=cuda), cuda)
    assert abs(got - v) <= 2.0**-51, got - v
