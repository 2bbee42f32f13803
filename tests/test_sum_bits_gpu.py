"""GPU: how many bits the sums keep, by inputs whose exact sum is known and
of which shorter sums lose a visible part."""
from fractions import Fraction

import numpy as np
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


@pytest.mark.parametrize("S_", [1, 3])
@pytest.mark.parametrize("dim,n", [(5, 13), (3, 33)])
def test_scale_of_the_weights(dim, n, S_, cuda):
    """Ones: the result is the product of the dimensions' weight scales times
    a whole number, rounded once (the product itself to about 2^-104)."""
    rng = np.random.default_rng(dim)
    for _ in range(20):
        dom = [[0.0, float(w)] for w in rng.uniform(0.3, 3.0, dim)]
        want = Fraction(1)
        for _, b in dom:
            step = b / (n - 1)  # the second node less the first (0)
            want *= Fraction(step / 2.0) * (2 * (n - 1))
        d = torch.tensor(dom, dtype=torch.float64, device=cuda)
        ones = torch.ones(n**dim, S_, dtype=torch.float64, device=cuda)
        for got in K.weighted_result(T, dim, n, d, None, 0, ones, torch.float64).tolist():
            assert abs(Fraction(got) - want) <= want * Fraction(1.01 * 2.0**-53), (got, float(want))


@pytest.mark.parametrize("bits", [60, 90, 105])
@pytest.mark.parametrize("rule", [L.TQ_RULE_MC, T])
def test_values_that_cancel(rule, bits, cuda):
    """2^bits, a small value and -2^bits in different lanes: the sums over the
    lanes keep the small one (bits of a value down to 2^-106 of the largest)."""
    n = 2 if rule == L.TQ_RULE_MC else 5
    values = torch.zeros(n**2, 1, dtype=torch.float64, device=cuda)
    at = [0, 1, 2] if rule == L.TQ_RULE_MC else [6, 7, 8]  # interior nodes of equal weight
    values[at, 0] = torch.tensor([2.0**bits, 1.5, -(2.0**bits)], dtype=torch.float64, device=cuda)
    got = total(rule, 2, n, values, cuda, width=4.0)
    want = 1.5 * 16.0 / 4 if rule == L.TQ_RULE_MC else 1.5
    assert got == want


def test_fp32_samples_beyond_a_float(cuda):
    """2^32 samples of one fp32 value: a thread's sum needs 24 + 15 bits, and
    its error term more than a float where it is not brought back into line."""
    n, c = 2**32, float(np.float32(1.2345678))
    lib = L.lib()
    dom = torch.tensor([[0.0, 1.0]], dtype=torch.float32, device=cuda)
    par = torch.tensor([c, 0.0, 0.0, 0.0], dtype=torch.float64, device=cuda)
    out = torch.empty((), dtype=torch.float64, device=cuda)
    ws = L.workspace.get(lib.tq_mc_fused_workspace_size(1, n), "fused")
    L.check(lib.tq_mc_fused(L.TQ_F32, 1, n, dom.data_ptr(), L.TQ_FN_EXP_SUM, par.data_ptr(), 1, 0, 0, None,
                            out.data_ptr(), ws.data_ptr(), ws.numel(), L.stream_handle()), "tq_mc_fused")
    assert abs(out.item() - c) <= 2.0**-44 * c  # f2_add: 2^-47 an addition of 2^15, mostly cancelling


@pytest.mark.parametrize("S_", [1, 3])
@pytest.mark.parametrize("rule,dim,n", [(L.TQ_RULE_BOOLE, 3, 13), (L.TQ_RULE_BOOLE, 3, 33), (L.TQ_RULE_BOOLE, 1, 101),
                                        (L.TQ_RULE_SIMPSON, 1, 4001), (L.TQ_RULE_SIMPSON, 4, 9), (T, 2, 300)])
def test_values_near_the_top_of_the_range(rule, dim, n, S_, cuda):
    """The whole-number weights of a rule times fp64 values of 1e305 leave the
    range of doubles; the integral over the unit cube does not."""
    values = torch.full((n**dim, S_), 1e305, dtype=torch.float64, device=cuda)
    dom = torch.tensor([[0.0, 1.0]] * dim, dtype=torch.float64, device=cuda)
    got = K.weighted_result(rule, dim, n, dom, None, 0, values, torch.float64)
    assert torch.allclose(got, torch.full_like(got, 1e305), rtol=1e-13, atol=0.0), got
