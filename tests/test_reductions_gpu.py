"""GPU: the fixed-point CTA sums against exact sums (math.fsum)."""
import math
import warnings

import numpy as np
import pytest
import torch

import torchquad_gb300 as tq

pytestmark = pytest.mark.gpu


def _mean(values, cuda):
    dom = torch.tensor([[0.0, 1.0]], dtype=torch.float64, device=cuda)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return tq.MonteCarlo().calculate_result(torch.tensor(values, device=cuda), dom).item()


@pytest.mark.parametrize("n", [1, 31, 257, 5000, 300_001])
@pytest.mark.parametrize("span", [0, 20, 200, 900])
def test_sum_of_wide_range_values(n, span, cuda):
    """Values of either sign over 2^-span .. 2^span that largely cancel: the
    mean within two roundings of the exact one, plus 2^-90 of the largest
    value (the threads' own compensated sums and the 96-bit window)."""
    rng = np.random.default_rng(n + span)
    v = rng.standard_normal(n) * 2.0 ** rng.uniform(-span, span, n)
    v[n // 2:2 * (n // 2)] = -v[:n // 2] * (1.0 + 2.0**-40)
    got = _mean(v, cuda)
    exact = math.fsum(v) / n
    assert abs(got - exact) <= 2 * 2.0**-53 * abs(exact) + 2.0**-90 * np.abs(v).max(), (got, exact)


@pytest.mark.parametrize("bad", [math.inf, -math.inf, math.nan])
def test_non_finite_values_do_not_give_a_number(bad, cuda):
    v = np.ones(1000)
    v[777] = bad
    assert not math.isfinite(_mean(v, cuda))


def test_zeros_and_subnormals(cuda):
    assert _mean(np.zeros(999), cuda) == 0.0
    tiny = 2.0**-1074
    assert _mean(np.full(1024, 3 * tiny), cuda) == 3 * tiny
