"""GPU: the weighted sums of materialised values (tq_weighted_sum) over the
shapes at which their walk changes: joined and split rows, ranges that start
and end inside a row, one and many values per node, both types, Monte Carlo.
Against exact sums (math.fsum)."""
import math

import numpy as np
import pytest
import torch

from oracle import grid as OG
from torchquad_gb300 import _lib as L
from torchquad_gb300.integration import _kernels as K

pytestmark = pytest.mark.gpu

T, S, B, G, MC = L.TQ_RULE_TRAPEZOID, L.TQ_RULE_SIMPSON, L.TQ_RULE_BOOLE, L.TQ_RULE_GAUSS, L.TQ_RULE_MC
DEN = {T: 2.0, S: 3.0, B: 22.5}


def unit_weights(rule, n):
    i = np.arange(n)
    if rule == T:
        c = np.full(n, 2.0)
    elif rule == S:
        c = np.where(i % 2 == 1, 4.0, 2.0)
    else:
        c = np.where(i % 2 == 1, 32.0, np.where(i % 4 == 2, 12.0, 14.0))
    c[[0, -1]] /= 2.0
    return c


def weights(rule, dim, n, dom, glw):
    if rule == MC:
        return None
    w = np.ones(1)
    for a, b in dom:
        if rule == G:
            one = 0.5 * (b - a) * glw
        else:  # the rules' step is the distance of the first two nodes
            x = OG.linspace(a, b, n, np.float64)
            one = (x[1] - x[0]) / DEN[rule] * unit_weights(rule, n)
        w = np.multiply.outer(w, one).ravel()
    return w


def run(rule, dim, n, dom, glw, values, bounds, cuda):
    """The running sums of values [count, S] fed in the ranges of bounds."""
    d = torch.tensor(dom, dtype=torch.float64, device=cuda)
    glt = None if rule != G else torch.tensor(glw, device=cuda)
    v = torch.from_numpy(values).to(cuda)
    acc = torch.zeros(2 * values.shape[1], dtype=torch.float64, device=cuda)
    for s, e in zip(bounds[:-1], bounds[1:]):
        if e > s:
            K.weighted_sum_into(acc, rule, dim, n, d, glt, int(s), v[s:e].contiguous())
    return acc.cpu().numpy().reshape(-1, 2).sum(axis=1)


def check(rule, dim, n, S_, dtype, count, bounds, cuda):
    rng = np.random.default_rng(n * 100 + S_ + dim)
    dom = [[-0.6 + 0.1 * k, 0.7 + 0.2 * k] for k in range(dim)]
    glw = np.polynomial.legendre.leggauss(n)[1] if rule == G else None
    values = (rng.standard_normal((count, S_)) * np.exp(rng.uniform(-3, 3, (count, 1)))).astype(dtype)
    got = run(rule, dim, n, dom, glw, values, bounds, cuda)
    w = weights(rule, dim, n, dom, glw)
    # fp64 values: one rounding per term and per addition of the few values a
    # lane meets; fp32 values: Kahan's sums leave two roundings of 2^-24 of
    # each unit of at most 64 values a lane, Gauss weights one of theirs
    tol = 2.0**-48 if dtype == np.float64 else (2.0**-22 if rule == G else 2.0**-23)
    for s in range(S_):
        terms = values[:, s].astype(np.float64) * (1.0 if w is None else w)
        want, mag = math.fsum(terms), np.abs(terms).sum()
        assert abs(got[s] - want) <= tol * mag, (rule, dim, n, S_, s, got[s], want, mag)


def ranges(count):
    cut = [0, count // 7 + 1, count // 2 + 3, count - 5, count]
    return [[0, count], sorted(min(max(c, 0), count) for c in cut)]


SHAPES = [(T, 1, 2), (S, 1, 33), (T, 1, 1001), (B, 1, 2053), (S, 1, 20_001), (G, 1, 130), (S, 2, 31), (S, 2, 33),
          (T, 2, 257), (G, 2, 31), (G, 2, 64), (B, 3, 5), (T, 3, 13), (S, 3, 45), (G, 3, 17), (S, 5, 9), (T, 10, 3),
          (T, 16, 2)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rule,dim,n", SHAPES)
def test_scalar_values(rule, dim, n, dtype, cuda):
    for bounds in ranges(n ** dim):
        check(rule, dim, n, 1, dtype, n ** dim, bounds, cuda)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("S_", [2, 3, 16, 31, 32, 33, 70])
@pytest.mark.parametrize("rule,dim,n", [(S, 1, 1001), (T, 2, 31), (B, 3, 13), (G, 2, 20), (G, 1, 97)])
def test_vector_values(rule, dim, n, S_, dtype, cuda):
    for bounds in ranges(n ** dim):
        check(rule, dim, n, S_, dtype, n ** dim, bounds, cuda)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("count,S_", [(1, 1), (127, 1), (40_003, 1), (1, 5), (999, 3), (5000, 40)])
def test_monte_carlo_values(count, S_, dtype, cuda):
    check(MC, 2, 1, S_, dtype, count, [0, count], cuda)


@pytest.mark.parametrize("value", [3e35, 1e-30])
@pytest.mark.parametrize("width", [1e-300, 1e-8, 1e6])
def test_fp32_values_of_extreme_size(value, width, cuda):
    """Unit sums of 2^80 and more leave the double-float sum; weights far
    from one do not cost precision."""
    n = 301
    values = np.full((n * n, 1), value, dtype=np.float32)
    got = run(S, 2, n, [[0.0, 1.0], [0.0, width]], None, values, [0, n * n], cuda)[0]
    want = float(values[0, 0]) * width
    assert abs(got - want) <= 2.0**-22 * want, (got, want)


def test_non_finite_values(cuda):
    for dtype in (np.float32, np.float64):
        for S_ in (1, 3):
            values = np.ones((101 * 101, S_), dtype=dtype)
            values[5000, S_ - 1] = np.inf
            values[7000, 0] = np.nan if S_ == 3 else np.inf
            got = run(S, 2, 101, [[0.0, 1.0]] * 2, None, values, [0, 101 * 101], cuda)
            assert not np.isfinite(got[0]) and not np.isfinite(got[S_ - 1])
            if S_ == 3:
                assert abs(got[1] - 1.0) < 1e-6
