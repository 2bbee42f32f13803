"""Map histogram of the fused sampler without warp histograms: every draw of
the counter-based stream (each dimension's alignment to the Philox blocks)
against the same draws by torch operations, with the counts in shared memory,
and added directly where a CTA may take 65,536 points or they do not fit."""
import pytest
import torch

import torchquad_gb300 as tq
from torchquad_gb300.integration.rng import RNG
from torchquad_gb300.integration._vegas_state import VegasDevice

pytestmark = pytest.mark.gpu


def warmed(dim, bins, n, dtype, cuda, seed=5):
    dev = VegasDevice(dim, dtype, bins, 1, cuda)
    dev.control[3] = seed
    dev.warmup_fused(tq.ExpSum(dim).family, tq.ExpSum(dim).device_params(cuda), n)
    return dev


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 16])
def test_counts_are_those_of_the_draws(dim, dtype, cuda):
    for bins, n in ((1001, 1), (1024, 33), (999, 4_099), (9_000, 3_000)):
        dev = warmed(dim, bins, n, dtype, cuda)
        y = RNG(seed=5).uniform([n, dim], dtype) * 0.999999
        ids = torch.floor(y * bins).long()
        want = torch.stack([torch.bincount(ids[:, k], minlength=bins) for k in range(dim)])
        assert torch.equal(dev.counts, want)
        # each dimension's weights hold the same fp64 sum, in another order
        # (at most n additions, each 2^-53 of the sum)
        tot = dev.weights.sum(1)
        assert float((tot - tot[0]).abs().max()) <= 2.0 * n * 2.0**-53 * float(tot[0])
        assert torch.equal(dev.weights > 0, want > 0)


@pytest.mark.parametrize("n", [39_800_000, 39_900_000])  # 2045.6 and 2050.8 tiles of 32 a CTA of 608
def test_counts_at_the_width_of_a_count(n, cuda):
    dev = warmed(1, 1001, n, torch.float32, cuda)
    assert int(dev.counts.sum()) == n
    # equal intervals: a count is binomial, nine standard deviations
    mean = n / 1001
    assert float((dev.counts.double() - mean).abs().max()) <= 9.0 * mean**0.5
