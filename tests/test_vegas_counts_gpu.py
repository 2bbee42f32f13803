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


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("strat", [1, 2, 3, 7, 10, 41, 255, 4_093, 65_537, 1_048_575, 3_000_017])
def test_stratified_draws_are_those_of_the_division(strat, dtype, cuda):
    """The quotient by n_strat to its last bits: 2^24 intervals, so that a
    count gives 24 bits of the y of its draw."""
    from torchquad_gb300 import _lib as L

    bins, f = 1 << 24, tq.ExpSum(1)
    dev = VegasDevice(1, dtype, bins, strat, cuda)
    dev.set_control(L.TQ_VC_NEVALS | L.TQ_VC_SEED | L.TQ_VC_STREAM, nevals=max(100_000, 2 * strat), seed=9, sid=0)
    dev.get_nh()
    dev.iterate_fused(f.family, f.device_params(cuda), True)
    pos = torch.repeat_interleave(torch.arange(strat, device=cuda), dev.neval)
    u = RNG(seed=9).uniform([pos.numel(), 1], dtype)[:, 0]
    y = (pos.to(dtype) + u) / torch.full((1,), strat, dtype=dtype, device=cuda)
    y = torch.where(y >= 1.0, torch.full_like(y, 0.999999), y)
    want = torch.bincount(torch.floor(y * bins).long(), minlength=bins)
    assert torch.equal(dev.counts[0], want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("bins", [2, 3, 5, 9, 17, 33])
def test_groups_of_every_size_in_warp_histograms(bins, dtype, cuda):
    """Few intervals: groups of up to 32 lanes share one, on both sides of the
    steps that are taken without a loop."""
    for n in (1, 31, 32, 33, 1_000, 70_001):
        dev = warmed(3, bins, n, dtype, cuda)
        y = RNG(seed=5).uniform([n, 3], dtype) * 0.999999
        ids = torch.floor(y * bins).long()
        x = y.double()
        f2 = torch.exp(x.sum(1)) ** 2
        for k in range(3):
            assert torch.equal(dev.counts[k], torch.bincount(ids[:, k], minlength=bins))
            want = torch.zeros(bins, dtype=torch.float64, device=cuda).index_add_(0, ids[:, k], f2)
            # fp32: squares rounded three times and more, warp sums of at most
            # n values in fp32 trees and one add a tile (70001/32/4864 tiles a warp)
            tol = 1e-5 if dtype == torch.float32 else 1e-12
            assert torch.allclose(dev.weights[k], want, rtol=tol, atol=0)
