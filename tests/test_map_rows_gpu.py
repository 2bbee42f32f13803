"""One-CTA-per-row map update at the edges of its helpers: runs of empty
intervals around the ten places that the fill reaches (both ends, ties, empty
intervals that carry weights), rows decided late by the zero-row test, long
spans and runs of equal delta multiples."""
import numpy as np
import pytest
import torch

from tests.test_vegas_gpu import _check_large_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("B", [33, 257, 1024])
@pytest.mark.parametrize("case", ["runs", "raw", "late", "peaked"])
def test_map_row_helpers_match_oracle(case, B, dtype, cuda):
    from oracle import vegas as OV

    rng = np.random.default_rng({"runs": 1, "raw": 2, "late": 3, "peaked": 4}[case] + B)
    d = 16  # every half-warp of a CTA tests a row
    counts = rng.integers(1, 30, size=(d, B)).astype(np.int64)
    weights = rng.uniform(0.05, 4.0, size=(d, B)) * counts
    if case in ("runs", "raw"):
        z = np.zeros((d, B), dtype=bool)
        for k in range(d):  # runs of 9 to 24, one a row at each end and inside
            n = 9 + k
            z[k, 2 : 2 + n] = True
            if k % 3 == 1:
                z[k, :11] = True
            if k % 3 == 2:
                z[k, -12:] = True
        counts[z] = 0
        if case == "runs":
            weights[z] = 0.0
    elif case == "late":  # the only intervals with weight stand last
        z = np.zeros((d, B), dtype=bool)
        z[:, : B - 2] = True
        counts[z] = 0
        weights[z] = 0.0
    else:
        x = (np.arange(B) + 0.5) / B
        for k in range(d):
            weights[k] = (np.exp(-(((x - rng.uniform(0.2, 0.8)) / 0.02) ** 2)) + 1e-7) * counts[k]
    # the bounds of the peaked and empty cases of the tiled update
    _check_large_map(OV, dtype, cuda, weights, counts, tol32=5e-5)
