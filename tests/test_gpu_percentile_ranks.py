"""The rank-bitmap percentile sweep (k_percentile.cu) against the oracle.

The outputs are selected inputs, so they are compared exactly.  Sizes sit at
the edges of the kernel's tiles (256 / 512 / 1,024 times), of its bitmap forms
(spans of 1,024 and 4,096 ranks) and of its staging (32 times); the data hold
NaN gaps longer than some windows, ties and infinities.
"""
import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def series(n, lead, seed=3, ticks=False):
    x = datagen.random_walk(n, seed=seed, nan_lead=lead)
    if ticks:
        x = np.round(x * 2.0) / 2.0  # many equal values
    x = x.astype(np.float32)
    if n > 900:
        x[700:705] = np.nan
        x[n // 2:n // 2 + 90] = np.nan  # empties the shorter windows
        x[n - 30] = np.inf
        x[n - 29] = -np.inf
    return x


CASES = [
    # (bars, lead, lengths, percentages, walk)
    (31, 0, (1, 31, 1), (0.0, 100.0, 50.0), "grow"),
    (257, 3, (2, 200, 9), (50.0, 50.0, 0.0), "slide"),
    (1000, 37, (5, 5, 0), (25.0, 25.0, 0.0), "grow"),
    (4099, 50, (15, 264, 1), (50.0, 50.0, 0.0), "grow"),
    (5000, 1, (63, 66, 1), (10.0, 90.0, 20.0), "slide"),
    (3001, 0, (511, 514, 1), (50.0, 75.0, 25.0), "grow"),
    (2999, 5, (768, 770, 1), (50.0, 50.0, 0.0), "grow"),
    (3001, 0, (500, 530, 2), (50.0, 50.0, 0.0), "slide"),
    (2600, 5, (700, 1020, 20), (50.0, 75.0, 25.0), "slide"),
    (6001, 9, (1020, 1030, 5), (1.0, 99.0, 49.0), "grow"),
    (2100, 7, (2, 9, 1), (25.0, 75.0, 25.0), "grow"),
    (1503, 2, (1, 800, 1), (50.0, 50.0, 0.0), "grow"),
    (1400, 2, (1200, 2, 3), (75.0, 75.0, 0.0), "slide"),
    (1400, 2, (1000, 2, 2), (75.0, 75.0, 0.0), "grow"),
    (4200, 0, (3840, 3841, 1), (50.0, 50.0, 0.0), "grow"),
    (4200, 0, (3842, 3842, 0), (50.0, 50.0, 0.0), None),
]


@pytest.mark.parametrize("ticks", [False, True])
@pytest.mark.parametrize("n,lead,length,pct,walk", CASES, ids=[f"{c[0]}-{c[2][0]}..{c[2][1]}" for c in CASES])
def test_rank_sweep_matches_oracle(n, lead, length, pct, walk, ticks):
    x = series(n, lead, ticks=ticks)
    xd = x.astype(np.float64)
    p = V.CudaPercentileNearestRank(0)
    sweep = {"length": length, "percentage": pct}
    got = p.batch_dev(x, sweep=sweep).to_host()
    # dense or short length axes grow the window, the others slide it; past the
    # bitmap one sorted array per thread
    assert p.last_kernel == ("percentile_ranks_" + walk if walk else "percentile_sorted_window")
    grid = p.expand_grid(sweep)
    assert got.shape == (len(grid), n)
    for row, g in zip(got, grid):
        # the library holds the fraction percentage / 100 as f32, so the rank
        # round(p * count) of a half-way product follows that value
        pct = float(np.float32(g["percentage"] * 0.01)) * 100.0
        exp = O.percentile_nearest_rank(xd, g["length"], pct)
        assert np.array_equal(row.astype(np.float64), exp, equal_nan=True), g
