"""Percentile sweeps with more percentages than a grid has rows (65,535)."""
import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def test_more_percentages_than_grid_rows():
    x = datagen.random_walk(64, seed=6, nan_lead=3).astype(np.float32)
    xd = x.astype(np.float64)
    p = V.CudaPercentileNearestRank(0)
    sweep = {"length": (4, 5, 1), "percentage": (0.0, 100.0, 0.0015)}
    got = p.batch_dev(x, sweep=sweep).to_host()
    assert p.last_kernel == "percentile_ranks_grow"
    grid = p.expand_grid(sweep)
    assert got.shape == (len(grid), 64) and len(grid) > 2 * 65_535
    for i in [*range(0, len(grid), 331), *range(65_530, 65_541), *range(len(grid) - 5, len(grid))]:
        g = grid[i]
        pct = float(np.float32(g["percentage"] * 0.01)) * 100.0  # (the fraction is held as f32)
        exp = O.percentile_nearest_rank(xd, g["length"], pct)
        assert np.array_equal(got[i].astype(np.float64), exp, equal_nan=True), g
