"""Many-series time-major kernels against the oracle at the sizes where their
tiling can go wrong: one series, series counts around a warp and a block,
NaN leads past one round of the first-valid scan, row counts around the time
chunks, window lengths around the chunk and 1, NaN (and infinite) bars inside
a series.  Tolerances are those of the crate's many-series tests."""
import numpy as np
import pytest

from test_gpu_parity import PARAMS, TOL_TM, assert_close, oracle_series
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu

SHAPES = [(1, 700), (31, 64), (33, 1029), (129, 333)]
# windows of the crate's running sums and selections, whose NaN rules are
# checked with gaps as well
GAPS = {"sma", "stddev", "zscore", "bollinger_bands", "wma", "trima", "donchian", "willr"}


def matrix(cols, rows, seed, gaps):
    c, h, l = (np.full((rows, cols), np.nan, dtype=np.float32) for _ in range(3))
    for j in range(cols):
        x = datagen.random_walk(rows, seed=seed + j)
        hi, lo = datagen.high_low(x, seed=seed + 500 + j)
        lead = min((37 * j) % 601, rows // 2 - 30)
        if gaps and j % 3 == 1:
            x[rows - 40], hi[rows - 40], lo[rows - 40] = np.nan, np.nan, np.nan
        if gaps and j % 5 == 2:
            hi[rows - 25] = np.inf
        c[lead:, j], h[lead:, j], l[lead:, j] = x[lead:], hi[lead:], lo[lead:]
    return c, h, l


def run(name, c, h, l, prm):
    ins = {"x": [c], "hl": [h, l], "hlc": [h, l, c]}[V.N.INDICATORS[name][0]]
    got = V.CLASSES[name](0).many_series_one_param_time_major_dev(*ins, params=prm)
    return [g.to_host() for g in (got if isinstance(got, tuple) else (got,))]


def check(name, c, h, l, prm):
    got = run(name, c, h, l, prm)
    exp = [np.full(c.shape, np.nan) for _ in got]
    for j in range(c.shape[1]):
        for k, row in enumerate(oracle_series(name, *(a[:, j].astype(np.float64) for a in (c, h, l)), prm)):
            exp[k][:, j] = row
    for k in range(len(got)):
        inf = np.isinf(exp[k])  # (a difference of infinities is NaN)
        assert np.array_equal(got[k][inf], exp[k][inf]), f"{name} {prm} tm[{k}]: infinities"
        exp[k][inf] = got[k][inf] = 0.0
        assert_close(got[k], exp[k], TOL_TM[name], f"{name} {prm} tm[{k}]")


@pytest.mark.parametrize("cols,rows", SHAPES)
@pytest.mark.parametrize("name", ["sma", "stddev", "zscore", "bollinger_bands", "wma", "trima", "alma", "ema", "dema",
                                  "tema", "rsi", "wilders", "atr", "donchian", "willr"])
def test_shapes(name, cols, rows):
    c, h, l = matrix(cols, rows, seed=40, gaps=name in GAPS)
    if name == "zscore":  # the oracle's running sums, not the window, decide an exactly flat window
        c = np.where(np.isinf(c), np.nan, c)
    prm = dict(PARAMS[name])
    check(name, c, h, l, prm)


@pytest.mark.parametrize("period", [1, 2, 31, 32, 33, 63, 64, 65, 200])
@pytest.mark.parametrize("name", ["sma", "bollinger_bands", "rsi", "ema", "wilders", "atr", "donchian", "willr"])
def test_periods(name, period):
    # (the crate's SMA copies x at period 1, the many-series one keeps its
    # running-sum NaN rule there)
    c, h, l = matrix(35, 700, seed=90, gaps=name in GAPS and (name, period) != ("sma", 1))
    check(name, c, h, l, dict(PARAMS[name], period=period))


@pytest.mark.parametrize("name", ["sma", "stddev", "bollinger_bands"])
def test_overflowing_values_poison_alike(name):
    """The running sums restart every 512 rows; shorter chunks (few series)
    poison the same outputs after an infinite or overflowing value as 512-row
    chunks (many series) do."""
    c, _, _ = matrix(32, 1029, seed=7, gaps=False)
    for j, v in enumerate([np.inf, -np.inf, 3e38, 2e19, 1e30]):
        c[400 + 70 * j, 3 * j] = v
        c[511 + j, 3 * j + 1] = v
    prm = dict(PARAMS[name], period=20)
    few = run(name, c, c, c, prm)
    many = run(name, np.tile(c, (1, 1600)), None, None, prm)
    for a, b in zip(few, many):
        b = b[:, :32]
        assert np.array_equal(np.isnan(a), np.isnan(b))
        ok = np.isfinite(b) & (np.abs(b) < 1e6)
        assert np.allclose(a[ok], b[ok], rtol=1e-5, atol=1e-4 * (name != "sma"))
