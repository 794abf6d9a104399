"""Many-series recurrences of short histories: one launch (a block per 32 series,
a warp per chunk of rows) against the three launches of a fixed chunk length, at
rows around the chunk and rule limits, ragged starts, NaN gaps, series that are
seeded in their last rows and idle lanes.  The two compose their carries over different
chunks: a few roundings of the f32 state."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V

pytestmark = pytest.mark.gpu


def run(name, ins, params, policy=None):
    ind = V.CLASSES[name](0)
    if policy:
        ind.set_policy(*policy)
    return ind.many_series_one_param_time_major_dev(*ins, params=params).to_host()


@pytest.mark.parametrize("rows", [7, 33, 256, 257, 500, 639, 640, 641])
@pytest.mark.parametrize("cols", [1, 33, 100])
@pytest.mark.parametrize("name,period", [("ema", 20), ("dema", 9), ("tema", 9), ("rsi", 14), ("wilders", 5), ("atr", 14),
                                         ("ema", 120), ("rsi", 130)])
def test_one_launch_equals_three(name, period, cols, rows):
    if rows < 4 * period:
        period = max(2, rows // 4)
    rng = np.random.default_rng(rows * 131 + cols)
    close = (100 * np.exp(np.cumsum(rng.normal(0, 0.01, (rows, cols)), 0))).astype(np.float32)
    high, low = close * np.float32(1.01), close * np.float32(0.99)
    for s in range(1, cols):  # leads of every length (the first series is whole)
        lead = rows - 3 * period - 1 if s == 5 else (s * 7) % max(1, rows // 4)
        for a in (close, high, low):
            a[:lead, s] = np.nan
    if cols > 10 and rows > 60:
        close[rows // 2, 9] = np.nan
    ins = (high, low, close) if name == "atr" else (close,)
    got = run(name, ins, {"period": period})
    want = run(name, ins, {"period": period}, ("recur_chunk", "64"))
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= 1e-4 + 1e-5 * np.abs(want[ok]))
