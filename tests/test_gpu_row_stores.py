"""Sweeps whose rows do not start at 32-byte sectors (lengths not a multiple of
eight): large outputs are stored cut at the sectors.  The rows must be those of
the same sweep on a padded series, whose rows do start at sectors, bit for bit
over the common bars: the chunks are the same, only the stores differ."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu

N = 72_001  # 240 rows: above the size from which stores are cut


def run(name, cols, sweep, chunk):
    ind = V.CLASSES[name](0)
    if chunk:
        ind.set_policy("recur_chunk", chunk)
    out = ind.batch_dev(*cols, sweep=sweep)
    outs = out if isinstance(out, (tuple, list)) else (out,)
    return [o.to_host() for o in outs]


def inputs(n, name):
    d = datagen.ohlcv(n, seed=71, nan_lead=33)
    if name in ("atr",):
        return tuple(np.asarray(d[k], np.float32) for k in ("high", "low", "close"))
    return (np.asarray(d["close"], np.float32),)


@pytest.mark.parametrize("chunk", ["96", "704", "1376"])
@pytest.mark.parametrize("extra", [0, 1, 2, 4, 5, 6])
@pytest.mark.parametrize("name", ["ema", "rsi", "atr"])
def test_recurrence_rows(name, extra, chunk):
    n = N + extra
    pad = (n + 7) // 8 * 8
    sweep = {"period": (2, 251, 1)}
    cols = inputs(pad, name)
    want = run(name, cols, sweep, chunk)
    got = run(name, tuple(np.ascontiguousarray(c[:n]) for c in cols), sweep, chunk)
    for g, w in zip(got, want):
        assert g.shape[1] == n
        assert np.array_equal(g, w[:, :n], equal_nan=True)


@pytest.mark.parametrize("gap", [None, 40_000])
@pytest.mark.parametrize("extra", [0, 1, 2, 5])
@pytest.mark.parametrize("name,n0,hi", [("bollinger_bands", 92_001, 254), ("sma", 200_001, 704), ("stddev", 92_001, 254)])
def test_prefix_window_rows(name, n0, hi, extra, gap):
    # a shifted tile may take its reference value one to seven bars away: the
    # rows agree to a few roundings of one f32 result
    n = n0 + extra
    pad = (n + 7) // 8 * 8
    sweep = {"period": (5, hi, 1), "devup": (2.0, 2.0, 0.0), "devdn": (2.0, 2.0, 0.0), "nbdev": (1.0, 1.0, 0.0)}
    (x,) = inputs(pad, name)
    if gap:
        x = x.copy()
        x[gap] = np.nan
    want = run(name, (x,), sweep, None)
    got = run(name, (np.ascontiguousarray(x[:n]),), sweep, None)
    for g, w in zip(got, want):
        w = w[:, :n]
        assert np.array_equal(np.isnan(g), np.isnan(w))
        d = np.abs(g - w)
        assert np.nanmax(d / np.maximum(np.abs(w), 1.0)) <= 1e-5
