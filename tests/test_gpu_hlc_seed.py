"""Seeding of the chunked ADX and SuperTrend sweeps: the bars' shared terms and
the branch-free seeding steps against the sequential kernel, bit for bit, where
they can go wrong: first valid bars around a 32-step tile's edges, the smallest
periods, NaN bars inside the seeding, and group sizes that leave lanes idle."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def run(ind_name, cols, sweep, policy=None):
    ind = V.CLASSES[ind_name](0)
    if policy:
        ind.set_policy(*policy)
    out = ind.batch_dev(*cols, sweep=sweep)
    outs = out if isinstance(out, (tuple, list)) else (out,)
    return [o.to_host() for o in outs], ind.last_kernel


@pytest.mark.parametrize("gap", [None, 3, 40])
@pytest.mark.parametrize("lead", [0, 31, 32, 33])
@pytest.mark.parametrize("name,sweep", [
    ("adx", {"period": (2, 5, 1)}), ("adx", {"period": (2, 34, 1)}),
    ("supertrend", {"period": (1, 5, 1), "factor": (1.0, 3.0, 0.25)}),
    ("supertrend", {"period": (16, 48, 1), "factor": (2.0, 2.0, 0.0)})])
def test_seeding_is_the_sequential_one(name, sweep, lead, gap):
    d = datagen.ohlcv(9_001, seed=91 + lead, nan_lead=lead)
    h, l, c = (np.asarray(d[k], np.float32).copy() for k in ("high", "low", "close"))
    if gap is not None:
        c[lead + gap] = np.nan
        h[lead + gap + 2] = np.nan
    got, kern = run(name, (h, l, c), sweep)
    assert kern == name + "_chunked", kern
    seq, _ = run(name, (h, l, c), sweep, ("recur_chunk", "sequential"))
    for g, s in zip(got, seq):
        assert np.array_equal(g, s, equal_nan=True)


@pytest.mark.parametrize("sweep", [{"period": (1, 4, 1)}, {"period": (1, 301, 100)}])
def test_period_one_has_no_nan(sweep):
    # period 1 keeps nothing of the bar before: +DM + -DM is 0 on inside bars,
    # where DX is 0
    d = datagen.ohlcv(9_001, seed=95, nan_lead=20)
    cols = tuple(np.asarray(d[k], np.float32) for k in ("high", "low", "close"))
    (got,), _ = run("adx", cols, sweep)
    (seq,), _ = run("adx", cols, sweep, ("recur_chunk", "sequential"))
    assert np.array_equal(np.isnan(got), np.isnan(seq))
    # period 1 is DX itself: full divide or hardware reciprocal, two ulps of 100
    assert np.nanmax(np.abs(got[0] - seq[0])) <= 2e-5
