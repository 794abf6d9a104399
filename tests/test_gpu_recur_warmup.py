"""Warm-up of the batch recurrences: seeds before, inside and across chunks and
32-step tiles, a series that ends during the warm-up of its longest combos,
NaN gaps and huge values inside the warm-up (which take the per-step path),
against the oracle with the crate's tolerances."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import TOL, assert_close
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def series(n, lead, bad):
    c = datagen.random_walk(n, seed=77, nan_lead=lead)
    if bad == "gap":
        c[lead + 40:lead + 43] = np.nan
    if bad == "huge":
        c[lead + 33] = 1e30
    hi, lo = datagen.high_low(c, seed=78)
    return [a.astype(np.float32) for a in (hi, lo, c)]


def expect(name, h, l, c, periods):
    h, l, c = (a.astype(np.float64) for a in (h, l, c))
    if name == "atr":
        return np.stack([O.atr(h, l, c, p) for p in periods])
    if name == "rsi":
        return O.rsi_batch(c, periods)
    if name == "wilders":
        return O.wilders_batch(c, periods)
    return np.stack([{"ema": O.ema, "dema": O.dema, "tema": O.tema}[name](c, p) for p in periods])


SWEEPS = [  # (bars, lead, lo, hi, step): 1 and 33 lanes, seeds at tile and chunk edges
    (257, 0, 1, 33, 1), (1000, 5, 31, 33, 1), (1500, 31, 2, 322, 10), (5000, 200, 250, 262, 1),
    (4096, 1, 2, 1000, 29), (1025, 33, 500, 500, 0), (700, 100, 2, 300, 7),
]


@pytest.mark.parametrize("n,lead,lo,hi,step", SWEEPS)
@pytest.mark.parametrize("name", ["ema", "dema", "tema", "rsi", "wilders", "atr"])
def test_warm_up_matches_oracle(name, n, lead, lo, hi, step):
    if name in ("dema", "tema"):  # the crate asks for 2 (p - 1) valid bars; TEMA starts at 3 (p - 1)
        hi = min(hi, (n - lead) // 3)
        lo = min(lo, hi)
    h, l, c = series(n, lead, None)
    ind = V.CLASSES[name](0)
    sweep = {"period": (lo, hi, step)}
    ps = [g["period"] for g in ind.expand_grid(sweep)]
    got = ind.batch_dev(*([h, l, c] if name == "atr" else [c]), sweep=sweep).to_host()
    assert_close(got, expect(name, h, l, c, ps), TOL[name], f"{name} ({ind.last_kernel})")


@pytest.mark.parametrize("chunk", ["auto", "64", "sequential"])
@pytest.mark.parametrize("name", ["ema", "rsi", "tema"])
def test_gap_in_warm_up(name, chunk):
    h, l, c = series(1500, 20, "gap")
    ind = V.CLASSES[name](0)
    ind.set_policy("recur_chunk", chunk)
    sweep = {"period": (3, 200, 9)}
    ps = [g["period"] for g in ind.expand_grid(sweep)]
    got = ind.batch_dev(c, sweep=sweep).to_host()
    assert_close(got, expect(name, h, l, c, ps), TOL[name], f"{name} gap")


@pytest.mark.parametrize("name", ["ema", "rsi", "wilders"])
def test_huge_value_in_warm_up(name):
    # against the sequential kernel: the sums of the crate's f64 hold what f32 cannot
    h, l, c = series(1500, 20, "huge")
    out = {}
    for mode in ("auto", "sequential"):
        ind = V.CLASSES[name](0)
        ind.set_policy("recur_chunk", mode)
        out[mode] = ind.batch_dev(c, sweep={"period": (3, 200, 9)}).to_host()
    assert np.array_equal(np.isnan(out["auto"]), np.isnan(out["sequential"]))
    m = np.isfinite(out["sequential"]) & (np.abs(out["sequential"]) > 1e20)
    assert np.allclose(out["auto"][m], out["sequential"][m], rtol=1e-5)
