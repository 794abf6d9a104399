"""Operands of the tensor-core weighted windows: NaN bars at the edges of the
32-bar words and 256-bar tiles they are recorded in, in both of the crate's
NaN rules, sweeps of one row up to more rows than a tile, rows shorter than an
octet, and windows longer than one K slice, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu

NANS = [(), (255,), (256,), (31, 32), (511, 512, 513), (1999,), (40, 700, 1500)]


@pytest.mark.parametrize("nans", NANS, ids=[str(n) for n in NANS])
@pytest.mark.parametrize("name,rng", [("wma", (2, 130, 1)), ("swma", (4, 40, 3)), ("alma", (3, 300, 2)),
                                      ("cwma", (2, 9, 1)), ("sinwma", (17, 17, 0)), ("alma", (5, 260, 255))])
def test_nan_bars(name, rng, nans):
    x = datagen.random_walk(2000, seed=21, nan_lead=7).astype(np.float32)
    x[list(nans)] = np.nan
    xd = x.astype(np.float64)
    sweep = {"period": rng}
    if name == "alma":
        sweep.update(offset=(0.85, 0.85, 0.0), sigma=(6.0, 6.0, 0.0))
    ind = V.CLASSES[name](0)
    got = ind.batch_dev(x, sweep=sweep).to_host().astype(np.float64)
    assert ind.last_kernel == "wwma_tc_fp16x3"
    fn = {"alma": lambda p: O.alma(xd, p, 0.85, 6.0), "wma": lambda p: O.wma(xd, p), "swma": lambda p: O.swma(xd, p),
          "cwma": lambda p: O.cwma(xd, p), "sinwma": lambda p: O.sinwma(xd, p)}[name]
    for row, g in zip(got, ind.expand_grid(sweep)):
        exp = fn(g["period"])
        assert np.array_equal(np.isnan(row), np.isnan(exp)), (g["period"], nans)
        m = ~np.isnan(exp)
        assert np.all(np.abs(row[m] - exp[m]) <= 1e-5 * np.abs(exp[m])), g["period"]
