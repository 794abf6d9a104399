"""Weighted windows of thousands of bars: around the lengths up to which a
preparation block stages four weight rows (7,232), and up to the longest strip
(28,656), against the oracle; longer ones are refused and leave no error behind.

Tolerance: with S the series' span, the values centred on a tile's reference lie
within S.  Splitting both operands into f16 pairs and leaving out the product of
the low parts costs at most 2^-22 each, the f32 accumulation at most 2^-23 of a
partial sum for each of the 3 K / 16 instructions a window of K bars takes
(2^-24 where they round, not truncate), the last steps a few 2^-24 of the
value."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["alma", "wma", "srwma"])
@pytest.mark.parametrize("rng", [(3384, 3400, 8), (7232, 7312, 16), (5, 12005, 3000), (28000, 28656, 656)],
                         ids=lambda r: f"{r[0]}-{r[1]}")
def test_long_windows(name, rng):
    x = datagen.random_walk(29_500, seed=4, nan_lead=3).astype(np.float32)
    xd = x.astype(np.float64)
    sweep = {"period": rng}
    if name == "alma":
        sweep.update(offset=(0.85, 0.85, 0.0), sigma=(6.0, 6.0, 0.0))
    ind = V.CLASSES[name](0)
    got = ind.batch_dev(x, sweep=sweep).to_host().astype(np.float64)
    assert ind.last_kernel == "wwma_tc_fp16x3"
    span = np.nanmax(xd) - np.nanmin(xd)
    fn = {"alma": lambda p: O.alma(xd, p, 0.85, 6.0), "wma": lambda p: O.wma(xd, p), "srwma": lambda p: O.srwma(xd, p)}[name]
    for row, g in zip(got, ind.expand_grid(sweep)):
        exp = fn(g["period"])
        assert np.array_equal(np.isnan(row), np.isnan(exp)), g
        m = ~np.isnan(exp)
        tol = span * (3 * g["period"] / 16 * 2**-23 + 3 * 2**-22) + 2**-22 * np.abs(exp[m])
        assert np.all(np.abs(row[m] - exp[m]) <= tol), g


def test_past_the_strip_is_refused():
    x = datagen.random_walk(29_500, seed=4).astype(np.float32)
    wma = V.CudaWma(0)
    for p in (28_657, 28_800):
        with pytest.raises(V.VtaError):
            wma.batch_dev(x, sweep={"period": (p, p, 0)})
        wma.batch_dev(x, sweep={"period": (9, 9, 0)}).free()


@pytest.mark.parametrize("p", [1504, 1512, 1536, 1537])
def test_shared_memory_of_a_plain_launch(p):
    """Around 48 KB of a preparation block's shared memory, in a process of its
    own: a longer window before it raises the kernel's limit for good."""
    code = ("import sys; sys.path.insert(0, sys.argv[1]); import numpy as np; from vectorta_gb300 import cuda as V\n"
            "x = np.linspace(1, 2, 4000, dtype=np.float32); p = int(sys.argv[2])\n"
            "V.CudaWma(0).batch_dev(x, sweep={'period': (p, p, 0)}).free()")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code, root, str(p)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-500:]
