"""Seeds of Wilders' average and ATR: the f32 nearest the exact mean, also for
values so small that the rounding error of an f32 product underflows.  (The
quotient of the exact sums is formed in f64; its rounding to f32 differs from
the exact mean's for one in 2^28.)"""
import math

import numpy as np
import pytest

from vectorta_gb300 import cuda as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0, -120], ids=["1", "2^-120"])
@pytest.mark.parametrize("name,n", [("wilders", 2048), ("wilders", 6000), ("atr", 2000), ("atr", 7001)])
def test_seed_is_the_rounded_mean(name, n, scale):
    rng = np.random.default_rng(12)
    lead = 7
    x = np.ldexp(1 + rng.random(n), scale).astype(np.float32)
    if name == "wilders":
        terms, ins = x, [x.copy()]
    else:
        spread = np.ldexp(rng.random((2, n)), scale - 3).astype(np.float32)
        h, l = x + spread[0], x - spread[1]
        terms = h - l  # f32, as every true range
        prev = x[:-1]
        terms[1:] = np.maximum(terms[1:], np.maximum(np.abs(h[1:] - prev), np.abs(l[1:] - prev)))
        terms[lead] = h[lead] - l[lead]
        ins = [h, l, x]
    ins = [a.copy() for a in ins]
    for a in ins:
        a[:lead] = np.nan
    hi = min(1900, n - lead - 1)
    got = V.CLASSES[name](0).batch_dev(*ins, sweep={"period": (2, hi, 1)}).to_host()
    exact = [float(t) for t in terms[lead:]]
    if name == "atr":  # the first true range enters exactly
        exact[0] = float(h[lead]) - float(l[lead])
    for p in range(2, hi + 1):
        want = np.float32(math.fsum(exact[:p]) / p)
        assert got[p - 2, lead + p - 1] == want, p
