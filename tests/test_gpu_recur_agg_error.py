"""The CUDA-core chunk aggregates against the tensor-core contraction's: the
2-norm of the output errors over an f64 reference is no larger (2% allowed
for the rounding of one series against another's order)."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def reference(name, x, periods):
    p = np.asarray(periods, dtype=np.float64)
    y = np.full((x.size, p.size), np.nan)
    if name == "ema":
        a, s = 2.0 / (p + 1.0), np.zeros_like(p)
        e = np.zeros_like(p)
        for t, v in enumerate(x):
            s = s + v * (t < p)
            e = np.where(t < p, s / (t + 1.0), e + a * (v - e))
            y[t] = e
        return y.T
    g = np.maximum(np.diff(x), 0.0)
    l = np.maximum(-np.diff(x), 0.0)
    ag, al = np.zeros_like(p), np.zeros_like(p)
    for t in range(1, x.size):
        gt, lt = g[t - 1], l[t - 1]
        warm = t <= p
        ag = np.where(warm, ag + gt / p, ag + (gt - ag) / p)
        al = np.where(warm, al + lt / p, al + (lt - al) / p)
        with np.errstate(invalid="ignore"):
            y[t] = np.where(t >= p, 100.0 * ag / (ag + al), np.nan)
    return y.T


@pytest.mark.parametrize("name,n,periods", [("rsi", 60_001, (2, 200, 3)), ("ema", 60_001, (5, 985, 20))])
def test_cuda_core_aggregates_are_as_exact(name, n, periods):
    x = datagen.random_walk(n, seed=5).astype(np.float32)
    ps = range(periods[0], periods[1] + 1, periods[2])
    want = reference(name, x.astype(np.float64), ps)
    err = []
    for agg in ("tc", "cuda"):
        ctx = V.Context(0)
        ctx.set_policy("tune", "off")
        ctx.set_policy("recur_agg", agg)
        ind = V.CLASSES[name](ctx=ctx)
        got = ind.batch_dev(x, sweep={"period": periods}).to_host().astype(np.float64)
        assert ("tc aggregates" in ind.last_kernel) == (agg == "tc")
        m = np.isfinite(want)
        assert np.array_equal(m, np.isfinite(got))
        err.append(np.linalg.norm(got[m] - want[m]) / np.linalg.norm(want[m]))
    assert err[1] <= 1.02 * err[0], err
