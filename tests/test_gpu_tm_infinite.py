"""Many-series recurrences with infinite inputs: what a chunk hands to the next
one is what one pass over the series would.  RSI holds an infinite average for
ever (0 or NaN out of it, as the oracle); EMA skips it; Wilders' average, whose
oracle refuses an infinite first window, against the recurrence itself."""
import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def matrix(rows, p):
    cols = []
    for s, (at, val, w) in enumerate([(17, -np.inf, 40), (rows // 2, -np.inf, rows), (rows // 3, np.inf, 1),
                                      (rows // 3, -np.inf, 1), (p + 1, np.inf, rows), (3, np.inf, 1),
                                      (rows - 2, -np.inf, 1), (rows, 0.0, 0), (40, np.nan, 3)]):
        x = datagen.random_walk(rows, seed=s, nan_lead=s % 3).astype(np.float32)
        x[at:at + w] = val
        cols.append(x)
    return np.stack(cols * 4, 1)


def wilders(x, p):
    f = int(np.argmax(~np.isnan(x)))
    y = np.full(x.size, np.nan)
    with np.errstate(invalid="ignore"):
        y[f + p - 1] = x[f:f + p].sum() / p
        for t in range(f + p, x.size):
            y[t] = (x[t] - y[t - 1]) / p + y[t - 1]
    return y


@pytest.mark.parametrize("policy", ["auto", "64"])  # one launch up to 640 rows / three
@pytest.mark.parametrize("name", ["rsi", "wilders", "ema"])
@pytest.mark.parametrize("rows,p", [(257, 9), (640, 42), (1500, 14)])
def test_infinite_inputs(name, rows, p, policy):
    import torch

    x = matrix(rows, p)
    ctx = V.Context(0)
    ctx.set_policy("recur_chunk", policy)
    d = torch.from_numpy(x).cuda()
    out = torch.empty_like(d)
    torch.cuda.synchronize()
    V.CLASSES[name](ctx=ctx).many_series_one_param_device([d], x.shape[1], rows, {"period": p}, [out])
    ctx.synchronize()
    got = out.cpu().numpy().astype(np.float64)
    for s in range(x.shape[1]):
        exp = (wilders if name == "wilders" else getattr(O, name))(x[:, s].astype(np.float64), p)
        assert np.array_equal(np.isnan(got[:, s]), np.isnan(exp)), s
        m = np.isfinite(exp)
        assert np.array_equal(got[~m & ~np.isnan(exp), s], exp[~m & ~np.isnan(exp)])
        assert np.all(np.abs(got[m, s] - exp[m]) <= 1e-4 + 1e-5 * np.abs(exp[m])), s


@pytest.mark.parametrize("n", [56, 2049, 5000])
def test_infinity_in_a_batch_seed(n):
    x = datagen.random_walk(n, seed=1).astype(np.float32)
    x[20] = np.inf
    got = V.CudaWilders(0).batch_dev(x, sweep={"period": (10, 53, 1)}).to_host().astype(np.float64)
    for row, p in zip(got, range(10, 54)):
        exp = wilders(x.astype(np.float64), p)
        assert np.array_equal(np.isnan(row), np.isnan(exp)), p
        assert np.array_equal(np.isinf(row), np.isinf(exp)), p
