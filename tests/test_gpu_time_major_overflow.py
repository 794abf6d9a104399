"""Many-series windows whose squares overflow: which outputs an overflowing
window poisons (up to the next multiple of 512 rows) does not depend on how
many series there are, and so on the rows a thread slides over."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,p", [("stddev", 400), ("bollinger_bands", 320), ("zscore", 500), ("sma", 400)])
def test_poisoned_rows_do_not_depend_on_the_series_count(name, p):
    import torch

    rows, few, many = 2048, 64, 39_000  # 512 rows a thread for many, 256 for few
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(rows, few, device="cuda", generator=g) + 100.0
    # p values in a row whose squares sum to more than 2^128, each below 2^60
    v = float(np.sqrt(2.0**128 / (0.85 * p)))
    assert v < 2.0**60
    x[600:600 + p, ::2] = v
    x[900:900 + p, 1::4] = -v
    wide = torch.rand(rows, many, device="cuda", generator=g) + 100.0
    wide[:, :few] = x
    prm = {"period": p}
    if name == "bollinger_bands":
        prm.update(devup=2.0, devdn=2.0)
    elif name != "sma":
        prm.update(nbdev=1.0)
    n_out = 3 if name == "bollinger_bands" else 1
    got = []
    for m in (x, wide):
        ctx = V.Context(0)
        outs = [torch.empty_like(m) for _ in range(n_out)]
        torch.cuda.synchronize()
        V.CLASSES[name](ctx=ctx).many_series_one_param_device([m], m.shape[1], rows, prm, outs)
        ctx.synchronize()
        got.append([o[:, :few].cpu().numpy() for o in outs])
    for a, b in zip(*got):
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
    if name in ("stddev", "zscore"):
        assert not np.isfinite(got[0][0][600 + p - 1, 0])  # the window of the p values
