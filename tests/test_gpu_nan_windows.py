"""Weighted windows over NaN bars far behind the output: windows whose oldest
bar is the NaN, or one past it, up to 3,400 bars back (a warp searches 1,024
bars a step), in rows of every alignment, against the oracle; and the time of
a series with one early NaN against a clean one's."""
import numpy as np
import pytest

from oracle import oracle as O
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [9000, 9001, 9002, 9003])
@pytest.mark.parametrize("nans", [(300,), (4095,), (4096, 4097), (31, 5119, 5120, 8991)], ids=str)
@pytest.mark.parametrize("name,rng", [("wma", (1500, 3400, 950)), ("alma", (4, 3398, 33)), ("alma", (1022, 1028, 1)),
                                      ("srwma", (2047, 2051, 1))])
def test_nan_far_back(name, rng, nans, n):
    x = datagen.random_walk(n, seed=8, nan_lead=5).astype(np.float32)
    x[list(nans)] = np.nan
    xd = x.astype(np.float64)
    sweep = {"period": rng}
    if name == "alma":
        sweep.update(offset=(0.85, 0.85, 0.0), sigma=(6.0, 6.0, 0.0))
    ind = V.CLASSES[name](0)
    got = ind.batch_dev(x, sweep=sweep).to_host()
    assert ind.last_kernel == "wwma_tc_fp16x3"
    fn = {"alma": lambda p: O.alma(xd, p, 0.85, 6.0), "wma": lambda p: O.wma(xd, p), "srwma": lambda p: O.srwma(xd, p)}[name]
    for row, g in zip(got, ind.expand_grid(sweep)):
        assert np.array_equal(np.isnan(row), np.isnan(fn(g["period"]))), g


def test_one_nan_costs_little():
    import torch

    x = datagen.random_walk(200_000, seed=8).astype(np.float32)
    ms = []
    for at in (None, 300):
        y = x.copy()
        if at:
            y[at] = np.nan
        ctx = V.Context(0)
        ctx.set_policy("timing", "on")
        alma = V.CudaAlma(ctx=ctx)
        sweep = {"period": (9, 2000, 9), "offset": (0.85, 0.85, 0.0), "sigma": (6.0, 6.0, 0.0)}
        d = torch.from_numpy(y).cuda()
        out = torch.empty(len(alma.expand_grid(sweep)), y.size, device="cuda")
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(8):
            alma.batch_device([d], y.size, 0, sweep, [out])
            ctx.synchronize()
            best = min(best, ctx.kernel_ms)
        ms.append(best)
    assert ms[1] <= 2 * ms[0], ms
