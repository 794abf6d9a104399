"""Prefix-window sweeps with long windows: a block's set-up grows with the
longest window, so their combos are not cut into as many blocks as short ones'
(126 us for the windows up to 5,000 when they were, 78 now; up to 2,500 47)."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def test_long_windows_are_not_cut_small():
    import torch

    x = torch.from_numpy(datagen.random_walk(300_001, seed=2).astype(np.float32)).cuda()
    out = torch.empty(100, x.numel(), device="cuda")
    ctx = V.Context(0)
    ctx.set_policy("timing", "on")
    sma = V.CudaSma(ctx=ctx)
    torch.cuda.synchronize()
    ms = []
    for step in (25, 50):
        best = 1e9
        for _ in range(10):
            sma.batch_device([x], x.numel(), 0, {"period": (step, 100 * step, step)}, [out])
            ctx.synchronize()
            best = min(best, ctx.kernel_ms)
        ms.append(best)
    assert ms[1] <= 2.2 * ms[0], ms
