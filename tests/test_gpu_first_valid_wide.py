"""The first-valid scan of very many series (blocks of 4 warps, 32 rows a round,
past 9,728 series; 32 warps up to there): the same outputs as for the series in
a narrow matrix, with leads at the edges of both rounds; and short leads cost
no more than a fraction of the call."""
import time

import numpy as np
import pytest

from vectorta_gb300 import cuda as V

pytestmark = pytest.mark.gpu
LEADS = (0, 1, 7, 8, 31, 32, 33, 63, 64, 255, 256, 257, 299)


@pytest.mark.parametrize("cols", [9728, 9729, 12_345])
@pytest.mark.parametrize("name,n_in,n_out", [("donchian", 2, 3), ("sma", 1, 1), ("adx", 3, 1)])
def test_wide_matches_narrow(name, n_in, n_out, cols):
    import torch

    rows = 340
    g = torch.Generator(device="cuda").manual_seed(2)
    c = torch.rand(rows, cols, device="cuda", generator=g) + 100.0
    ins = [c + 0.5, c - 0.5, c][:n_in] if n_in > 1 else [c]
    pick = [i * (cols - 1) // (len(LEADS) - 1) for i in range(len(LEADS))]
    for s, lead in zip(pick, LEADS):
        for a in ins:
            a[:lead, s] = float("nan")
    out = []
    for xs in (ins, [a[:, pick].contiguous() for a in ins]):
        ctx = V.Context(0)
        ys = [torch.empty_like(xs[0]) for _ in range(n_out)]
        torch.cuda.synchronize()
        V.CLASSES[name](ctx=ctx).many_series_one_param_device(xs, xs[0].shape[1], rows, {"period": 9}, ys)
        ctx.synchronize()
        out.append(ys)
    for a, b in zip(*out):
        a = a[:, pick].cpu().numpy()
        b = b.cpu().numpy()
        assert np.array_equal(np.isnan(a), np.isnan(b))
        for i, lead in enumerate(LEADS):
            assert np.isnan(a[:min(rows, lead + 8), i]).all()
        assert np.allclose(a, b, rtol=1e-5, equal_nan=True)


def test_short_leads_of_many_series_cost_little():
    import torch

    took = []
    for rows in (32, 250):  # a scan of 256 rows reads all of the second
        c = torch.rand(rows, 50_000, device="cuda") + 100.0
        ins = [c + 0.5, c - 0.5]
        ys = [torch.empty_like(c) for _ in range(3)]
        ctx = V.Context(0)
        don = V.CudaDonchian(ctx=ctx)
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(10):
            t = time.perf_counter()
            for _ in range(20):
                don.many_series_one_param_device(ins, 50_000, rows, {"period": 14}, ys)
            ctx.synchronize()
            best = min(best, time.perf_counter() - t)
        took.append(best / 20)
    assert took[1] - took[0] <= 57e-6, took  # 46 us; 67 with the scan of all rows
