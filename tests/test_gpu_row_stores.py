"""Sweeps whose rows do not start at 32-byte sectors (lengths not a multiple of
eight): large outputs are stored cut at the sectors.  The rows must be those of
the same sweep on a padded series, whose rows do start at sectors, bit for bit
over the common bars: the chunks are the same, only the stores differ."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu

N = 72_001  # 240 rows: above the size from which stores are cut


def run(name, cols, sweep, chunk):
    ind = V.CLASSES[name](0)
    if chunk:
        ind.set_policy("recur_chunk", chunk)
    out = ind.batch_dev(*cols, sweep=sweep)
    outs = out if isinstance(out, (tuple, list)) else (out,)
    return [o.to_host() for o in outs]


def inputs(n, name):
    d = datagen.ohlcv(n, seed=71, nan_lead=33)
    if name in ("atr",):
        return tuple(np.asarray(d[k], np.float32) for k in ("high", "low", "close"))
    return (np.asarray(d["close"], np.float32),)


@pytest.mark.parametrize("chunk", ["96", "704", "1376"])
@pytest.mark.parametrize("extra", [0, 1, 2, 4, 5, 6])
@pytest.mark.parametrize("name", ["ema", "rsi", "atr"])
def test_recurrence_rows(name, extra, chunk):
    n = N + extra
    pad = (n + 7) // 8 * 8
    sweep = {"period": (2, 251, 1)}
    cols = inputs(pad, name)
    want = run(name, cols, sweep, chunk)
    got = run(name, tuple(np.ascontiguousarray(c[:n]) for c in cols), sweep, chunk)
    for g, w in zip(got, want):
        assert g.shape[1] == n
        assert np.array_equal(g, w[:, :n], equal_nan=True)


@pytest.mark.parametrize("gap", [None, 40_000])
@pytest.mark.parametrize("extra", [0, 1, 2, 5])
@pytest.mark.parametrize("name,n0,hi", [("bollinger_bands", 92_001, 254), ("sma", 200_001, 704), ("stddev", 92_001, 254)])
def test_prefix_window_rows(name, n0, hi, extra, gap):
    # a shifted tile may take its reference value one to seven bars away: the
    # rows agree to a few roundings of one f32 result
    n = n0 + extra
    pad = (n + 7) // 8 * 8
    sweep = {"period": (5, hi, 1), "devup": (2.0, 2.0, 0.0), "devdn": (2.0, 2.0, 0.0), "nbdev": (1.0, 1.0, 0.0)}
    (x,) = inputs(pad, name)
    if gap:
        x = x.copy()
        x[gap] = np.nan
    want = run(name, (x,), sweep, None)
    got = run(name, (np.ascontiguousarray(x[:n]),), sweep, None)
    for g, w in zip(got, want):
        w = w[:, :n]
        assert np.array_equal(np.isnan(g), np.isnan(w))
        d = np.abs(g - w)
        assert np.nanmax(d / np.maximum(np.abs(w), 1.0)) <= 1e-5


@pytest.mark.parametrize("gap", [None, 700])
@pytest.mark.parametrize("n", [1, 3, 29, 251, 253, 254, 257, 505, 1_537, 1_638, 2_047])
@pytest.mark.parametrize("rows", [130, 35, 2])
def test_tensor_core_rows(rows, n, gap):
    # four tensor maps and 252-bar time tiles against the CUDA-core kernel, at
    # the bound the two kernels are held to on aligned rows
    (x,) = inputs(n, "wma")
    x = np.where(np.isnan(x), np.float32(50), x) if n < 600 else x.copy()
    if gap and gap < n:
        x[gap] = np.nan
    sweep = {"period": (1, min(rows, n - int(np.isnan(x[0])) * 33), 1)}
    res = []
    for policy in ("plain", "tc_fp16x3"):
        ind = V.CLASSES["swma"](0)
        ind.set_policy("wma_batch", policy)
        res.append(ind.batch_dev(x, sweep=sweep).to_host())
        assert policy == "plain" or ind.last_kernel == "wwma_tc_fp16x3"
    w, g = res
    assert np.array_equal(np.isnan(g), np.isnan(w))
    d = np.abs(g - w) / np.abs(w)
    assert np.all(np.isnan(d)) or np.nanmax(d) < 2e-6


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 5])
@pytest.mark.parametrize("n", [2_048, 2_049])
@pytest.mark.parametrize("name", ["wma", "ema", "sma"])
def test_outputs_at_any_float(name, n, offset):
    # rows written inside a larger buffer: nothing outside them changes
    import torch
    (x,) = inputs(n, name)
    sweep = {"period": (5, 74, 1)}
    rows = 70
    ind = V.CLASSES[name](0)
    if name == "wma":
        ind.set_policy("wma_batch", "tc_fp16x3")
    want = ind.batch_dev(x, sweep=sweep).to_host()
    xd = torch.from_numpy(x).cuda()
    buf = torch.full((rows * n + 64,), 7.0, device="cuda")
    out = buf[16 + offset:16 + offset + rows * n]
    torch.cuda.synchronize()
    ind.batch_device(xd, n, 33, sweep, out)
    ind.synchronize()
    got = out.cpu().numpy().reshape(rows, n)
    if name == "wma":
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.nanmax(np.abs(got - want) / np.abs(want)) < 2e-6
    else:
        assert np.array_equal(got, want, equal_nan=True)
    assert bool((buf[:16 + offset] == 7.0).all()) and bool((buf[16 + offset + rows * n:] == 7.0).all())


@pytest.mark.parametrize("extra", [0, 1, 2, 5, 6])
def test_adx_scan_rows(extra):
    # same chunks, same carries: only the stores differ
    n = 280_001 + extra
    pad = (n + 7) // 8 * 8
    d = datagen.ohlcv(pad, seed=74, nan_lead=33)
    cols = tuple(np.asarray(d[k], np.float32) for k in ("high", "low", "close"))
    res = []
    for m in (pad, n):
        ind = V.CLASSES["adx"](0)
        ind.set_policy("scan_chunk", "1056")
        res.append(ind.batch_dev(*(np.ascontiguousarray(c[:m]) for c in cols),
                                 sweep={"period": (160, 409, 1)}).to_host())
        assert "exact scan" in ind.last_kernel
    assert np.array_equal(res[1], res[0][:, :n], equal_nan=True)
