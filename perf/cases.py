"""Performance cases: the calls that users of the library make, each through
its public entry points, from one chart's moving averages to full parameter
grids, many-series screens, ragged plans and live stream banks.

A case is a dict of plain values; "call" says which entry point it takes:

  batch_device  CudaX.batch_device: one device-resident series (or high / low /
                close), a sweep of parameters, the caller's output buffers
  batch_dev     CudaX.batch_dev: host arrays in, a new device array out
  many_series   CudaX.many_series_one_param_device over a time-major matrix,
                one call for each of the case's indicators
  plan          TmPlan.run: ATR, ADX, SuperTrend and percentile over ragged
                series in one work list
  streams       StreamBank.update_device: one bar for every stream of each bank
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

# input series and outputs of the indicators used here
INPUTS = {"willr": 3, "adx": 3, "atr": 3, "donchian": 2}
OUTPUTS = {"bollinger_bands": 3, "donchian": 3}
# fixed parameters of the many-series and stream cases: the usual chart settings
SCREEN = {"sma": {"period": 50}, "ema": {"period": 20}, "rsi": {"period": 14}, "atr": {"period": 14},
          "bollinger_bands": {"period": 20, "devup": 2.0, "devdn": 2.0}, "donchian": {"period": 20},
          "willr": {"period": 14}, "alma": {"period": 9, "offset": 0.85, "sigma": 6.0}}
BANKS = {"ema": {"period": 20}, "sma": {"period": 50}, "rsi": {"period": 14}, "atr": {"length": 14},
         "bollinger_bands": {"period": 20, "devup": 2.0, "devdn": 2.0, "matype": "sma"}, "donchian": {"period": 20}}
STREAM_WARM = 64  # bars a bank has seen before the measured update
PLAN_JOBS = (("atr", 14, 0.0), ("adx", 14, 0.0), ("supertrend", 10, 3.0), ("percentile_nearest_rank", 50, 50.0))


def listed():
    return [
        # a chart redraw: a handful of EMAs over a thousand bars
        {"name": "ema_chart", "call": "batch_device", "indicator": "ema", "bars": 1001, "lead": 0,
         "lo": 5, "hi": 50, "step": 5},
        # the full recurrence grid of a strategy search (the default benchmark's EMA sweep)
        {"name": "ema_grid", "call": "batch_device", "indicator": "ema", "bars": 1_000_000, "lead": 200,
         "lo": 2, "hi": 1000, "step": 1},
        # an RSI sweep over a recorded history of whatever length it has
        {"name": "rsi_history", "call": "batch_device", "indicator": "rsi", "bars": 100_003, "lead": 17,
         "lo": 2, "hi": 201, "step": 1},
        # the ALMA grid: periods x offsets x sigmas, 17,920 combinations
        {"name": "alma_grid", "call": "batch_device", "indicator": "alma", "bars": 200_000, "lead": 0,
         "lo": 5, "hi": 260, "step": 1, "o0": 0.5, "o1": 0.95, "os": 0.05, "s0": 3.0, "s1": 9.0, "ss": 1.0},
        # the crate's x_batch_dev: a notebook passes a host array and gets a device array
        {"name": "alma_from_host", "call": "batch_dev", "indicator": "alma", "bars": 20_001, "lead": 11,
         "lo": 9, "hi": 240, "step": 1, "o0": 0.85, "o1": 0.85, "os": 0.0, "s0": 6.0, "s1": 6.0, "ss": 0.0},
        # Bollinger bands over the crate's default range
        {"name": "bollinger_range", "call": "batch_device", "indicator": "bollinger_bands", "bars": 200_000,
         "lead": 100, "lo": 20, "hi": 269, "step": 1, "k": 2.0},
        # Williams %R windows of the default benchmark
        {"name": "willr_grid", "call": "batch_device", "indicator": "willr", "bars": 1_000_000, "lead": 200,
         "lo": 5, "hi": 500, "step": 5},
        # the ADX sweep of the benchmark
        {"name": "adx_grid", "call": "batch_device", "indicator": "adx", "bars": 1_000_000, "lead": 100,
         "lo": 2, "hi": 400, "step": 1},
        # the running median over the crate's default range of lengths
        {"name": "percentile_range", "call": "batch_device", "indicator": "percentile_nearest_rank",
         "bars": 100_000, "lead": 50, "lo": 15, "hi": 264, "step": 1, "k": 50.0},
        # a daily screen: ten years of 3,000 symbols, six indicators
        {"name": "daily_screen", "call": "many_series", "indicators": "sma rsi atr bollinger_bands donchian alma",
         "series": 3000, "rows": 2520, "leads": 250},
        # ragged histories of many symbols in one plan
        {"name": "ragged_plan", "call": "plan", "series": 1024, "rows": 20_000, "leads": 500},
        # one bar of a live feed
        {"name": "live_bar", "call": "streams", "indicators": "ema rsi bollinger_bands atr", "streams": 8192},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _axis(rng, combos, lo, hi):
    """A period axis of about `combos` values within [lo, hi]."""
    combos = max(1, min(combos, hi - lo + 1))
    step = rng.randint(1, max(1, min(10, (hi - lo) // combos)))
    start = rng.randint(lo, max(lo, hi - (combos - 1) * step))
    return {"lo": start, "hi": min(hi, start + (combos - 1) * step), "step": step}


def draw(rng):
    call = rng.choice(["recurrence", "weighted", "host", "window", "minmax", "adx", "percentile", "many_series",
                       "plan", "streams"])
    if call == "recurrence":
        bars = _log(rng, 1001, 1_000_000)
        return {"call": "batch_device", "indicator": rng.choice(["ema", "dema", "tema", "rsi"]), "bars": bars,
                "lead": rng.randint(0, 200), **_axis(rng, _log(rng, 8, 999), 2, min(1000, bars // 5))}
    if call in ("weighted", "host"):
        grid = call == "weighted"
        ind = rng.choice(["alma", "wma"])
        bars = _log(rng, 2000, 200_000 if grid else 100_000)
        ax = _axis(rng, _log(rng, 16, 256), 5, 260)
        c = {"call": "batch_device" if grid else "batch_dev", "indicator": ind, "bars": bars,
             "lead": rng.randint(0, 200), **ax}
        if ind == "alma":
            no, ns = (rng.randint(1, 10), rng.randint(1, 7)) if grid else (1, 1)
            c.update(o0=0.5, o1=0.5 + 0.05 * (no - 1), os=0.05, s0=3.0, s1=3.0 + (ns - 1), ss=1.0)
        return c
    if call == "window":
        return {"call": "batch_device", "indicator": rng.choice(["sma", "stddev", "zscore", "bollinger_bands"]),
                "bars": _log(rng, 2000, 1_000_000), "lead": rng.randint(0, 200),
                **_axis(rng, _log(rng, 5, 250), 5, 500), "k": rng.choice([1.0, 2.0, 2.5])}
    if call == "minmax":
        return {"call": "batch_device", "indicator": rng.choice(["willr", "donchian"]),
                "bars": _log(rng, 2000, 1_000_000), "lead": rng.randint(0, 200),
                **_axis(rng, _log(rng, 5, 250), 5, 500)}
    if call == "adx":
        return {"call": "batch_device", "indicator": "adx", "bars": _log(rng, 5000, 1_000_000),
                "lead": rng.randint(0, 200), **_axis(rng, _log(rng, 5, 399), 2, 400)}
    if call == "percentile":
        return {"call": "batch_device", "indicator": "percentile_nearest_rank", "bars": _log(rng, 2000, 100_000),
                "lead": rng.randint(0, 200), **_axis(rng, _log(rng, 5, 250), 5, 264),
                "k": rng.choice([10.0, 25.0, 50.0, 75.0, 90.0])}
    if call == "many_series":
        inds = rng.sample(sorted(SCREEN), rng.randint(1, 6))
        return {"call": "many_series", "indicators": " ".join(inds), "series": _log(rng, 100, 4096),
                "rows": _log(rng, 500, 4000), "leads": rng.randint(1, 250)}
    if call == "plan":
        return {"call": "plan", "series": _log(rng, 64, 1024), "rows": _log(rng, 2000, 20_000),
                "leads": rng.randint(1, 500)}
    inds = rng.sample(sorted(BANKS), rng.randint(1, 4))
    return {"call": "streams", "indicators": " ".join(inds), "streams": _log(rng, 500, 100_000)}


# ------------------------------------------------------------------ inputs --
_CTX: list = []


def _ctx():
    """The program's one context (its stream and workspaces)."""
    if not _CTX:
        _CTX.append(V.Context(0))
    return _CTX[0]


def _series(case, seed):
    """One series as float32 host arrays: [close], [high, low] or [high, low, close]."""
    n, lead = case["bars"], case["lead"]
    close = datagen.random_walk(n, seed=seed, nan_lead=lead)
    n_in = INPUTS.get(case["indicator"], 1)
    if n_in == 1:
        return [close.astype(np.float32)]
    hi, lo = datagen.high_low(close, seed=seed)
    return [a.astype(np.float32) for a in ([hi, lo] if n_in == 2 else [hi, lo, close])]


def _matrix(rows, cols, seed, leads, lengths=None):
    """Time-major float32 high, low, close on the GPU: random walks around 100
    with 1% steps, a NaN lead per series, and a NaN tail past `lengths`."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    eps = torch.randn(rows, cols, generator=g, device="cuda", dtype=torch.float64).mul_(0.01)
    close = torch.cumsum(eps, 0).exp_().mul_(100.0)
    spread = torch.randn(2, rows, cols, generator=g, device="cuda", dtype=torch.float64).mul_(0.005).abs_()
    lead = torch.randint(0, leads + 1, (cols,), generator=g, device="cuda")
    t = torch.arange(rows, device="cuda")[:, None]
    gone = t < lead
    if lengths is not None:
        gone = gone | (t >= lengths)
    out = []
    for a in (close * (1.0 + spread[0]), close * (1.0 - spread[1]), close):
        a = a.to(torch.float32)
        a[gone] = float("nan")
        out.append(a)
    return out[0], out[1], out[2], lead


def _lengths(case, seed):
    """Series lengths of a plan, uniform in [1000, rows]; the last row is in use."""
    lens = np.random.default_rng(seed).integers(1000, case["rows"] + 1, case["series"])
    lens[0] = case["rows"]
    return lens


def _sweep(case):
    per = (case["lo"], case["hi"], case["step"])
    ind = case["indicator"]
    if ind == "alma":
        return {"period": per, "offset": (case["o0"], case["o1"], case["os"]),
                "sigma": (case["s0"], case["s1"], case["ss"])}
    if ind in ("stddev", "zscore"):
        return {"period": per, "nbdev": (case["k"], case["k"], 0.0)}
    if ind == "bollinger_bands":
        return {"period": per, "devup": (case["k"], case["k"], 0.0), "devdn": (case["k"], case["k"], 0.0)}
    if ind == "percentile_nearest_rank":
        return {"length": per, "percentage": (case["k"], case["k"], 0.0)}
    return {"period": per}


def _grid(case):
    """The sweep's combinations: [(period, offset, sigma)] for ALMA, [(period,)] otherwise."""
    ps = list(range(case["lo"], case["hi"] + 1, case["step"]))
    if case["indicator"] != "alma":
        return [(p,) for p in ps]

    def axis(a, b, s):
        if abs(s) < 1e-12 or abs(a - b) < 1e-12:
            return [a]
        v, x = [], a
        while x <= b + 1e-12:
            v.append(x)
            x += s
        return v

    return [(p, o, s) for p in ps for o in axis(case["o0"], case["o1"], case["os"])
            for s in axis(case["s0"], case["s1"], case["ss"])]


def _bank_inputs(ind, high, low, close):
    return {"atr": [high, low, close], "donchian": [high, low]}.get(ind, [close])


def prepare(case, seed):
    call, st = case["call"], {"case": case}
    if call == "batch_device":
        st["obj"] = V.CLASSES[case["indicator"]](ctx=_ctx())
        st["sweep"] = _sweep(case)
        st["ins"] = [torch.from_numpy(a).cuda() for a in _series(case, seed)]
        rows = len(_grid(case))
        st["outs"] = [torch.empty(rows, case["bars"], device="cuda") for _ in range(OUTPUTS.get(case["indicator"], 1))]
    elif call == "batch_dev":
        st["obj"] = V.CLASSES[case["indicator"]](ctx=_ctx())
        st["sweep"] = _sweep(case)
        st["ins"] = _series(case, seed)
    elif call == "many_series":
        hlc = _matrix(case["rows"], case["series"], seed, case["leads"])[:3]
        st["work"] = []
        for ind in case["indicators"].split():
            ins = {1: [hlc[2]], 2: list(hlc[:2]), 3: list(hlc)}[INPUTS.get(ind, 1)]
            outs = [torch.empty_like(hlc[2]) for _ in range(OUTPUTS.get(ind, 1))]
            st["work"].append((ind, V.CLASSES[ind](ctx=_ctx()), ins, SCREEN[ind], outs))
    elif call == "plan":
        lens = _lengths(case, seed)
        hlc = _matrix(case["rows"], case["series"], seed, case["leads"], torch.from_numpy(lens).cuda())[:3]
        st["outs"], jobs = {}, []
        for kind, period, param in PLAN_JOBS:
            o = [torch.full_like(hlc[2], float("nan")) for _ in range(2 if kind == "supertrend" else 1)]
            st["outs"][kind] = o
            jobs.append({"kind": kind, "period": period, "param": param, "out0": o[0],
                         "out1": o[1] if len(o) > 1 else None})
        torch.cuda.synchronize()
        st["plan"] = V.TmPlan(*hlc, case["series"], case["rows"], lens, jobs, ctx=_ctx())
    else:
        high, low, close = _matrix(STREAM_WARM + 1, case["streams"], seed, 0)[:3]
        torch.cuda.synchronize()
        st["work"] = []
        for ind in case["indicators"].split():
            bank = V.StreamBank(ind, case["streams"], BANKS[ind], ctx=_ctx())
            out = torch.empty(bank.n_outputs, case["streams"], device="cuda")
            ins = _bank_inputs(ind, high, low, close)
            for t in range(STREAM_WARM):
                bank.update_device(*[a[t] for a in ins], d_out=out)
            st["work"].append((ind, bank, [a[STREAM_WARM] for a in ins], out))
    torch.cuda.synchronize()  # the library runs on its own stream
    return st


def run(st):
    case = st["case"]
    call = case["call"]
    if call == "batch_device":
        st["obj"].batch_device(st["ins"], case["bars"], case["lead"], st["sweep"], st["outs"])
        return st["outs"]
    if call == "batch_dev":
        return torch.as_tensor(st["obj"].batch_dev(*st["ins"], sweep=st["sweep"]), device="cuda")
    if call == "many_series":
        for _, obj, ins, params, outs in st["work"]:
            obj.many_series_one_param_device(ins, case["series"], case["rows"], params, outs)
        return {ind: outs for ind, _, _, _, outs in st["work"]}
    if call == "plan":
        st["plan"].run()
        return st["outs"]
    for _, bank, ins, out in st["work"]:
        bank.update_device(*ins, d_out=out)
    return {ind: out for ind, _, _, out in st["work"]}


def work(case):
    call = case["call"]
    if call in ("batch_device", "batch_dev"):
        ind, n, grid = case["indicator"], case["bars"], _grid(case)
        flops = 2.0 * n * sum(g[0] for g in grid) if ind in ("alma", "wma") else 0.0
        return {"bytes": 4.0 * n * (INPUTS.get(ind, 1) + len(grid) * OUTPUTS.get(ind, 1)), "flops": flops}
    if call == "many_series":
        cells = case["rows"] * case["series"]
        return {"bytes": 4.0 * cells * sum(INPUTS.get(i, 1) + OUTPUTS.get(i, 1) for i in case["indicators"].split()),
                "flops": 0.0}
    if call == "plan":  # lengths are uniform in [1000, rows]; 3 inputs and 5 outputs of each cell in use
        return {"bytes": 4.0 * 8 * case["series"] * 0.5 * (1000 + case["rows"]), "flops": 0.0}
    return {"bytes": 4.0 * case["streams"] * sum(
        len(_bank_inputs(i, 0, 0, 0)) + OUTPUTS.get(i, 1) for i in case["indicators"].split()), "flops": 0.0}


# ------------------------------------------------- 64-bit reference values --
def _linrec(v, b):
    """y[c][t] = b[c] y[c][t-1] + v[c][t] from y = 0, in blocks of 256 steps."""
    C, T = v.shape
    B = min(256, T)
    i = torch.arange(B, device=v.device, dtype=torch.float64)
    e = i[None, :] - i[:, None]  # [j][i]: i - j
    L = torch.where(e >= 0, b[:, None, None] ** e.clamp(min=0.0), 0.0)  # [c][j][i]
    if T <= B:
        return torch.bmm(v[:, None, :], L)[:, 0]
    nb = -(-T // B)
    y = torch.bmm(torch.nn.functional.pad(v, (0, nb * B - T)).reshape(C, nb, B), L)
    ends = _linrec(y[:, :, -1], b ** B)
    y[:, 1:] += ends[:, :-1, None] * (b[:, None] ** (i + 1.0))[:, None, :]
    return y.reshape(C, nb * B)[:, :T]


def _started(u, a, b, at, seed):
    """y[at] = seed, y[t] = b y[t-1] + a u[t] after; NaN-free zeros before.
    u is [T] or [C][T], the others are per row."""
    t = torch.arange(u.shape[-1], device=u.device)
    v = torch.where(t > at[:, None], a[:, None] * u, 0.0)
    v = torch.where(t == at[:, None], seed[:, None], v)
    return _linrec(v, b)


def _hide(y, until):
    """NaN before each row's first output."""
    t = torch.arange(y.shape[-1], device=y.device)
    return torch.where(t < until[:, None], float("nan"), y)


def _sums(x, first, count):
    """Sums of x[first : first + count] per row; x is [T] or [C][T]."""
    t = torch.arange(x.shape[-1], device=x.device)
    m = (t >= first[:, None]) & (t < (first + count)[:, None])
    return torch.where(m, x, 0.0).sum(-1)


def _at(x, i):
    return x[i] if x.dim() == 1 else x.gather(1, i[:, None])[:, 0]


def _recurrence(ind, ins, first, p):
    """EMA / DEMA / TEMA / RSI / ATR / ADX rows for periods p from first valid
    indices `first` ([C] tensors); the inputs are [T] (a sweep) or [C][T]."""
    x = ins[-1]
    f, pd = first, p.to(torch.float64)
    if ind in ("ema", "dema", "tema"):
        a = 2.0 / (pd + 1.0)
        if ind == "ema":
            seed = _sums(x, f, p) / pd
            y = _started(x, a, 1.0 - a, f + p - 1, seed)
            t = torch.arange(x.shape[-1], device=x.device)
            c = torch.where(t >= f[:, None], x, 0.0).cumsum(-1) / (t - f[:, None] + 1.0)
            return _hide(torch.where(t < (f + p - 1)[:, None], c, y), f)
        e1 = _started(x, a, 1.0 - a, f, _at(x, f))
        if ind == "dema":
            return _hide(2.0 * e1 - _started(e1, a, 1.0 - a, f, _at(e1, f)), f + p - 1)
        last = x.shape[-1] - 1
        s2, s3 = (f + p - 1).clamp(max=last), (f + 2 * (p - 1)).clamp(max=last)
        e2 = _started(e1, a, 1.0 - a, s2, _at(e1, s2))
        e3 = _started(e2, a, 1.0 - a, s3, _at(e2, s3))
        return _hide(3.0 * e1 - 3.0 * e2 + e3, f + 3 * (p - 1))
    r = 1.0 / pd
    if ind == "rsi":
        d = torch.nn.functional.pad(x[..., 1:] - x[..., :-1], (1, 0))
        g, lo = d.clamp(min=0.0), (-d).clamp(min=0.0)
        ag = _started(g, r, 1.0 - r, f + p, _sums(g, f + 1, p) * r)
        al = _started(lo, r, 1.0 - r, f + p, _sums(lo, f + 1, p) * r)
        return _hide(torch.where(ag + al == 0.0, 50.0, 100.0 * ag / (ag + al)), f + p)
    h, lo, c = ins
    pc = torch.nn.functional.pad(c[..., :-1], (1, 0))
    tr = torch.maximum(torch.maximum(h - lo, (h - pc).abs()), (lo - pc).abs())
    if ind == "atr":
        t = torch.arange(x.shape[-1], device=x.device)
        tr = torch.where(t == f[:, None], h - lo, tr)
        return _hide(_started(tr, r, 1.0 - r, f + p - 1, _sums(tr, f, p) * r), f + p - 1)
    up = torch.nn.functional.pad(h[..., 1:] - h[..., :-1], (1, 0))
    dn = torch.nn.functional.pad(lo[..., :-1] - lo[..., 1:], (1, 0))
    one = torch.ones_like(r)
    level = [_started(u, one, 1.0 - r, f + p, _sums(u, f + 1, p))
             for u in (torch.where((up > dn) & (up > 0.0), up, 0.0), torch.where((dn > up) & (dn > 0.0), dn, 0.0))]
    den = level[0] + level[1]
    dx = torch.where(den == 0.0, 0.0, 100.0 * (level[0] - level[1]).abs() / den)
    return _hide(_started(dx, r, 1.0 - r, f + 2 * p - 1, _sums(dx, f + p, p) * r), f + 2 * p - 1)


def _window_max(x, p):
    """max over [t - p + 1, t] along the last axis (-inf padded), by doubling."""
    m, w = x, 1
    while 2 * w <= p:
        m = torch.maximum(m, torch.nn.functional.pad(m[..., :-w], (w, 0), value=-math.inf))
        w *= 2
    s = p - w
    return torch.maximum(m, torch.nn.functional.pad(m[..., :-s], (s, 0), value=-math.inf)) if s else m


def _windows(ind, ins, first, p, k, k2=0.0):
    """One window length p for every row of the inputs ([R][T], NaN where not valid)."""
    x = ins[-1]
    until = first + p - 1
    if ind in ("willr", "donchian"):
        hi = _window_max(torch.nan_to_num(ins[0], nan=-math.inf), p)
        lo = -_window_max(torch.nan_to_num(-ins[1], nan=-math.inf), p)
        if ind == "willr":
            return [_hide(torch.where(hi == lo, 0.0, -100.0 * (hi - x) / (hi - lo)), until)]
        return [_hide(v, until) for v in (hi, (hi - lo) * 0.5 + lo, lo)]
    out = [torch.full_like(x, float("nan")) for _ in range(OUTPUTS.get(ind, 1))]
    for r0 in range(0, x.shape[0], 64):  # windows of 64 rows at a time
        xr = x[r0:r0 + 64]
        for t0 in range(0, xr.shape[1] - p + 1, 1 << 18):
            w = xr[:, t0:t0 + (1 << 18) + p - 1].unfold(1, p, 1)
            to = slice(t0 + p - 1, t0 + p - 1 + w.shape[1])
            if ind == "percentile_nearest_rank":
                rank = min(p - 1, max(0, int(math.floor(k * 0.01 * p + 0.5)) - 1))
                out[0][r0:r0 + 64, to] = w.sort(-1).values[..., rank]  # (NaN sorts last)
                continue
            mean = w.mean(-1)
            if ind == "sma":
                out[0][r0:r0 + 64, to] = mean
                continue
            sd = (w - mean[..., None]).square_().mean(-1).sqrt_()
            if ind == "stddev":
                out[0][r0:r0 + 64, to] = sd * k
            elif ind == "zscore":
                out[0][r0:r0 + 64, to] = torch.where(sd == 0.0, float("nan"), (w[..., -1] - mean) / (sd * k))
            else:
                out[0][r0:r0 + 64, to] = mean + k * sd
                out[1][r0:r0 + 64, to] = mean
                out[2][r0:r0 + 64, to] = mean - k2 * sd
    return [_hide(o, until) for o in out]


def _weights(ind, g, kmax):
    """The normalised weights of one combination, right-aligned in kmax."""
    p = g[0]
    i = np.arange(p, dtype=np.float64)
    if ind == "wma":
        w = i + 1.0
    else:
        m, s = g[1] * (p - 1), p / g[2]
        w = np.exp(-((i - m) ** 2) / (2.0 * s * s))
    return np.concatenate([np.zeros(kmax - p), w / w.sum()])


def _weighted(ind, x, first, grid):
    kmax = max(g[0] for g in grid)
    n = x.shape[0]
    out = torch.empty(len(grid), n, dtype=torch.float64, device=x.device)
    padded = torch.nn.functional.pad(torch.nan_to_num(x, nan=0.0), (kmax - 1, 0))
    hankel = padded.unfold(0, kmax, 1)  # [n][kmax]
    for c0 in range(0, len(grid), 512):
        w = torch.from_numpy(np.stack([_weights(ind, g, kmax) for g in grid[c0:c0 + 512]])).to(x.device)
        for t0 in range(0, n, 1 << 17):
            out[c0:c0 + 512, t0:t0 + (1 << 17)] = w @ hankel[t0:t0 + (1 << 17)].t()
    for c, g in enumerate(grid):
        out[c, :first + g[0] - 1] = float("nan")
    return out


def _rows64(ind, ins, first, params):
    """One parameter set over the rows of [R][T] inputs (NaN before `first`)."""
    p = params.get("period", params.get("length", 0))
    if ind in ("ema", "rsi", "atr", "adx"):
        zeroed = [torch.nan_to_num(a, nan=0.0) for a in ins]
        return [_recurrence(ind, zeroed, first, torch.full_like(first, p))]
    if ind == "alma":
        w = torch.from_numpy(_weights(ind, (p, params["offset"], params["sigma"]), p)).to(first.device)
        y = torch.nn.functional.pad(torch.nan_to_num(ins[0], nan=0.0), (p - 1, 0)).unfold(1, p, 1) @ w
        return [_hide(y, first + p - 1)]
    return _windows(ind, ins, first, p, params.get("devup", params.get("percentage", 1.0)), params.get("devdn", 1.0))


def exact(case, seed):
    call, f64 = case["call"], torch.float64
    if call in ("batch_device", "batch_dev"):
        ind, n, grid = case["indicator"], case["bars"], _grid(case)
        ins = [torch.from_numpy(a).cuda().to(f64) for a in _series(case, seed)]
        if ind in ("alma", "wma"):
            y = _weighted(ind, ins[0], case["lead"], grid)
            return y if call == "batch_dev" else [y]
        if ind in ("ema", "dema", "tema", "rsi", "adx"):
            zeroed = [torch.nan_to_num(a, nan=0.0) for a in ins]
            out = torch.empty(len(grid), n, dtype=f64, device="cuda")
            for c0 in range(0, len(grid), 64):
                p = torch.tensor([g[0] for g in grid[c0:c0 + 64]], device="cuda")
                out[c0:c0 + 64] = _recurrence(ind, zeroed, torch.full_like(p, case["lead"]), p)
            return [out]
        first = torch.tensor([case["lead"]], device="cuda")
        outs = [torch.empty(len(grid), n, dtype=f64, device="cuda") for _ in range(OUTPUTS.get(ind, 1))]
        rows = [a[None] for a in ins]
        for c, g in enumerate(grid):
            for o, v in zip(outs, _windows(ind, rows, first, g[0], case.get("k", 1.0), case.get("k", 1.0))):
                o[c] = v[0]
        return outs
    if call == "many_series":
        *hlc, lead = _matrix(case["rows"], case["series"], seed, case["leads"])
        hlc = [a.to(f64).t().contiguous() for a in hlc]
        return {ind: [v.t() for v in _rows64(ind, {1: hlc[2:], 2: hlc[:2], 3: hlc}[INPUTS.get(ind, 1)], lead,
                                             SCREEN[ind])] for ind in case["indicators"].split()}
    if call == "plan":
        lens = torch.from_numpy(_lengths(case, seed)).cuda()
        *hlc, lead = _matrix(case["rows"], case["series"], seed, case["leads"], lens)
        hlc = [a.to(f64).t().contiguous() for a in hlc]
        past = torch.arange(case["rows"], device="cuda") >= lens[:, None]
        out = {"supertrend": [None, None]}  # its band flips are decisions, not rounded values
        for kind, p, param in PLAN_JOBS:
            if kind != "supertrend":
                ins = hlc[2:] if kind == "percentile_nearest_rank" else hlc
                y = torch.cat([_rows64(kind, [a[r:r + 128] for a in ins], lead[r:r + 128],
                                       {"period": p, "percentage": param})[0] for r in range(0, case["series"], 128)])
                out[kind] = [torch.where(past, float("nan"), y).t()]
        return out
    *hlc, lead = _matrix(STREAM_WARM + 1, case["streams"], seed, 0)
    hlc = [a.to(f64).t().contiguous() for a in hlc]
    out = {}
    for ind in case["indicators"].split():
        prm = {("period" if k == "length" else k): v for k, v in BANKS[ind].items()}
        out[ind] = torch.stack([v[:, -1] for v in _rows64(ind, _bank_inputs(ind, *hlc), lead, prm)])
    return out
