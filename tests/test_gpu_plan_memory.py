"""A plan on a nearly full GPU: the short chunks tried at its creation do not
take the memory that longer ones leave (in a process of its own)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import sys, torch
sys.path.insert(0, sys.argv[1])
from vectorta_gb300 import cuda as V
cols, rows = 20_000, 4000
g = torch.Generator(device="cuda").manual_seed(1)
c = torch.rand(rows, cols, device="cuda", generator=g) + 100.0
h, l = c + 0.5, c - 0.5
outs = [torch.empty_like(c) for _ in range(2)]
jobs = [{"kind": k, "period": 14, "param": 0.0, "out0": o} for k, o in zip(("atr", "adx"), outs)]
ctx = V.Context(0)
small = [{"kind": k, "period": 14, "param": 0.0, "out0": o} for k, o in zip(("atr", "adx"), outs)]
V.TmPlan(h, l, c, 64, 500, None, small, ctx=ctx).run()  # (loads the kernels)
torch.cuda.synchronize()
torch.cuda.empty_cache()
if sys.argv[2] == "cached":  # short chunks picked before memory was short
    print(V.TmPlan(h, l, c, cols, rows, None, jobs, ctx=ctx).info()["chunk"][:2])
hold = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20) - (40 << 20), dtype=torch.uint8, device="cuda")
plan = V.TmPlan(h, l, c, cols, rows, None, jobs, ctx=ctx)
plan.run()
print(plan.info()["chunk"][:2])
"""


@pytest.mark.parametrize("choice", ["timed", "cached"])
def test_plan_on_a_nearly_full_gpu(choice):
    env = {k: v for k, v in os.environ.items() if k != "VTA_TUNE_CACHE"}
    r = subprocess.run([sys.executable, "-c", _CHILD, ROOT, choice], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
