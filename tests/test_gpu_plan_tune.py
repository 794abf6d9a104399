"""A mixed plan's chunk lengths, timed at creation, are kept in the tuning cache
file like those of single jobs: a new process with the file times nothing and
takes the same ones."""
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
cols, rows = 600, 6000
g = torch.Generator(device="cuda").manual_seed(1)
c = torch.cumsum(torch.randn(rows, cols, device="cuda", generator=g), 0) * 0.01 + 100
h, l = c + 0.5, c - 0.5
outs = [torch.empty_like(c) for _ in range(3)]
jobs = [{"kind": k, "period": p, "param": a, "out0": o} for (k, p, a), o in
        zip((("atr", 14, 0.0), ("adx", 14, 0.0), ("percentile_nearest_rank", 30, 50.0)), outs)]
torch.cuda.synchronize()
for _ in range(2):
    i = V.TmPlan(h, l, c, cols, rows, None, jobs).info()
    print(i["n_items"] > 4 * 152, i["tuned"], *i["chunk"][:3])
"""


def test_mix_choice_persists(tmp_path):
    env = dict(os.environ, VTA_TUNE_CACHE=str(tmp_path / "tune.txt"))
    outs = []
    for _ in range(2):
        r = subprocess.run([sys.executable, "-c", _CHILD, ROOT], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        outs += [ln.split() for ln in r.stdout.strip().splitlines()]
    assert [o[0] for o in outs] == ["True"] * 4
    assert [o[1] for o in outs] == ["True", "False", "False", "False"]
    assert outs[0][2:] == outs[1][2:] == outs[2][2:] == outs[3][2:]
    assert len((tmp_path / "tune.txt.mixes").read_text().splitlines()) == 1
    assert len((tmp_path / "tune.txt").read_text().splitlines()) == 3
