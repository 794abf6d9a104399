"""Result arrays and the library's pool of freed blocks: freeing one twice, and
freeing one after the last context (in a process of its own: other tests'
contexts would keep the pool), and beside another thread's stream capture."""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from vectorta_gb300 import _native as N
from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def test_second_free_is_refused():
    x = datagen.random_walk(3000, seed=4).astype(np.float32)
    sma = V.CudaSma(0)
    want = sma.batch_dev(x, sweep={"period": (2, 60, 1)}).to_host()
    a = sma.batch_dev(x, sweep={"period": (2, 60, 1)})
    again = N.DeviceArrayC(a._c.ptr, a._c.rows, a._c.cols, a._c.device)
    a.free()
    assert N.lib().vta_device_array_free(C.byref(again)) == 1  # Cuda
    b, c = (sma.batch_dev(x, sweep={"period": (2, 60, 1)}) for _ in range(2))
    assert b.ptr != c.ptr
    for r in (b, c):
        assert np.array_equal(r.to_host(), want, equal_nan=True)


_CHILD = """
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch
from vectorta_gb300 import _native as N
from vectorta_gb300 import cuda as V

torch.zeros(1, device="cuda")
x = np.linspace(1, 2, 100_000, dtype=np.float32)

def last_array():
    sma = V.CudaSma(0)
    a = sma.batch_dev(x, sweep={"period": (2, 201, 1)})  # 80 MB
    c = N.DeviceArrayC(a._c.ptr, a._c.rows, a._c.cols, a._c.device)
    a._c.ptr = None  # c owns the block now
    sma.ctx.close()
    return c

c = last_array()  # (the first call's module load is not the pool's)
N.lib().vta_device_array_free(C.byref(c))
free0 = torch.cuda.mem_get_info()[0]
for _ in range(3):
    c = last_array()
    assert N.lib().vta_device_array_free(C.byref(c)) == 0
assert free0 - torch.cuda.mem_get_info()[0] < 16 << 20, (free0, torch.cuda.mem_get_info()[0])
held = torch.cuda.mem_get_info()[0]
c = last_array()
assert held - torch.cuda.mem_get_info()[0] >= 64 << 20  # it was in use
assert N.lib().vta_device_array_free(C.byref(c)) == 0
assert held - torch.cuda.mem_get_info()[0] < 16 << 20
print("ok")
"""


def test_no_block_outlives_the_last_context():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _CHILD, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_free_beside_another_threads_capture():
    import torch

    x = datagen.random_walk(3000, seed=4).astype(np.float32)
    sma = V.CudaSma(0)
    a = sma.batch_dev(x, sweep={"period": (2, 60, 1)})
    y = torch.ones(1000, device="cuda")
    ready, done = threading.Event(), threading.Event()

    def free():
        ready.wait()
        a.free()
        done.set()

    t = threading.Thread(target=free)
    t.start()
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g, capture_error_mode="thread_local"):
            z = y * 2
            ready.set()
            done.wait(30)
            z = z + 1
    finally:
        ready.set()
        t.join()
    g.replay()
    torch.cuda.synchronize()
    assert torch.all(z == 3)
