"""Result arrays (vta_device_array): freed blocks are reused for later results
only after the device's work on them, at most 256 MiB of them are kept, and
all go back with the last context; several threads may allocate and free."""
import gc
import threading

import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def test_reuse_keeps_values_apart():
    import torch

    x = datagen.random_walk(5000, seed=3, nan_lead=2).astype(np.float32)
    sma = V.CudaSma(0)
    want = sma.batch_dev(x, sweep={"period": (2, 60, 1)}).to_host()
    for i in range(12):
        a = sma.batch_dev(x, sweep={"period": (2, 60, 1)})
        t = torch.as_tensor(a, device="cuda")
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):  # work on another stream, still queued when the array is freed
            acc = torch.zeros_like(t)
            for _ in range(20):
                acc += t
        del t
        a.free()
        b = sma.batch_dev(x * 3, sweep={"period": (2, 60, 1)})  # takes the block over
        side.synchronize()
        assert np.allclose(acc.cpu().numpy(), 20 * want, rtol=1e-5, equal_nan=True)
        assert np.allclose(b.to_host(), 3 * want, rtol=1e-5, equal_nan=True)


def test_threads():
    x = datagen.random_walk(3000, seed=4).astype(np.float32)
    want = V.CudaEma(0).batch_dev(x, sweep={"period": (3, 40, 1)}).to_host()
    bad = []

    def work():
        ema = V.CudaEma(0)
        for _ in range(30):
            r = ema.batch_dev(x, sweep={"period": (3, 40, 1)})
            if not np.array_equal(r.to_host(), want, equal_nan=True):
                bad.append(1)
            r.free()

    ts = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_idle_blocks_are_bounded():
    import torch

    x = datagen.random_walk(100_000, seed=5).astype(np.float32)
    sma = V.CudaSma(0)
    gc.collect()
    free0 = torch.cuda.mem_get_info()[0]
    arrays = [sma.batch_dev(x, sweep={"period": (2, 201, 1)}) for _ in range(8)]  # 80 MB each
    for a in arrays:
        a.free()
    assert free0 - torch.cuda.mem_get_info()[0] <= (256 << 20) + (64 << 20)
