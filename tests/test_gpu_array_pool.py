"""Result arrays and the library's pool of freed blocks: freeing one twice."""
import ctypes as C

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
