"""A pipeline wait that ran out, reported after the call returned: the test
sets the context's error word (as the kernel would) through the internal
header; the report comes once, from synchronize or from the next call, which
does not run, and names the sweep."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def set_error(tmp_path):
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    src, so = tmp_path / "err.cpp", tmp_path / "err.so"
    src.write_text('#include "vta_internal.h"\n'
                   'extern "C" void set_error(vta_ctx* c) { *static_cast<volatile int*>(c->err_host) = 1; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "vectorta_gb300", "csrc"),
                    "-I", os.path.join(cuda, "include"), str(src), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).set_error
    fn.argtypes = [C.c_void_p]
    return fn


def test_reported_once(set_error):
    import torch

    x = torch.from_numpy(datagen.random_walk(4000, seed=5).astype(np.float32)).cuda()
    ctx = V.Context(0)
    wma, sma = V.CudaWma(ctx=ctx), V.CudaSma(ctx=ctx)
    out = torch.zeros(5, 4000, device="cuda")
    torch.cuda.synchronize()
    wma.batch_device([x], 4000, 0, {"period": (10, 14, 1)}, [out])
    ctx.synchronize()

    set_error(ctx.handle)
    with pytest.raises(V.VtaError, match=r"wma, 5 rows of 4000 bars\)$") as e:
        ctx.synchronize()
    assert e.value.kind == "Cuda"
    ctx.synchronize()

    set_error(ctx.handle)
    out.zero_()
    torch.cuda.synchronize()
    with pytest.raises(V.VtaError, match="wma, 5 rows of 4000 bars.*did not run"):
        sma.batch_device([x], 4000, 0, {"period": (10, 14, 1)}, [out])
    ctx.synchronize()
    assert not out.any()
    sma.batch_device([x], 4000, 0, {"period": (10, 14, 1)}, [out])
    ctx.synchronize()
    assert out.nan_to_num(1.0).any()
