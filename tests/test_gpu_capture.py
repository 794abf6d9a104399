"""Weighted-window sweeps are refused inside a stream capture (a replay would
read operands that later calls have replaced); the context works on."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu


def test_weighted_windows_are_not_captured():
    import torch

    x = torch.from_numpy(datagen.random_walk(4000, seed=5).astype(np.float32)).cuda()
    st = torch.cuda.Stream()
    ctx = V.Context(0)
    ctx.set_stream(st.cuda_stream)
    alma = V.CudaAlma(ctx=ctx)
    sweep = {"period": (9, 40, 1), "offset": (0.85, 0.85, 0.0), "sigma": (6.0, 6.0, 0.0)}
    want, got = (torch.full((32, 4000), -1.0, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    alma.batch_device([x], 4000, 0, sweep, [want])  # its constants are on the device now
    ctx.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        with pytest.raises(V.VtaError):
            alma.batch_device([x], 4000, 0, sweep, [got])
        got.fill_(0.0)
    alma.batch_device([x], 4000, 0, sweep, [got])
    ctx.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
