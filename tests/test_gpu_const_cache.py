"""Sweeps whose period list repeats while another parameter changes on every
call, until the context's constant cache has been filled and started over:
each result around that is the one of a context that never filled its cache."""
import numpy as np
import pytest

from vectorta_gb300 import cuda as V
from vectorta_gb300 import datagen

pytestmark = pytest.mark.gpu

# bars, sweep of call i, calls that fill 4 MiB (20,480, 10,240, 40,960 and 2,048
# new bytes each)
CASES = {
    "alma": (3000, lambda i: {"period": (5, 2564, 1), "offset": (0.3 + 0.001 * i, 0.3 + 0.001 * i, 0.0),
                              "sigma": (6.0, 6.0, 0.0)}, 205),
    "bollinger_bands": (3000, lambda i: {"period": (5, 2564, 1), "devup": (1 + 0.01 * i, 1 + 0.01 * i, 0.0),
                                         "devdn": (2.0, 2.0, 0.0)}, 410),
    # the growing walk's item list, and the sliding walk's fractions
    "percentile_nearest_rank": (3000, lambda i: {"length": (5, 2564, 1), "percentage": (1 + 0.1 * i, 1 + 0.1 * i, 0.0)},
                                103),
    "percentile_nearest_rank slide": (4000, lambda i: {"length": (5, 3837, 8),
                                                       "percentage": (1 + 0.04 * i, 1 + 0.04 * i, 0.0)}, 2050),
}


@pytest.mark.parametrize("case", CASES)
def test_full_cache_changes_no_result(case):
    import torch

    name = case.split()[0]
    bars, sweep, fills = CASES[case]
    x = torch.from_numpy(datagen.random_walk(bars, seed=9).astype(np.float32)).cuda()
    ctx = V.Context(0)
    ind = V.CLASSES[name](ctx=ctx)
    rows = len(ind.expand_grid(sweep(0)))
    n_out = 3 if name == "bollinger_bands" else 1
    outs = [torch.empty(rows, bars, device="cuda") for _ in range(n_out)]
    want = [torch.empty_like(o) for o in outs]
    torch.cuda.synchronize()
    for i in range(fills + 6):
        ind.batch_device([x], bars, 0, sweep(i), outs)
        if i < 2 or i > fills - 12:
            ctx.synchronize()
            other = V.Context(0)
            V.CLASSES[name](ctx=other).batch_device([x], bars, 0, sweep(i), want)
            other.synchronize()
            for a, b in zip(outs, want):
                assert torch.equal(a.view(torch.int32), b.view(torch.int32)), i
    if "slide" in case:
        assert ind.last_kernel == "percentile_ranks_slide"
