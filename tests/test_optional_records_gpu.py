"""Walk data that a domain can do without (FP64 records, the row order) must not
cost a domain that fits memory without them: it is built, and walks the same."""
import numpy as np
import pytest

from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu


def build(ctx, op):
    return capi.Domain(ctx, op, None, precision=capi.FP64, rng_mode=capi.RNG_COUNTER, seed=4,
                       direction=capi.FORWARD, estimator=capi.COLLISION, sample_ratio=1.0,
                       history_length=4)


def test_fp64_domain_in_scarce_memory(ctx):
    import torch

    A = P.poisson2d(1400)
    n = A.shape[0]
    A = A * (1.0 / A.diagonal()[0])
    op = capi.Operator(ctx, A)
    b = torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda:0")
    x = torch.empty_like(b)
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    dom = build(ctx, op)
    free1 = torch.cuda.mem_get_info()[0]
    st = dom.mc_solve_dev(b.data_ptr(), x.data_ptr())
    want, steps = x.cpu().numpy(), st["walk_steps"]
    dom.close()
    # Everything but half of the 96-byte records.
    room = (free0 - free1) - 48 * n
    assert room > 0
    hog, left = [], torch.cuda.mem_get_info()[0] - room
    while left > 1 << 21:
        size = min(left, 16 << 30) >> 21 << 21
        hog.append(torch.empty(size, dtype=torch.uint8, device="cuda:0"))
        left = torch.cuda.mem_get_info()[0] - room
    try:
        dom = build(ctx, op)
    finally:
        del hog
        torch.cuda.empty_cache()
    x.zero_()
    st = dom.mc_solve_dev(b.data_ptr(), x.data_ptr())
    assert st["walk_steps"] == steps and np.array_equal(x.cpu().numpy(), want)
    dom.close()
