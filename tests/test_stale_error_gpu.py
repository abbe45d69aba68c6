"""An error that the program left in the CUDA runtime (here a rejected device
ordinal) belongs to no call of the library."""
import ctypes

import numpy as np
import pytest

from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["mc", "mcsa", "mcsa_host_loop", "anderson", "apply", "precond",
                                  "batch", "agreement", "infer"])
def test_calls_after_a_stale_error(ctx, call):
    A = P.poisson2d(16)
    b = np.ones(A.shape[0])
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    dom = capi.Domain(ctx, op, pc, precision=capi.FP32, direction=capi.FORWARD,
                      estimator=capi.COLLISION, sample_ratio=1.0)
    net = capi.SpaiNet(ctx, 5, seed=0)
    calls = {
        "mc": lambda: dom.mc_solve(b),
        "mcsa": lambda: dom.mcsa_solve(b, tolerance=0.0, max_iters=2),
        "mcsa_host_loop": lambda: dom.mcsa_solve(b, tolerance=0.0, max_iters=2, host_loop=1),
        "anderson": lambda: dom.anderson_solve(b, tolerance=0.0, max_iters=2),
        "apply": lambda: op.apply(b),
        "precond": lambda: capi.Precond(ctx, op, capi.PREC_POINT_JACOBI).close(),
        "batch": lambda: capi.Batch(ctx, [A], [1], direction=capi.FORWARD,
                                    precision=capi.FP32).close(),
        "agreement": lambda: dom.walk_agreement(100),
        "infer": lambda: net.infer(op, A.nnz),
    }
    runtime = ctypes.CDLL("libcudart.so.12")
    assert runtime.cudaSetDevice(1000) != 0 and runtime.cudaPeekAtLastError() != 0
    try:
        calls[call]()
    finally:
        runtime.cudaGetLastError()
