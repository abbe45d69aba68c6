"""The residual norm and the loop's end, from one cluster (small stencil systems)
and from a grid of blocks: the reported norm is that of b - A x, at sizes around
the cluster's threads and the largest it takes."""
import numpy as np
import pytest

from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [3, 31, 32, 90, 91, 110, 111])  # 110^2 <= 12288 < 111^2
@pytest.mark.parametrize("direction", [capi.FORWARD, capi.ADJOINT])
@pytest.mark.parametrize("jacobi", [False, True])
def test_norm_of_the_returned_iterate(ctx, size, direction, jacobi):
    A = P.poisson2d(size)
    A = A / A.diagonal().max()  # H = I - A without a preconditioner
    b = np.random.default_rng(size).uniform(0.5, 1.0, A.shape[0])
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI) if jacobi else None
    dom = capi.Domain(ctx, op, pc, precision=capi.FP32, rng_mode=capi.RNG_COUNTER, seed=1,
                      direction=direction, estimator=capi.COLLISION, sample_ratio=1.0)
    x, st = dom.mcsa_solve(b, tolerance=0.0, max_iters=7)
    assert st["iterations"] == 7 and st["histories"] > 0
    r = b - A @ x
    if jacobi:
        r = r / A.diagonal()
    # Five products a row and a sum of n squares in any order.
    n = A.shape[0]
    scale = np.linalg.norm(np.abs(b) + abs(A) @ np.abs(x))
    assert abs(st["residual_norm"] - np.linalg.norm(r)) <= 2.0 ** -53 * (
        16 * scale / A.diagonal().min() + n * np.linalg.norm(r))
