"""The learned preconditioner's residual in one pass over blocks with a halo:
bit for bit the general path's, at sizes around the blocks' rows, where the
number of rows per block changes and where two passes take over."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi, spai
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu


# Rows: 256, 1024, 1089 (blocks of 256), 160^2 = 25600 (of 512), 320^2 = 102400
# (of 1024), 393^2 = 154449 (more than a wave on 148 SMs).
@pytest.mark.parametrize("size", [16, 32, 33, 159, 160, 161, 320, 393])
@pytest.mark.parametrize("direction", [capi.FORWARD, capi.ADJOINT])
def test_learned_iteration_matches_the_general_path(ctx, size, direction):
    import torch

    # Shifted, so that the network is a good enough inverse at every size.
    A = P.anisotropic2d(size, 3.0, 0.4)
    A = (A + sp.diags(A.diagonal())).tocsr()
    b = np.random.default_rng(2).uniform(-1.0, 1.0, size * size)
    op = capi.Operator(ctx, A)
    net = capi.SpaiNet(ctx, spai.stencil_slots(A), seed=1)
    V = torch.randn((6, A.shape[0]), dtype=torch.float64, device="cuda:0")
    spai.train(net, [(op, V)], steps=150, lr=3e-3)
    pl = capi.Precond(ctx, op, capi.PREC_LEARNED_SPAI, net=net)
    M = pl.to_scipy(A.shape[0])
    assert M.nnz == A.nnz  # kept on A's pattern, not the Jacobi fallback
    pu = capi.Precond(ctx, op, capi.PREC_USER_CSR, user=M)
    kw = dict(precision=capi.FP32, rng_mode=capi.RNG_COUNTER, seed=11, direction=direction,
              estimator=capi.COLLISION, sample_ratio=1.0)
    its = 4 if direction == capi.FORWARD else 1
    x, s = zip(*(capi.Domain(ctx, op, p, **kw).mcsa_solve(b, tolerance=0.0, max_iters=its)
                 for p in (pl, pu)))
    assert s[0]["iterations"] == s[1]["iterations"] == its
    if direction == capi.FORWARD:
        assert np.array_equal(x[0], x[1])
    else:  # FP64 tallies in the order the histories arrive
        np.testing.assert_allclose(x[0], x[1], rtol=1e-11, atol=1e-11 * np.abs(x[1]).max())
    # n squares in any order.
    assert abs(s[0]["residual_norm"] - s[1]["residual_norm"]) <= \
        2.0 ** -53 * A.shape[0] * s[1]["residual_norm"] + 1e-10 * s[1]["residual_norm"] * (
            direction == capi.ADJOINT)
