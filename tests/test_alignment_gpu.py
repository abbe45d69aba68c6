"""Device vectors of the caller that start anywhere in a larger allocation: the
kernels' wide accesses must not assume more than the element's own alignment."""
import numpy as np
import pytest

from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 13])  # an even and an odd count of rows
@pytest.mark.parametrize("depth", [0, 3])
def test_anderson_corrections_at_odd_places(ctx, n, depth):
    import torch

    A = P.poisson2d(n, 7)
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    m = A.shape[0]
    b = torch.linspace(0.5, 1.0, m, dtype=torch.float64, device="cuda:0")
    x0 = torch.zeros_like(b)
    out = []
    for at in (0, 1, 2, 3):
        # Forward, one history a row: the same bits on every run.
        dom = capi.Domain(ctx, op, pc, precision=capi.FP64, rng_mode=capi.RNG_COUNTER, seed=4,
                          estimator=capi.EXPECTED_VALUE, direction=capi.FORWARD,
                          sample_ratio=1.0)
        buf = torch.zeros(m + 4, dtype=torch.float64, device="cuda:0")
        delta = buf[at:at + m]
        dom.anderson_begin(b.data_ptr(), x0.data_ptr(), tolerance=0.0, max_iters=6,
                           storage_depth=depth)
        for _ in range(5):
            dom.anderson_correction(delta.data_ptr())
            dom.anderson_apply(delta.data_ptr())
        x = torch.empty_like(b)
        dom.anderson_finish(x.data_ptr())
        assert not buf[:at].any() and not buf[at + m:].any()
        out.append(x.cpu().numpy())
    for x in out[1:]:
        assert np.isfinite(x).all() and np.array_equal(x, out[0])


@pytest.mark.parametrize("dims", [2, 3])
def test_network_outputs_at_odd_places(ctx, dims):
    import torch

    A = P.poisson2d(12, 7) if dims == 2 else P.diffusion3d_varcoef(9, seed=1)[0]
    n = A.shape[0]
    op = capi.Operator(ctx, A)
    net = capi.SpaiNet(ctx, 5 if dims == 2 else 7, seed=3)
    want, m_want = net.infer(op, A.nnz)
    for at in (0, 1, 2, 4, 8):  # floats: aligned to 32, 4, 8, 16 and 32 bytes
        buf = torch.zeros(16 * n + 16, dtype=torch.float32, device="cuda:0")
        mbuf = torch.zeros(A.nnz + 2, dtype=torch.float64, device="cuda:0")
        out, m = buf[at:at + 16 * n], mbuf[at % 2:at % 2 + A.nnz]
        net.infer_dev(op, out.data_ptr(), m.data_ptr())
        assert np.array_equal(out.cpu().numpy().reshape(n, 16), want)
        assert np.array_equal(m.cpu().numpy(), m_want)
        assert not buf[:at].any() and not buf[at + 16 * n:].any()
