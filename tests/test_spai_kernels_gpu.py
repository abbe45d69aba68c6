"""Learned-SPAI kernels at the edges: tile remainders, slot counts with and
without an unrolled kernel, rows that miss pattern entries, vector counts
around the loss kernel's groups."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi
from mcls_b200 import problems as P
from mcls_b200 import spai
from oracle import spai_oracle as so

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed):
    """Diagonally dominant matrix on the given offsets, some entries absent."""
    gen = np.random.default_rng(seed)
    A = sp.lil_matrix((n, n))
    for i in range(n):
        for o in offsets:
            if o != 0 and 0 <= i + o < n and gen.uniform() > 0.1:
                A[i, i + o] = -gen.uniform(0.2, 1.0)
        A[i, i] = len(offsets) + gen.uniform()
    A = sp.csr_matrix(A)
    A.sort_indices()
    return A


@pytest.mark.parametrize("n", [1, 127, 128, 129, 900])
@pytest.mark.parametrize("offsets", [(-1, 0, 1), (-7, -1, 0, 1, 7), (-20, -7, -1, 0, 1, 7),
                                     (-50, -7, -1, 0, 1, 7, 50),
                                     (-60, -50, -7, -1, 0, 1, 7, 50, 60)])
def test_forward_and_gradient_at_the_edges(ctx, n, offsets):
    import torch

    A = banded(n, offsets, seed=n + len(offsets))
    k = spai.stencil_slots(A)
    if k < 3:
        pytest.skip("fewer than three offsets present")
    op = capi.Operator(ctx, A)
    if not op_has_dia(ctx, op):
        pytest.skip("not stored by diagonals")
    net = capi.SpaiNet(ctx, k, seed=1)
    p = so.init_params(3, zero_last=False)
    net.params = p
    out, m = net.infer(op, A.nnz)
    ref, _ = so.forward(p, so.features(A))
    # The forward bounds of test_spai_gpu (BF16 activations).
    np.testing.assert_allclose(out[:, :k], ref[:, :k], rtol=2e-2,
                               atol=2e-3 * np.abs(ref[:, :k]).max())
    np.testing.assert_allclose(m, so.mvalues(A, out), rtol=1e-12, atol=0)
    # An output array aligned to 16 bytes only.
    raw = torch.zeros(n * 16 + 4, dtype=torch.float32, device="cuda:0")
    net.infer_dev(op, raw[4:].data_ptr(), None)
    assert np.array_equal(raw[4:].cpu().numpy().reshape(n, 16), out)
    for nvec in (1, 8, 9):
        V = np.random.default_rng(nvec).standard_normal((nvec, n))
        Vt = torch.tensor(V, device="cuda:0").contiguous()
        loss, g = net.gradient(op, Vt.data_ptr(), nvec)
        loss_o, g_o = so.loss_and_gradient(p, A, V, rounded=True)
        np.testing.assert_allclose(loss, loss_o, rtol=5e-3)
        # A BF16 activation that rounds the other way moves single rows; few
        # rows average little, so the whole gradient is compared.
        assert np.linalg.norm(g - g_o) <= 3e-2 * np.linalg.norm(g_o)


def op_has_dia(ctx, op):
    dom = capi.Domain(ctx, op, None, precision=capi.FP64)
    try:
        return dom.info()["operator_dia"] > 0
    finally:
        dom.close()
