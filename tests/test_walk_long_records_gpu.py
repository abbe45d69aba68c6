"""Packed records of more than 64 bytes: a step reads the first 7 entries and
the others only when the draw lies past them.  The same histories as the
stencil records of the same matrix (read whole), in every walk kernel."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi

pytestmark = pytest.mark.gpu


def banded(n, offsets, seed, short):
    """I minus small entries at the offsets; every third row keeps only the
    first `short` of them."""
    gen = np.random.default_rng(seed)
    rows, cols, vals = [], [], []
    for i in range(n):
        k = offsets[:short] if i % 3 == 0 else offsets
        for o in k:
            if 0 <= i + o < n and o:
                rows.append(i)
                cols.append(i + o)
                vals.append(gen.choice([-1.0, 1.0]) * gen.uniform(0.2, 1.0) * 0.6 / len(offsets))
    return (sp.eye(n) * 1.05 + sp.csr_matrix((vals, (rows, cols)), (n, n))).tocsr()


# 8 entries (one past the first half) up to 30, the most of the widest stencil
# record; the packed strides are 12, 16, 24 and 32 slots.
@pytest.mark.parametrize("entries", [8, 11, 12, 15, 16, 23, 24, 30])
@pytest.mark.parametrize("direction", [capi.FORWARD, capi.ADJOINT])
@pytest.mark.parametrize("cutoff", [0.0, 1e-3])
def test_packed_walks_like_stencil(ctx, entries, direction, cutoff):
    n = 700
    half = entries // 2
    offsets = [o * 3 for o in range(-half, entries - half)]
    A = banded(n, offsets, entries, short=min(5, entries))
    if direction == capi.ADJOINT:
        A = A.T.tocsr()
    b = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    xs = []
    for fmt in (capi.RECORD_PACKED, capi.RECORD_STENCIL):
        dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP32,
                          rng_mode=capi.RNG_COUNTER, seed=3, history_length=8, sample_ratio=3.0,
                          direction=direction, estimator=capi.COLLISION, record_format=fmt,
                          weight_cutoff=cutoff)
        assert dom.info()["max_row_entries"] == entries
        x, st = dom.mc_solve(b)
        xs.append((x, st["histories"], st["walk_steps"]))
    assert xs[0][1:] == xs[1][1:]
    if direction == capi.FORWARD and cutoff == 0.0:
        assert np.array_equal(xs[0][0], xs[1][0])
    else:
        # FP64 sums of the same terms in the order the histories arrive: at
        # most a few thousand terms a state, each within |b|_1.
        np.testing.assert_allclose(xs[0][0], xs[1][0], rtol=0,
                                   atol=2.0 ** -53 * 4096 * np.abs(b).sum())
