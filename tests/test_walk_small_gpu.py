"""Walks of a domain whose records fit a block's shared memory, on both sides of
that limit: the transitions do not depend on where the records are read."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi

pytestmark = pytest.mark.gpu


def ring(n, seed):
    """I minus small entries at six offsets (a matrix of rings, so that row i of
    a longer one is row i of a shorter one away from its ends)."""
    gen = np.random.default_rng(seed)
    d = {o: gen.uniform(0.02, 0.12, 20000)[:n] for o in (-7, -2, -1, 1, 3, 8)}
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [np.ones(n)]
    for o, v in d.items():
        i = np.arange(n)
        keep = (i + o >= 0) & (i + o < n)
        rows.append(i[keep])
        cols.append(i[keep] + o)
        vals.append(-v[keep])
    return sp.csr_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))),
                         (n, n))


# 200 KB hold 6400 records of 32 bytes, 3200 of 64 and 2133 of 96: sizes next to
# the limits, one row, one block and its remainder; histories of one step.
@pytest.mark.parametrize("n", [1, 2, 127, 129, 2133, 2134, 3200, 3201, 6400, 6401])
@pytest.mark.parametrize("fmt", [capi.RECORD_PACKED, capi.RECORD_STENCIL])
@pytest.mark.parametrize("length", [1, 10])
def test_rows_do_not_depend_on_the_size(ctx, n, fmt, length):
    if n <= 2 and fmt == capi.RECORD_STENCIL:
        pytest.skip("no six offsets")
    gen = np.random.default_rng(5)
    big = 12000  # past every limit
    v = gen.uniform(-1.0, 1.0, big)
    out = []
    for m in (n, big):
        A = ring(m, 3) if m > 8 else sp.csr_matrix(0.7 * sp.eye(m))
        dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP32,
                          rng_mode=capi.RNG_COUNTER, seed=2, history_length=length,
                          sample_ratio=1.0, direction=capi.FORWARD, estimator=capi.COLLISION,
                          record_format=fmt)
        x, st = dom.mc_solve(v[:m])
        assert st["histories"] == m and st["walk_steps"] == m * length
        out.append(x)
    if n <= 2:
        # H = 0.3 I: the sum of 0.3^k, each history staying at its state.
        want = v[:n] * sum(0.3 ** k for k in range(length))
        np.testing.assert_allclose(out[0], want, rtol=2.0 ** -22 * (length + 2))
    else:
        # A row farther from the end than ten steps of 8 rows reach.
        k = n - 8 * length
        assert k > 0 and np.array_equal(out[0][:k], out[1][:k])


@pytest.mark.parametrize("n", [1, 129, 6400, 6401])
def test_adjoint_tallies(ctx, n):
    """x is the tallies' mean: |x|'s signed sum over one step's histories is the
    sum of the weights, whatever the records are read from."""
    A = ring(n, 3) if n > 8 else sp.csr_matrix(0.7 * sp.eye(n))
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP32,
                      rng_mode=capi.RNG_COUNTER, seed=2, history_length=6, sample_ratio=2.0,
                      direction=capi.ADJOINT, estimator=capi.COLLISION)
    ref = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP64,
                      rng_mode=capi.RNG_COUNTER, seed=2, history_length=6, sample_ratio=2.0,
                      direction=capi.ADJOINT, estimator=capi.COLLISION)
    v = np.random.default_rng(6).uniform(0.5, 1.0, n)
    x, st = dom.mc_solve(v)
    y, rt = ref.mc_solve(v)
    assert st["histories"] == rt["histories"] and st["walk_steps"] == rt["walk_steps"]
    # FP32 weights (a few roundings a step) and 24-bit draws, which choose
    # another entry where the 53-bit draw lies within 2^-23 of a CDF value: over
    # 6 * 12800 steps of 6 entries fewer than a handful of histories.
    scale = np.abs(v).sum() / st["histories"]
    assert np.sum(np.abs(x - y) > 1e-5 * np.abs(y) + 1e-6 * scale) <= 12 * 6
