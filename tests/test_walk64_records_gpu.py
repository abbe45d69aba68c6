"""FP64 walks over packed records (rows of at most 7 entries) and over the CSR
domain (longer rows) take the transitions that the exported domain gives for
the same random draws, bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi

pytestmark = pytest.mark.gpu


def splitmix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def step(x):
    x = x ^ (x << np.uint64(13))
    x = x ^ (x >> np.uint64(7))
    return x ^ (x << np.uint64(17))


def matrix(n, entries, gen):
    """Rows of 1..entries off-diagonal entries of both signs, row n-1 full."""
    rows, cols, vals = [], [], []
    for i in range(n):
        k = min(entries if i % 5 == 0 else 1 + i % entries, n - 1)
        others = np.delete(np.arange(n), i)
        for j in gen.choice(others, k, replace=False):
            rows.append(i)
            cols.append(j)
            vals.append(gen.choice([-1.0, 1.0]) * gen.uniform(0.05, 0.12))
    return (sp.eye(n) + sp.csr_matrix((vals, (rows, cols)), (n, n))).tocsr()


@pytest.mark.parametrize("entries", [1, 2, 6, 7, 8, 20])
@pytest.mark.parametrize("direction", [capi.ADJOINT, capi.FORWARD])
def test_transitions_are_the_exported_domains(ctx, entries, direction):
    n, L = 333, 9
    gen = np.random.default_rng(entries)
    A = matrix(n, entries, gen)
    if direction == capi.ADJOINT:
        A = A.T.tocsr()  # the walk's matrix has the rows made above
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP64,
                      rng_mode=capi.RNG_COUNTER, seed=4, history_length=L, sample_ratio=2.0,
                      direction=direction, estimator=capi.COLLISION)
    v = gen.uniform(0.5, 1.0, n)
    x, nh, tr = dom.mc_trace(v, 4 * n, internal=True)
    d = dom.export()
    assert dom.info()["max_row_entries"] == entries
    with np.errstate(over="ignore"):
        ekey = splitmix(np.uint64(4) ^ splitmix(np.uint64(0)))
        e = np.arange(nh, dtype=np.uint64)
        u = splitmix(ekey ^ splitmix((np.uint64(2) << np.uint64(56)) ^ e))
    s = tr["states"][:, 0].copy()
    w = np.ones(nh) if direction == capi.FORWARD else np.full(nh, np.abs(v).sum())
    for k in range(L):
        with np.errstate(over="ignore"):
            u = step(u)
        r = np.minimum(u.astype(np.float64) * 2.0 ** -64, 1.0 - 2.0 ** -53)
        nxt = np.empty_like(s)
        for t in range(nh):
            a, b = d["rowptr"][s[t]], d["rowptr"][s[t] + 1]
            j = a + np.searchsorted(d["cdf"][a:b], r[t], side="left")
            w[t] *= d["weights"][s[t]] * (1.0 if d["h"][j] > 0 else -1.0)
            nxt[t] = d["col"][j]
        s = nxt
        assert np.array_equal(tr["states"][:, k + 1], s)
    # The starting weight is a sum in another order; the products are L more
    # roundings on each side.
    np.testing.assert_allclose(tr["final_weight"], w, rtol=2.0 ** -52 * (n + 2 * L))
