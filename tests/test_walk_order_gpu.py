"""The FP32 walks' thread layout: rows in bricks, lanes that share a row,
histories per lane.  The schedule must not change any history."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1
L = 10


def grid_matrix(shape, seed):
    """Diagonally dominant matrix of a grid (x fastest): the nearest
    neighbours along each axis, random weights of both signs."""
    gen = np.random.default_rng(seed)
    n = int(np.prod(shape))
    idx = np.arange(n).reshape(shape[::-1])
    rows, cols = [], []
    for ax in range(len(shape)):
        a = np.moveaxis(idx, ax, 0)
        rows += [a[:-1].ravel(), a[1:].ravel()]
        cols += [a[1:].ravel(), a[:-1].ravel()]
    i, j = np.concatenate(rows), np.concatenate(cols)
    v = gen.uniform(0.05, 0.15, i.size) * gen.choice([-1.0, 1.0], i.size)
    return sp.csr_matrix(sp.eye(n) + sp.csr_matrix((v, (i, j)), shape=(n, n)))


def splitmix(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def xorshift(x):
    x ^= (x << 13) & M64
    x ^= x >> 7
    return x ^ ((x << 17) & M64)


def walk_reference(d, src, per, seed):
    """Collision estimate of every row by its histories, one at a time, and the
    sum of the terms' magnitudes (64-bit sums of the 32-bit weights' terms)."""
    n = src.size
    ekey = splitmix(seed ^ splitmix(0))
    c = src.astype(np.float32)
    W = d["weights"].astype(np.float32)
    cdf = d["cdf"].astype(np.float32)
    x, mag = np.zeros(n), np.zeros(n)
    for e in range(n * per):
        s, w = e // per, np.float32(1.0)
        r = splitmix(ekey ^ splitmix((2 << 56) ^ e)) or 0x9E3779B97F4A7C15
        for _ in range(L):
            x[e // per] += float(w) * float(c[s])
            mag[e // per] += abs(float(w) * float(c[s]))
            r = xorshift(r)
            u = np.float32(r >> 40) * np.float32(2.0 ** -24)
            a, b = d["rowptr"][s], d["rowptr"][s + 1]
            k = a + int(np.searchsorted(cdf[a:b], u, side="left"))
            w = np.float32(w * W[s])
            if not d["h"][k] > 0:
                w = -w
            s = int(d["col"][k])
    return x / per, mag / per


@pytest.mark.parametrize("shape", [(1,), (2,), (31,), (4, 2), (7, 5), (33, 9), (5, 3, 2), (4, 4, 4),
                                   (9, 5, 3), (2, 2, 3)])
@pytest.mark.parametrize("per", [1, 2, 3, 4, 6])
def test_forward_rows_match_the_histories(ctx, shape, per):
    n = int(np.prod(shape))
    A = grid_matrix(shape, seed=n) if n > 1 else sp.csr_matrix(np.array([[0.7]]))
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP32,
                      direction=capi.FORWARD, estimator=capi.COLLISION, sample_ratio=float(per),
                      history_length=L, seed=11)
    src = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    x, st = dom.mc_solve(src, internal=True)
    ref, mag = walk_reference(dom.export(), src, per, 11)
    assert st["histories"] == n * per and st["walk_steps"] == n * per * L
    # A history's compensated FP32 sum is within 2^-22 of its terms' magnitude.
    assert np.all(np.abs(x - ref) <= 2.0 ** -22 * mag)


@pytest.mark.parametrize("ratio", [0.3, 1.0, 2.7])
@pytest.mark.parametrize("fmt", [capi.RECORD_STENCIL, capi.RECORD_PACKED])
def test_adjoint_launch_shapes_agree(ctx, ratio, fmt):
    A = grid_matrix((9, 7, 5), seed=3)
    op = capi.Operator(ctx, A)
    src = np.random.default_rng(2).uniform(-1.0, 1.0, A.shape[0])
    xs = []
    for hpl, blk, l1 in ((1, 256, 0), (2, 128, 0), (4, 256, 1), (8, 128, 0)):
        dom = capi.Domain(ctx, op, None, precision=capi.FP32, sample_ratio=ratio, seed=5,
                          history_length=L, record_format=fmt)
        dom.set_launch(hpl, blk)
        dom.set_record_cache(l1)
        x, st = dom.mc_solve(src, internal=True)
        assert st["walk_steps"] == st["histories"] * L
        xs.append(x)
    # FP64 sums of the same terms in another order.
    for x in xs[1:]:
        assert np.allclose(x, xs[0], rtol=0, atol=1e-13 * np.abs(xs[0]).max())
