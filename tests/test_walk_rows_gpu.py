"""The FP32 walks from global memory, history by history against the host walk:
domains past the limit of the walks from shared memory (200 KB of records)."""
import numpy as np
import pytest
import scipy.sparse as sp

import walk_host
from mcls_b200 import capi

pytestmark = pytest.mark.gpu
L = 10
SETTINGS = [(1, 256, 0), (2, 128, 0), (4, 256, 1), (8, 128, 1)]


def grid_matrix(shape, seed):
    """I plus small entries of both signs at the nearest neighbours of a grid
    (x fastest)."""
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


def domain(ctx, A, setting, **kw):
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP32,
                      estimator=capi.COLLISION, history_length=L, seed=11, **kw)
    dom.set_launch(*setting[:2])
    dom.set_record_cache(setting[2])
    return dom


def check_forward(ctx, A, per, setting, **kw):
    dom = domain(ctx, A, setting, direction=capi.FORWARD, sample_ratio=float(per), **kw)
    n = A.shape[0]
    src = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    x, st = dom.mc_solve(src, internal=True)
    ref, mag, steps = walk_host.forward(dom.export(), src, per, 11, L,
                                        cutoff=kw.get("weight_cutoff", 0.0))
    assert st["histories"] == n * per and st["walk_steps"] == steps
    # A history's compensated FP32 sum is within 2^-22 of its terms' magnitude.
    assert np.all(np.abs(x - ref) <= (2.0 ** -22 + per * 2.0 ** -53) * mag)


def check_adjoint(ctx, A, ratio, setting, **kw):
    dom = domain(ctx, A.T.tocsr(), setting, direction=capi.ADJOINT, sample_ratio=ratio, **kw)
    n = A.shape[0]
    src = np.random.default_rng(2).uniform(-1.0, 1.0, n)
    src[0] = 0.5
    x, st = dom.mc_solve(src, internal=True)
    nh = st["histories"]
    assert abs(nh - int(ratio * n)) <= 1
    at, sign = walk_host.starts(src, nh, 11)
    ref, mag, steps = walk_host.adjoint(dom.export(), at, sign, np.abs(src).sum(), 11, L,
                                        cutoff=kw.get("weight_cutoff", 0.0))
    assert st["walk_steps"] == steps
    # FP64 sums of the same terms in any order (a state gets far fewer than 4096),
    # |b|_1 summed in another order.
    assert np.all(np.abs(x - ref) <= 4096 * 2.0 ** -53 * mag)


@pytest.mark.parametrize("setting", SETTINGS)
@pytest.mark.parametrize("fmt", [capi.RECORD_STENCIL, capi.RECORD_PACKED])
@pytest.mark.parametrize("cutoff", [0.03, 0.3])
def test_histories_ended_by_a_cutoff(ctx, setting, fmt, cutoff):
    A = grid_matrix((21, 19, 23), seed=3)
    check_forward(ctx, A, 2, setting, record_format=fmt, weight_cutoff=cutoff)
    check_adjoint(ctx, A, 1.7, setting, record_format=fmt, weight_cutoff=cutoff)
