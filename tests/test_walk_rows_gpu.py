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


def positive(A):
    """The same pattern with H = I - A without a negative entry."""
    D = sp.diags(A.diagonal())
    return sp.csr_matrix(D - abs(A - D))


# Just past 6,400 rows of 32 bytes, with remainders of the 4 x 4 x 2 bricks (4 x 8
# in two dimensions, fewer lines with more lanes a row) along every axis; one that
# divides evenly; grids thinner than a brick; a chain (no grid behind it).
@pytest.mark.parametrize("shape", [(83, 79), (80, 88), (19, 18, 20), (16, 16, 26), (33, 7, 31),
                                   (5, 3, 450), (2, 2, 1700), (3, 2300), (6901,)])
@pytest.mark.parametrize("per", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("fmt,signs", [(capi.RECORD_STENCIL, 1), (capi.RECORD_STENCIL, 0),
                                       (capi.RECORD_PACKED, 1)])
def test_rows_in_bricks(ctx, shape, per, fmt, signs):
    A = grid_matrix(shape, seed=int(np.prod(shape)))
    check_forward(ctx, A if signs else positive(A), per, SETTINGS[per % 4], record_format=fmt)


@pytest.mark.parametrize("setting", SETTINGS)
@pytest.mark.parametrize("ratio", [0.3, 1.0, 2.7])
@pytest.mark.parametrize("fmt,signs", [(capi.RECORD_STENCIL, 1), (capi.RECORD_STENCIL, 0),
                                       (capi.RECORD_PACKED, 1)])
def test_adjoint_histories(ctx, setting, ratio, fmt, signs):
    A = grid_matrix((21, 19, 23), seed=3)
    check_adjoint(ctx, A if signs else positive(A), ratio, setting, record_format=fmt)


def banded(n, entries, seed):
    """I plus up to `entries` entries a row at even offsets; every third row
    keeps five of them."""
    gen = np.random.default_rng(seed)
    off = np.arange(entries) - entries // 2
    off = np.where(off >= 0, off + 1, off) * 2
    i, j = np.repeat(np.arange(n), off.size), np.arange(n)[:, None] + off
    j = j.ravel()
    keep = (j >= 0) & (j < n) & ((i % 3 > 0) | (np.tile(np.arange(off.size), n) < 5))
    v = gen.uniform(0.2, 1.0, i.size) * gen.choice([-1.0, 1.0], i.size) * 0.8 / entries
    # The last rows have few neighbours above them: one each, whatever is left.
    return sp.csr_matrix(sp.eye(n) + sp.csr_matrix((v[keep], (i[keep], j[keep])), shape=(n, n))
                         + sp.diags([0.05], [-1], shape=(n, n))
                         + sp.diags([0.05], [n - 1], shape=(n, n)))


# Packed strides of 8, 12, 16, 24 and 32 slots, read in two parts from 12 on, and
# stencil records of 64 and 128 bytes; every one past 200 KB.
@pytest.mark.parametrize("entries", [5, 7, 9, 10, 13, 14, 21, 22, 28])
@pytest.mark.parametrize("setting", [SETTINGS[0], SETTINGS[1], SETTINGS[3]])
@pytest.mark.parametrize("cutoff", [0.0, 0.01])
@pytest.mark.parametrize("fmt", [capi.RECORD_PACKED, capi.RECORD_STENCIL])
def test_records_of_every_length(ctx, entries, setting, cutoff, fmt):
    A = banded(3300, entries, entries)
    kw = dict(record_format=fmt, weight_cutoff=cutoff)
    check_forward(ctx, A, 2, setting, **kw)
    check_adjoint(ctx, A.T.tocsr(), 1.5, setting, **kw)  # the rows walked are A's


@pytest.mark.parametrize("shape", [(2,), (11, 9, 13), (79, 81)])
@pytest.mark.parametrize("ratio", [0.5, 2.0])
@pytest.mark.parametrize("fmt", [capi.RECORD_STENCIL, capi.RECORD_PACKED])
def test_adjoint_histories_from_shared_memory(ctx, shape, ratio, fmt):
    check_adjoint(ctx, grid_matrix(shape, seed=3), ratio, SETTINGS[0], record_format=fmt)


def test_stencil16_rows_do_not_depend_on_the_size(ctx):
    """16-bit thresholds have no host walk here: the rows that no end of the grid
    reaches are those of a domain that walks from shared memory."""
    out = []
    for ny in (40, 400):  # 2,400 and 24,000 rows
        A = positive(grid_matrix((60, ny), seed=1))
        A.data[:] = np.where(A.data > 0, 1.0, -0.2)  # the same row everywhere
        src = np.zeros(A.shape[0])
        src[:60 * 40] = np.random.default_rng(5).uniform(0.1, 1.0, 60 * 40)
        dom = domain(ctx, A, SETTINGS[0], direction=capi.FORWARD, sample_ratio=1.0,
                     record_format=capi.RECORD_STENCIL16)
        out.append(dom.mc_solve(src, internal=True)[0])
    # Ten steps reach ten lines of the grid at most.
    assert np.array_equal(out[0][:60 * 29], out[1][:60 * 29]) and out[0].any()
