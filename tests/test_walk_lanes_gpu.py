"""Many histories per row: lanes, a warp and several warps that share a row.  How
a row's histories are shared out changes none of them."""
import numpy as np
import pytest
import scipy.sparse as sp

import walk_host
from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu
L = 10


def matrix(n):
    """A chain with a few distant entries, random weights of both signs."""
    gen = np.random.default_rng(n)
    if n == 1:
        return sp.csr_matrix(np.array([[0.7]]))
    i = np.repeat(np.arange(n), 4)
    j = (i + np.tile([1, -1, 5, 17], n)) % n
    keep = i != j
    v = gen.uniform(0.05, 0.2, i.size) * gen.choice([-1.0, 1.0], i.size)
    return sp.csr_matrix(sp.eye(n) + sp.csr_matrix((v[keep], (i[keep], j[keep])), shape=(n, n)))


# 148 SMs hold 303,104 lanes: 9,472 rows of a warp each, 18,944 of 16 lanes.
@pytest.mark.parametrize("n,per", [(1, 5), (1, 33), (1, 5000), (2, 64), (3, 31), (40, 1000),
                                   (700, 3), (700, 7), (700, 32), (700, 100), (4736, 65),
                                   (4737, 65), (9472, 33), (9473, 33), (18944, 17), (18945, 17),
                                   (20000, 9)])
@pytest.mark.parametrize("estimator", [capi.COLLISION, capi.EXPECTED_VALUE])
@pytest.mark.parametrize("block,l1", [(256, 0), (128, 1)])
def test_forward_rows_match_the_histories(ctx, n, per, estimator, block, l1):
    dom = capi.Domain(ctx, capi.Operator(ctx, matrix(n)), None, precision=capi.FP32,
                      direction=capi.FORWARD, estimator=estimator, sample_ratio=float(per),
                      history_length=L, seed=11)
    dom.set_launch(1, block)
    dom.set_record_cache(l1)
    src = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    x, st = dom.mc_solve(src, internal=True)
    d = dom.export()
    c, extra, err = src, 0.0, 0.0
    if estimator == capi.EXPECTED_VALUE:
        # The tally source H src in FP64 (its sum in any order), then FP32.
        H = sp.csr_matrix((d["h"], d["col"], d["rowptr"]), shape=(n, n))
        c, extra = H @ src, src
        err = 2.0 ** -23 * walk_host.forward(d, abs(H) @ abs(src), per, 11, L)[1]
    ref, mag, steps = walk_host.forward(d, c, per, 11, L)
    assert st["histories"] == n * per and st["walk_steps"] == n * per * L == steps
    # A history's compensated FP32 sum is within 2^-22 of its terms' magnitude,
    # the 64-bit sum of the histories within per roundings of it.
    assert np.all(np.abs(x - (extra + ref)) <= (2.0 ** -22 + per * 2.0 ** -53) * mag + err
                  + 2.0 ** -52 * np.abs(extra))


@pytest.mark.parametrize("n,per", [(10, 900), (50, 40)])
def test_loops_with_many_histories(ctx, n, per):
    A, b = P.diffusion3d_varcoef(4, seed=3) if n == 50 else (P.poisson2d(n), np.ones(n * n))
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    for kw in (dict(), dict(host_loop=1)):
        dom = capi.Domain(ctx, op, pc, precision=capi.FP32, direction=capi.FORWARD,
                          estimator=capi.EXPECTED_VALUE, sample_ratio=float(per), seed=5)
        for solve in (dom.mcsa_solve, dom.anderson_solve):
            x, st = solve(b, tolerance=1e-9, max_iters=1000, **kw)
            assert st["converged"] == 1
            assert st["histories"] == st["iterations"] * A.shape[0] * per
            r = (b - A @ x) / A.diagonal()
            assert np.linalg.norm(r) <= 1.0001e-9 * np.linalg.norm(b) * max(
                1.0, (1 / A.diagonal()).max())


@pytest.mark.parametrize("n,order", [(24, 0), (80, 0), (90, 1), (200, 1)])
def test_small_domains_hold_no_row_order(ctx, n, order):
    # 80^2 records of 32 bytes are the last to fit a block's shared memory, where
    # rows are taken as they come.  A domain of histories ended by a weight
    # cutoff never has an order and allocates the same otherwise.
    op = capi.Operator(ctx, P.poisson2d(n) / 4.0)
    count = []
    for cutoff in (0.0, 1e-3):
        before = capi.device_allocations()[0]
        dom = capi.Domain(ctx, op, None, precision=capi.FP32, direction=capi.FORWARD,
                          estimator=capi.COLLISION, sample_ratio=1.0, weight_cutoff=cutoff)
        count.append(capi.device_allocations()[0] - before)
        dom.close()
    assert count[0] - count[1] == order


def test_autotune_of_a_walk_with_one_shape(ctx):
    import torch

    op = capi.Operator(ctx, matrix(700))
    dom = capi.Domain(ctx, op, None, precision=capi.FP32, direction=capi.FORWARD,
                      estimator=capi.COLLISION, sample_ratio=1.0, seed=1)
    v = torch.ones(700, dtype=torch.float64, device="cuda:0")
    for _ in range(5):
        t = dom.autotune(v.data_ptr(), reps=1)
        assert (t["histories_per_lane"], t["block_size"], t["record_cache_l1"]) == (1, 256, 0)
