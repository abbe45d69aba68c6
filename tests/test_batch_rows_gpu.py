"""One batched MCSA iteration, element by element against the host: every width,
rows of up to 16 entries and one with many zeros, warps whose rows straddle
systems and width classes, one history per row (finished by the walk) and
several (tallied)."""
import numpy as np
import pytest
import scipy.sparse as sp

import walk_host
from mcls_b200 import capi
from mcls_b200 import problems as P

pytestmark = pytest.mark.gpu
L = 6


def banded(n, entries, seed):
    """Rows of up to `entries` entries, the diagonal among them."""
    gen = np.random.default_rng(seed)
    off = np.arange(entries - 1) - (entries - 1) // 2
    off = np.where(off >= 0, off + 1, off) * 2
    i = np.repeat(np.arange(n), off.size)
    j = i + np.tile(off, n)
    keep = (j >= 0) & (j < n)
    v = gen.uniform(0.2, 1.0, i.size) * gen.choice([-1.0, 1.0], i.size) * 0.8 / entries
    return sp.csr_matrix(sp.eye(n) * 2.0 + sp.csr_matrix((v[keep], (i[keep], j[keep])),
                                                         shape=(n, n)))


def long_row(n, row):
    """A tridiagonal matrix with zeros stored all along one row."""
    A = sp.diags([-0.4, 2.0, -0.3], [-1, 0, 1], shape=(n, n)).tocoo()
    c = np.setdiff1d(np.arange(n), [row - 1, row, row + 1])
    return sp.csr_matrix((np.concatenate([A.data, np.zeros(c.size)]),
                          (np.concatenate([A.row, np.full(c.size, row)]),
                           np.concatenate([A.col, c]))), shape=(n, n))


FULL3 = sp.csr_matrix(np.array([[2.0, -0.5, 0.3], [0.4, 2.0, -0.6], [0.2, 0.3, 2.0]]))
SETS = {
    "stencils": ([P.poisson2d(3), P.poisson2d(5, 7), P.diffusion3d_varcoef(5, seed=1)[0],
                  P.poisson2d(20, 13), P.diffusion3d_varcoef(9, seed=2)[0], FULL3],
                 [1, 16, 3, 2, 7, 4]),
    "nine": ([P.anisotropic2d(9, 2.5, 0.7), P.poisson2d(6), P.anisotropic2d(17, 2.0, 0.3)],
             [5, 1, 16]),
    "longer": ([banded(150, 10, 1), banded(333, 12, 2), banded(70, 13, 3), banded(65, 16, 4),
                P.poisson2d(8), banded(257, 9, 5)], [2, 1, 9, 4, 8, 16]),
    "zeros": ([P.poisson2d(11), long_row(300, 7), P.poisson2d(4)], [3, 2, 1]),
    "one": ([P.poisson2d(33)], [16]),
    "narrow": ([P.poisson2d(33), P.poisson2d(7), banded(41, 16, 6)], [1, 1, 1]),
}


@pytest.mark.parametrize("name", list(SETS))
@pytest.mark.parametrize("estimator", [capi.EXPECTED_VALUE, capi.COLLISION])
@pytest.mark.parametrize("per", [1, 2, 3])
@pytest.mark.parametrize("block,grab", [(256, 1), (128, 4)])
def test_iterations_match_the_host(ctx, name, estimator, per, block, grab):
    import torch

    systems, nrhs = SETS[name]
    kw = dict(direction=capi.FORWARD, estimator=estimator, precision=capi.FP32,
              sample_ratio=float(per), history_length=L, seed=9)
    bt = capi.Batch(ctx, systems, nrhs, **kw)
    bt.set_launch(block, grab)
    # The batch's rows in placement order, as one system of the same histories.
    order = np.argsort(bt.elem_offsets)
    S = sp.csr_matrix(sp.block_diag([systems[s] for s in order]))
    op = capi.Operator(ctx, S)
    dom = capi.Domain(ctx, op, capi.Precond(ctx, op, capi.PREC_POINT_JACOBI), **kw)
    d = dom.export()
    n = S.shape[0]
    H = sp.csr_matrix((d["h"], d["col"], d["rowptr"]), shape=(n, n))
    first = dict(zip(order, np.concatenate([[0], np.cumsum([systems[s].shape[0]
                                                            for s in order])[:-1]])))
    width = max(nrhs)

    def columns(blocks):
        out = np.zeros((n, width))
        for s, v in enumerate(blocks):
            out[first[s]:first[s] + v.shape[0], :v.shape[1]] = v
        return out

    gen = np.random.default_rng(3)
    Bb = [gen.uniform(-1, 1, (A.shape[0], r)) for A, r in zip(systems, nrhs)]
    Xb = [gen.uniform(-1, 1, (A.shape[0], r)) for A, r in zip(systems, nrhs)]
    B = torch.tensor(bt.pack(Bb), device="cuda:0")
    X = torch.tensor(bt.pack(Xb), device="cuda:0")
    b, inv, omega = columns(Bb), 1.0 / S.diagonal()[:, None], 0.9
    for epoch in range(2):
        x = columns(bt.unpack(X.cpu().numpy()))
        st, _, _ = bt.mcsa_solve_dev(B.data_ptr(), X.data_ptr(), tolerance=0.0, max_iters=1,
                                     richardson_omega=omega)
        assert st["iterations"] == 1 and st["walk_steps"] == n * per * L
        got = columns(bt.unpack(X.cpu().numpy()))
        x2 = x + omega * (inv * (b - S @ x))
        rp2 = inv * (b - S @ x2)
        eps = 2.0 ** -50 * (abs(inv) * (abs(b) + abs(S) @ (abs(x2) + abs(x))) + abs(x2))
        for q in range(width):
            c, extra, scale = rp2[:, q], 0.0, abs(rp2[:, q])
            if estimator == capi.EXPECTED_VALUE:
                c, extra, scale = H @ rp2[:, q], rp2[:, q], abs(H) @ abs(rp2[:, q])
            y, mag, _ = walk_host.forward(d, c, per, 9, L, epoch=epoch)
            # The FP32 tally source of a value known to eps, the compensated
            # FP32 sums, and the 64-bit sums around them.
            weight = walk_host.forward(d, scale + eps[:, q], per, 9, L, epoch=epoch)[1]
            err = 2.0 ** -22 * mag + 2.0 ** -23 * weight
            source = walk_host.forward(d, eps[:, q], per, 9, L, epoch=epoch)[1]
            want = x2[:, q] + extra + y
            assert np.all(abs(got[:, q] - want) <= err + 16 * source + 4 * eps[:, q])
    bt.close()
