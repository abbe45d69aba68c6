"""The captured solver loops of one domain (MCSA, multi-set MCSA, Anderson) share
its buffers: a solve with more iterations than any before replaces the residual
history, and the loops captured earlier must not write to the old one."""
import os
import re

import numpy as np
import pytest

from mcls_b200 import capi
from mcls_b200 import problems as P

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcls_b200", "csrc")


def test_the_history_of_a_live_domain_is_replaced_in_one_place():
    # release_domain (capi.cu), the fixed-point scratch and grow_history (mcsa.cu).
    places = {}
    for f in sorted(os.listdir(CSRC)):
        hits = len(re.findall(r"dfree\([^)]*d_resid\)", open(os.path.join(CSRC, f)).read()))
        if hits:
            places[f] = hits
    assert places == {"capi.cu": 1, "fixedpoint.cu": 1, "mcsa.cu": 1}
    body = open(os.path.join(CSRC, "mcsa.cu")).read().split("int grow_history(")[1].split("\n}")[0]
    assert body.index("drop_loops(dom)") < body.index("dfree(dom->d_resid)")


@pytest.mark.parametrize("function", ["mcsa.cu:mclsgpu_domain_set_launch",
                                      "mcsa.cu:mclsgpu_domain_set_record_cache",
                                      "capi.cu:mclsgpu_domain_reseed"])
def test_a_setting_baked_into_the_walks_drops_every_loop(function):
    # The launch shape changes no result, so the loops themselves cannot show it.
    name, fn = function.split(":")
    body = open(os.path.join(CSRC, name)).read().split("int " + fn + "(")[1].split("\n}")[0]
    assert "drop_loops(dom)" in body


@pytest.mark.gpu
@pytest.mark.parametrize("order", [("sets", "mcsa", "sets"), ("sets", "anderson", "sets"),
                                   ("mcsa", "anderson", "mcsa"), ("anderson", "mcsa", "anderson"),
                                   ("mcsa", "sets", "mcsa"), ("anderson", "sets", "anderson")])
def test_solvers_in_turn_with_growing_iteration_limits(ctx, order):
    A = P.poisson2d(12)
    b = np.linspace(0.5, 1.0, A.shape[0])
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    one = capi.set_params(1, lambda ptr, n, stream: None, capturable=True)

    def solve(dom, what, iters, host):
        if what == "anderson":
            return dom.anderson_solve(b, tolerance=0.0, max_iters=iters, host_loop=host)[0]
        if what == "mcsa":
            return dom.mcsa_solve(b, tolerance=0.0, max_iters=iters, host_loop=host)[0]
        return dom.mcsa_solve_sets(one, b, tolerance=0.0, max_iters=iters, host_loop=host)[0]

    out = []
    for host in (0, 1):
        # Forward, one history a row: the same bits on every run.
        dom = capi.Domain(ctx, op, pc, precision=capi.FP64, rng_mode=capi.RNG_COUNTER, seed=4,
                          estimator=capi.EXPECTED_VALUE, direction=capi.FORWARD,
                          sample_ratio=1.0)
        out.append([solve(dom, w, n, host) for w, n in zip(order, (5, 60, 20))])
    for x, y in zip(*out):
        assert np.isfinite(x).all() and np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["mcsa", "sets", "anderson"])
def test_settings_between_solves(ctx, solver):
    A, b = P.diffusion3d_varcoef(21, seed=3)  # 9261 rows: walks from global memory
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    one = capi.set_params(1, lambda ptr, n, stream: None, capturable=True)
    out = []
    for change in (False, True):
        dom = capi.Domain(ctx, op, pc, precision=capi.FP32, direction=capi.FORWARD,
                          estimator=capi.EXPECTED_VALUE, sample_ratio=2.0, seed=2)
        for blk, l1 in ((256, 0), (128, 0), (128, 1), (256, 1)):
            if change:
                dom.set_launch(1, blk)
                dom.set_record_cache(l1)
            if solver == "anderson":
                x = dom.anderson_solve(b, tolerance=0.0, max_iters=4)[0]
            elif solver == "mcsa":
                x = dom.mcsa_solve(b, tolerance=0.0, max_iters=4)[0]
            else:
                x = dom.mcsa_solve_sets(one, b, tolerance=0.0, max_iters=4)[0]
            out.append(x)
    for x, y in zip(out[:4], out[4:]):
        assert np.array_equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["mcsa", "sets", "batch"])
def test_a_kept_loop_has_the_relaxation_asked_for(ctx, solver):
    """The relaxation is baked into the captured loop: one that agrees with the
    last to six decimals gives what a loop captured for it gives."""
    A, b = P.diffusion3d_varcoef(9, seed=1)
    op = capi.Operator(ctx, A)
    pc = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    one = capi.set_params(1, lambda ptr, n, stream: None, capturable=True)
    kw = dict(precision=capi.FP32, direction=capi.FORWARD, estimator=capi.EXPECTED_VALUE,
              sample_ratio=1.0, seed=2)
    near = 0.9 + 4e-7
    out = []
    for first in (0.9, 0.5, 1.25):
        if solver == "batch":
            import torch

            bt = capi.Batch(ctx, [A], [1], **kw)
            B = torch.tensor(bt.pack([b[:, None]]), device="cuda:0")

            def solve(w):
                X = torch.zeros_like(B)
                bt.mcsa_solve_dev(B.data_ptr(), X.data_ptr(), tolerance=0.0, max_iters=5,
                                  richardson_omega=w)
                return X.cpu().numpy()
        else:
            dom = capi.Domain(ctx, op, pc, **kw)

            def solve(w):
                p = dict(tolerance=0.0, max_iters=5, richardson_omega=w)
                return (dom.mcsa_solve(b, **p) if solver == "mcsa" else
                        dom.mcsa_solve_sets(one, b, **p))[0]
        solve(first)  # every domain is then at the same histories
        out.append(solve(near))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[2], out[1])
