"""Timed workloads of the library, each through the calls a program makes.

A case is one call of a public entry point (mcls_b200.capi) on one problem
size: Monte Carlo solves, MCSA and Anderson-accelerated MCSA solves of a fixed
number of iterations, the batched solve, and the learned preconditioner's
inference and training gradient.  A solve to a tolerance repeats the same
iteration until the residual test ends it, so a fixed count (tolerance 0)
times the same work without depending on where a run happens to stop.

The matrices are the generators of mcls_b200.problems (the benchmark's and the
tests' systems) with seeded coefficients and right-hand sides, and an
unstructured sparse matrix for the records that store columns.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mcls_b200 import capi
from mcls_b200 import problems

DEVICE = "cuda:0"
HISTORY_LENGTH = 10
_CTX = None


def _context():
    """A program opens one context per device and keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(0)
    return _CTX


# ---- the cases --------------------------------------------------------------

def listed():
    return [
        # One Monte Carlo solve of a small system (host vectors, the C++
        # facade's MonteCarloSolverManager): all latency.
        dict(name="mc_adjoint_small", kind="mc", problem="poisson2d", size=32,
             direction="adjoint", estimator="collision", precision="fp32", ratio=1.0,
             cutoff=0.0, host=True),
        # The 100^2 Poisson workload of the benchmark: adjoint collision,
        # FP64 walks ended by a weight cutoff.
        dict(name="mcsa_adjoint_fp64_100", kind="mcsa", problem="poisson2d", size=100,
             direction="adjoint", estimator="collision", precision="fp64", ratio=1.0,
             cutoff=1e-4, iterations=25, host=False),
        # A small 2D system with the default FP32 forward walk, host vectors
        # (what MCSASolverManager::solve does with a user's vectors).
        dict(name="mcsa_forward_77", kind="mcsa", problem="varcoef2d", size=77,
             direction="forward", estimator="expected_value", precision="fp32", ratio=2.0,
             cutoff=0.0, iterations=40, host=True),
        # The default manager ("Adjoint MCSA", collision, random sampling) on
        # a middle-sized 3D system.
        dict(name="mcsa_adjoint_64", kind="mcsa", problem="diffusion3d", size=64,
             direction="adjoint", estimator="collision", precision="fp32", ratio=1.0,
             cutoff=0.0, iterations=20, host=False),
        # The benchmark's headline: 128^3 variable-coefficient diffusion.
        dict(name="mcsa_forward_128", kind="mcsa", problem="diffusion3d", size=128,
             direction="forward", estimator="expected_value", precision="fp32", ratio=2.0,
             cutoff=0.0, iterations=20, host=False),
        # Diffusion-reaction on material blocks, records larger than L2.
        dict(name="mcsa_blocks_160", kind="mcsa", problem="blocks3d", size=160,
             direction="forward", estimator="expected_value", precision="fp32", ratio=1.0,
             cutoff=0.0, iterations=10, host=False),
        # Unstructured sparsity: packed (column, CDF) records, general layout.
        dict(name="mcsa_unstructured", kind="mcsa", problem="unstructured", size=100003,
             direction="forward", estimator="collision", precision="fp32", ratio=2.0,
             cutoff=0.0, iterations=20, host=False),
        # Learned preconditioner on the anisotropic 9-point family (25-offset
        # H, 16-bit stencil records).
        dict(name="mcsa_learned_aniso_384", kind="mcsa", problem="aniso2d", size=384,
             direction="forward", estimator="expected_value", precision="fp32", ratio=2.0,
             cutoff=0.0, iterations=20, host=False),
        # Anderson-accelerated MCSA, the fastest solver on the 3D workloads.
        dict(name="anderson_96", kind="anderson", problem="diffusion3d", size=96, depth=6,
             ratio=2.0, iterations=12),
        # Many systems with many right-hand sides in one loop.
        dict(name="batch_128", kind="batch", systems=128, nmin=1000, nmax=10000, rhs_max=16,
             ratio=1.0, iterations=15),
        # Learned-preconditioner inference over a large operator.
        dict(name="spai_infer_128", kind="infer", problem="diffusion3d", size=128),
        # One training gradient of that network (a 32^3 sample, residual-like
        # and random vectors), taken thousands of times per training run.
        dict(name="spai_gradient_32", kind="gradient", problem="diffusion3d", size=32,
             vectors=15),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mc", "mcsa64", "mcsa2d", "mcsa_adjoint", "mcsa3d", "mcsa3d", "blocks",
                       "unstructured", "learned", "anderson", "batch", "infer", "gradient"])
    walk = dict(direction="forward", estimator="expected_value", precision="fp32", cutoff=0.0,
                host=False)
    if kind == "mc":
        return dict(kind="mc", problem=rng.choice(["poisson2d", "varcoef2d"]),
                    size=_log_int(rng, 12, 200), direction=rng.choice(["adjoint", "forward"]),
                    estimator=rng.choice(["collision", "expected_value"]),
                    precision="fp32", ratio=rng.choice([1.0, 2.0, 4.0]), cutoff=0.0,
                    host=rng.choice([True, False]))
    if kind == "mcsa64":
        return dict(kind="mcsa", problem="poisson2d", size=_log_int(rng, 24, 220),
                    direction=rng.choice(["adjoint", "forward"]), estimator="collision",
                    precision="fp64", ratio=1.0, cutoff=rng.choice([0.0, 1e-4]),
                    iterations=rng.randint(10, 25), host=False)
    if kind == "mcsa2d":
        return dict(walk, kind="mcsa", problem=rng.choice(["poisson2d", "varcoef2d"]),
                    size=_log_int(rng, 16, 700), ratio=float(rng.randint(1, 4)),
                    iterations=rng.randint(10, 30), host=rng.choice([True, False]))
    if kind == "mcsa_adjoint":
        return dict(kind="mcsa", problem=rng.choice(["diffusion3d", "varcoef2d"]),
                    size=_log_int(rng, 24, 100), direction="adjoint",
                    estimator=rng.choice(["collision", "collision", "expected_value"]),
                    precision="fp32", ratio=rng.choice([0.5, 1.0, 2.0]), cutoff=0.0,
                    iterations=rng.randint(8, 20), host=False)
    if kind == "mcsa3d":
        return dict(walk, kind="mcsa", problem="diffusion3d", size=_log_int(rng, 20, 140),
                    estimator=rng.choice(["expected_value", "expected_value", "collision"]),
                    ratio=float(rng.randint(1, 4)), iterations=rng.randint(6, 14))
    if kind == "blocks":
        return dict(walk, kind="mcsa", problem="blocks3d", size=8 * rng.randint(6, 19),
                    ratio=float(rng.randint(1, 2)), iterations=rng.randint(5, 10))
    if kind == "unstructured":
        return dict(walk, kind="mcsa", problem="unstructured", size=_log_int(rng, 3000, 300000),
                    estimator=rng.choice(["collision", "expected_value"]),
                    direction=rng.choice(["forward", "adjoint"]), ratio=float(rng.randint(1, 2)),
                    iterations=rng.randint(8, 20))
    if kind == "learned":
        return dict(walk, kind="mcsa", problem="aniso2d", size=_log_int(rng, 64, 512), ratio=2.0,
                    iterations=rng.randint(8, 20))
    if kind == "anderson":
        return dict(kind="anderson", problem="diffusion3d", size=_log_int(rng, 20, 112),
                    depth=rng.randint(1, 8), ratio=float(rng.randint(1, 2)),
                    iterations=rng.randint(8, 12))
    if kind == "batch":
        return dict(kind="batch", systems=_log_int(rng, 4, 128), nmin=500,
                    nmax=_log_int(rng, 2000, 10000), rhs_max=rng.choice([1, 4, 16]), ratio=1.0,
                    iterations=rng.randint(6, 15))
    if kind == "infer":
        return dict(kind="infer", problem="diffusion3d", size=_log_int(rng, 16, 128))
    return dict(kind="gradient", problem="diffusion3d", size=_log_int(rng, 12, 48),
                vectors=rng.randint(4, 20))


# ---- inputs -------------------------------------------------------------------

def _diffusion2d(n, gen):
    """5-point variable-coefficient diffusion on an n x n grid (coefficients
    log-uniform in [0.1, 10] per cell): the batched workload's 2D systems."""
    D = np.exp(gen.uniform(np.log(0.1), np.log(10.0), size=(n, n)))
    return problems._diffusion2d(D, np.full((n, n), 0.01), 1.0 / (n + 1))


def _unstructured(n, gen):
    """Symmetric diagonally dominant matrix of a random graph: every vertex
    is joined to three others within a bandwidth, as a numbered unstructured
    mesh is (5 to about 16 entries per row)."""
    width = max(8, n // 50)
    i = np.repeat(np.arange(n), 3)
    j = (i + gen.integers(1, width, size=3 * n)) % n
    w = np.exp(gen.uniform(np.log(0.3), np.log(3.0), size=3 * n))
    keep = i != j
    i, j, w = i[keep], j[keep], w[keep]
    # The CSR type of the generators, without naming its package here.
    csr = type(problems.poisson2d(3))
    off = csr((w, (i, j)), shape=(n, n))
    off = off + off.T
    deg = np.asarray(off.sum(axis=1)).reshape(-1)
    r = np.arange(n)
    A = csr((deg * 1.05 + 0.01, (r, r)), shape=(n, n)) - off
    A = csr(A)
    A.sort_indices()
    return A


def _matrix(case, gen, seed):
    p, n = case["problem"], case["size"]
    if p == "poisson2d":
        return problems.poisson2d(n)
    if p == "varcoef2d":
        return _diffusion2d(n, gen)
    if p == "diffusion3d":
        return problems.diffusion3d_varcoef(n, seed=seed)[0]
    if p == "blocks3d":
        return problems.diffusion3d_blocks(n, 8, seed=seed)[0]
    if p == "aniso2d":
        # Rotated tensors of moderate anisotropy, where the walk's weights
        # stay bounded without a trained network.
        return problems.anisotropic2d(n, float(gen.uniform(2.0, 4.0)),
                                      float(gen.uniform(0.0, np.pi)))
    return _unstructured(n, gen)


def _net_params(slots, gen):
    """Parameters of a network as training leaves them: He-uniform hidden
    layers, a small output layer, and output biases that add a positive
    fraction of each neighbour (an approximate inverse of a diffusion row)."""
    k = dict(f=16, h=64, o=16)
    w1 = gen.uniform(-1, 1, (k["h"], k["f"])) * math.sqrt(6.0 / k["f"])
    w2 = gen.uniform(-1, 1, (k["h"], k["h"])) * math.sqrt(6.0 / k["h"])
    w3 = gen.uniform(-1, 1, (k["o"], k["h"])) * 2e-3
    b3 = np.zeros(k["o"])
    b3[:slots] = 0.03
    b3[slots // 2] = 0.05
    z = np.zeros(k["h"])
    b1 = gen.uniform(-0.1, 0.1, k["h"])
    return np.concatenate([v.reshape(-1) for v in (w1, b1, w2, z, w3, b3)]).astype(np.float32)


def _slots(A):
    n = A.shape[0]
    rows = np.repeat(np.arange(n), np.diff(A.indptr))
    return np.unique(A.indices - rows)


def _vectors(n, count, size, seed):
    """Half random, half smooth vectors (a residual after some iterations)."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    V = torch.randn((count, n), dtype=torch.float64, device=DEVICE, generator=g)
    k = count // 2
    if k:
        s = V[:k].reshape(k, 1, size, size, size)
        box = torch.ones((1, 1, 3, 3, 3), dtype=torch.float64, device=DEVICE) / 27.0
        for _ in range(3):
            s = torch.nn.functional.conv3d(s, box, padding=1)
        V[:k] = s.reshape(k, n)
    return V.contiguous()


def _batch(case, seed):
    """The batched workload: 2D and 3D Poisson and variable-coefficient
    systems, sizes log-uniform on square and cube grids.  The grids and
    right-hand-side counts belong to the case, the coefficients and
    right-hand sides to the seed."""
    shape = np.random.Generator(np.random.PCG64(case["systems"] * 1000003 + case["nmax"]))
    gen = np.random.Generator(np.random.PCG64(seed))
    systems, nrhs, rhs = [], [], []
    for _ in range(case["systems"]):
        kind = int(shape.integers(0, 4))
        rows = float(np.exp(shape.uniform(np.log(case["nmin"]), np.log(case["nmax"]))))
        r = int(shape.integers(1, case["rhs_max"] + 1))
        n = max(3, int(round(rows ** (0.5 if kind < 2 else 1.0 / 3.0))))
        if kind == 0:
            A = problems.poisson2d(n)
        elif kind == 1:
            A = _diffusion2d(n, gen)
        elif kind == 2:
            A = problems._diffusion3d(np.ones((n, n, n)), np.zeros((n, n, n)), 1.0 / (n + 1))
        else:
            A = problems.diffusion3d_varcoef(n, seed=int(gen.integers(1 << 31)))[0]
        systems.append(A)
        nrhs.append(r)
        rhs.append(gen.uniform(0.0, 1.0, size=(A.shape[0], r)))
    return systems, nrhs, rhs


def _inputs(case, seed):
    """The problem data of a case, host side: (matrix, right-hand side, extra)."""
    gen = np.random.Generator(np.random.PCG64(seed))
    A = _matrix(case, gen, seed)
    b = gen.uniform(0.0, 1.0, size=A.shape[0])
    net = _net_params(_slots(A).size, gen) if case["kind"] in ("infer", "gradient") or \
        case["problem"] == "aniso2d" else None
    return A, b, net


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    s = dict(case=case, kind=kind, ctx=ctx)
    if kind == "batch":
        systems, nrhs, rhs = _batch(case, seed)
        bt = capi.Batch(ctx, systems, nrhs, direction=capi.FORWARD,
                        estimator=capi.EXPECTED_VALUE, precision=capi.FP32,
                        sample_ratio=case["ratio"], history_length=HISTORY_LENGTH, seed=seed)
        s["batch"] = bt
        s["b"] = torch.from_numpy(bt.pack(rhs)).to(DEVICE)
        s["x"] = torch.empty_like(s["b"])
        s["params"] = capi.mcsa_params(tolerance=0.0, max_iters=case["iterations"])
        return s
    A, b, net = _inputs(case, seed)
    n = A.shape[0]
    s["op"] = op = capi.Operator(ctx, A)
    if net is not None:
        s["net"] = capi.SpaiNet(ctx, _slots(A).size, seed=0)
        s["net"].params = net
    if kind == "infer":
        s["out"] = torch.empty((n, 16), dtype=torch.float32, device=DEVICE)
        s["m"] = torch.empty(A.nnz, dtype=torch.float64, device=DEVICE)
        return s
    if kind == "gradient":
        s["V"] = _vectors(n, case["vectors"], case["size"], seed)
        return s
    if net is not None:
        s["pc"] = capi.Precond(ctx, op, capi.PREC_LEARNED_SPAI, net=s["net"], rho_fallback=2.0)
    else:
        s["pc"] = capi.Precond(ctx, op, capi.PREC_POINT_JACOBI)
    fp64 = case.get("precision") == "fp64"
    s["dom"] = capi.Domain(
        ctx, op, s["pc"], seed=seed, history_length=HISTORY_LENGTH, sample_ratio=case["ratio"],
        direction=capi.ADJOINT if case.get("direction") == "adjoint" else capi.FORWARD,
        estimator=capi.COLLISION if case.get("estimator") == "collision" else capi.EXPECTED_VALUE,
        precision=capi.FP64 if fp64 else capi.FP32, weight_cutoff=case.get("cutoff", 0.0),
        rng_mode=capi.RNG_COUNTER,
        record_format=capi.RECORD_STENCIL16 if net is not None else capi.RECORD_AUTO)
    if case.get("host"):
        s["b"] = b
    else:
        s["b"] = torch.from_numpy(b).to(DEVICE)
        s["x"] = torch.empty_like(s["b"])
        if n >= 1 << 18:
            # Large systems are solved many thousand iterations long: the
            # launch shape is tuned once, as the benchmark does.
            s["dom"].autotune(s["b"].data_ptr(), reps=1)
    if kind == "mcsa":
        s["params"] = capi.mcsa_params(tolerance=0.0, max_iters=case["iterations"])
    elif kind == "anderson":
        s["params"] = capi.anderson_params(tolerance=0.0, max_iters=case["iterations"],
                                           storage_depth=case["depth"])
    return s


# ---- one pass ------------------------------------------------------------------

def _stats(st):
    return {k: st[k] for k in ("iterations", "histories", "walk_steps", "residual_norm")}


def run(s):
    kind = s["kind"]
    if kind == "infer":
        s["net"].infer_dev(s["op"], s["out"].data_ptr(), s["m"].data_ptr())
        return {"out": s["out"], "m": s["m"]}
    if kind == "gradient":
        loss, grad = s["net"].gradient(s["op"], s["V"].data_ptr(), s["V"].shape[0])
        return {"loss": loss, "grad": grad}
    if kind == "batch":
        s["x"].zero_()
        st, _, rel = s["batch"].mcsa_solve_dev(s["b"].data_ptr(), s["x"].data_ptr(),
                                               params=s["params"])
        return {"x": s["x"], "rel": rel, "iterations": st["iterations"],
                "walk_steps": st["walk_steps"]}
    dom = s["dom"]
    if kind == "mc":
        if s["case"]["host"]:
            x, st = dom.mc_solve(s["b"])
        else:
            st, x = dom.mc_solve_dev(s["b"].data_ptr(), s["x"].data_ptr()), s["x"]
        return {"x": x, "histories": st["histories"], "walk_steps": st["walk_steps"]}
    if kind == "anderson":
        s["x"].zero_()
        st = dom.anderson_solve_dev(s["b"].data_ptr(), s["x"].data_ptr(), params=s["params"])
        return {"x": s["x"], **_stats(st)}
    if s["case"]["host"]:
        x, st = dom.mcsa_solve(s["b"], params=s["params"])
    else:
        s["x"].zero_()
        st, x = dom.mcsa_solve_dev(s["b"].data_ptr(), s["x"].data_ptr(), params=s["params"]), s["x"]
    return {"x": x, **_stats(st)}


# ---- the work of one pass ---------------------------------------------------------

def _rows_entries(case):
    p, n = case["problem"], case["size"]
    if p in ("diffusion3d", "blocks3d"):
        return n ** 3, 7 * n ** 3
    if p == "unstructured":
        return n, 7 * n
    return n * n, (9 if p == "aniso2d" else 5) * n * n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # Log-uniform sizes and 1..rhs_max right-hand sides, on average.
        lo, hi = case["nmin"], case["nmax"]
        rows = case["systems"] * (hi - lo) / math.log(hi / lo)
        cols = (1 + case["rhs_max"]) / 2
        steps = rows * case["ratio"] * HISTORY_LENGTH
        it = case["iterations"]
        return {"bytes": it * (rows * 6 * 8 + rows * cols * 4 * 8),
                "flops": it * (rows * cols * 6 * 2 * 2 + steps * (8 + 2 * cols))}
    n, nnz = _rows_entries(case)
    mlp = 2 * (16 * 64 + 64 * 64 + 64 * 16)
    if kind == "infer":
        return {"bytes": 8 * nnz + 8 * nnz + 64 * n, "flops": mlp * n}
    if kind == "gradient":
        r = case["vectors"]
        return {"bytes": 8 * nnz + 8 * n * r, "flops": 4 * mlp * n + 6 * nnz * r}
    steps = n * case["ratio"] * HISTORY_LENGTH
    if kind == "mc":
        return {"bytes": 8 * nnz + 16 * n, "flops": 8 * steps}
    # Per iteration: the operator's values, the right-hand side and the
    # iterate and residual in and out.
    it = case["iterations"]
    extra = 3 * case["depth"] * 8 * n if kind == "anderson" else 0
    return {"bytes": it * (8 * nnz + 5 * 8 * n + extra),
            "flops": it * (4 * nnz + 8 * steps)}


# ---- 64-bit values -----------------------------------------------------------------

def _dia(A, offsets):
    """A's values by diagonal offset, [slots, n], and their pattern."""
    n = A.shape[0]
    rows = np.repeat(np.arange(n), np.diff(A.indptr))
    k = np.searchsorted(offsets, A.indices - rows)
    val, has = np.zeros((offsets.size, n)), np.zeros((offsets.size, n), bool)
    val[k, rows] = A.data
    has[k, rows] = True
    return val, has, k, rows


def _shift(v, o):
    """v[i + o] along the last axis, 0 outside."""
    r = torch.zeros_like(v)
    n = v.shape[-1]
    if o >= 0:
        r[..., : n - o] = v[..., o:]
    else:
        r[..., -o:] = v[..., : n + o]
    return r


def _mlp64(A, params):
    """Raw network outputs [n, 16] in 64 bits (differentiable in params)."""
    off = _slots(A)
    val, has, k, rows = _dia(A, off)
    val, has = torch.from_numpy(val).to(DEVICE), torch.from_numpy(has).to(DEVICE)
    c = int(np.searchsorted(off, 0))
    n = A.shape[0]
    f = torch.zeros((n, 16), dtype=torch.float64, device=DEVICE)
    q = 0
    for j, o in enumerate(off):
        if j == c:
            continue
        live = has[j] & (val[j] != 0)
        d = torch.where(live, _shift(val[c], int(o)) / val[c], torch.ones_like(val[c]))
        f[:, 2 * q] = torch.where(live, val[j] / val[c], torch.zeros_like(val[c]))
        f[:, 2 * q + 1] = torch.log(d)
        q += 1
    w1, b1, w2, b2, w3, b3 = torch.split(params, [1024, 64, 4096, 64, 1024, 16])
    h = torch.relu(f @ w1.reshape(64, 16).T + b1)
    h = torch.relu(h @ w2.reshape(64, 64).T + b2)
    return h @ w3.reshape(16, 64).T + b3, val, has, off, c, k, rows


def exact(case, seed):
    """The network's outputs, loss and gradient in 64 bits.  A Monte Carlo
    estimate has no such value."""
    kind = case["kind"]
    if kind not in ("infer", "gradient"):
        return None
    A, _, net = _inputs(case, seed)
    p = torch.from_numpy(net.astype(np.float64)).to(DEVICE)
    if kind == "infer":
        out, val, _, off, c, k, rows = _mlp64(A, p)
        kk, rr = torch.from_numpy(k).to(DEVICE), torch.from_numpy(rows).to(DEVICE)
        m = ((kk == c).double() + out[rr, kk]) / val[c][rr]
        return {"out": out, "m": m}
    p.requires_grad_(True)
    out, val, has, off, c, _, _ = _mlp64(A, p)
    V = _vectors(A.shape[0], case["vectors"], case["size"], seed)
    Z = sum(val[j] * _shift(V, int(o)) for j, o in enumerate(off))
    MZ = sum(torch.where(has[j], (float(j == c) + out[:, j]) / val[c], torch.zeros_like(val[c])) *
             _shift(Z, int(o)) for j, o in enumerate(off))
    E = V - MZ
    loss = ((E * E).sum(1) / (V * V).sum(1)).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": p.grad}
