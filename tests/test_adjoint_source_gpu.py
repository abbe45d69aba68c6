"""The adjoint source build: starting states, emission order and step-0
weights against a direct evaluation, at the edges of its tiles, of the one-CTA
kernel's range, and for sources concentrated in few states."""
import numpy as np
import pytest
import scipy.sparse as sp

from mcls_b200 import capi

pytestmark = pytest.mark.gpu

M = np.uint64(0xFFFFFFFFFFFFFFFF)


def splitmix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def uniforms(count, seed, epoch=0):
    with np.errstate(over="ignore"):
        ekey = splitmix(np.uint64(seed) ^ splitmix(np.uint64(epoch)))
        k = np.arange(count, dtype=np.uint64)
        x = splitmix(ekey ^ splitmix((np.uint64(1) << np.uint64(56)) ^ k))
        x ^= x << np.uint64(13)
        x ^= x >> np.uint64(7)
        x ^= x << np.uint64(17)
    return np.minimum(x.astype(np.float64) * 2.0 ** -64, 1.0 - 2.0 ** -53)


def source(kind, n, gen):
    v = gen.uniform(0.1, 1.0, n) * gen.choice([-1.0, 1.0], n)
    if kind == "spike":
        v *= 1e-9
        v[n // 3] = 1.0
    elif kind == "last":
        v[:] = 0.0
        v[-1] = -2.0
    elif kind == "positive_first":
        v[0] = 3.0
    elif kind == "negative_first":
        v[0] = -0.01
    return v


@pytest.mark.parametrize("n", [1, 2, 17, 1023, 2048, 2049, 16384, 16385, 40000, 70001])
@pytest.mark.parametrize("kind", ["positive_first", "negative_first", "spike", "last"])
@pytest.mark.parametrize("ratio", [0.5, 2.0])
def test_random_starts_are_lower_bounds_of_the_draws(ctx, n, kind, ratio):
    if n == 1 and kind in ("negative_first", "last"):
        pytest.skip("one negative state: the signed first element leaves no histories")
    gen = np.random.default_rng(n)
    A = sp.csr_matrix(0.7 * sp.eye(n))
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP64,
                      rng_mode=capi.RNG_COUNTER, seed=9, history_length=1, sample_ratio=ratio)
    v = source(kind, n, gen)
    x, nh, tr = dom.mc_trace(v, 4 * n + 4, internal=True)
    terms = np.abs(v)
    terms[0] = v[0]
    cdf = np.cumsum(terms.astype(np.longdouble))
    total, norm1 = cdf[-1], np.abs(v).astype(np.longdouble).sum()
    want = int(float(int(n * ratio) * total / norm1))
    # The count truncates a rounded quotient, which may sit on an integer.
    assert abs(nh - want) <= (1 if abs(float(int(n * ratio) * total / norm1) - round(
        float(int(n * ratio) * total / norm1))) < 1e-9 * n else 0)
    u = uniforms(nh, 9)
    c = (cdf / total).astype(np.float64)
    c[-1] = 1.0
    lo = np.searchsorted(c - 1e-12, u, side="left")
    hi = np.searchsorted(c + 1e-12, u, side="left")
    # Emitted from the highest state down; a draw within 1e-12 of a CDF value
    # may fall on either side (the sums' rounding).
    got = tr["start"]
    assert got.size == nh and np.all(np.diff(got) <= 0)
    counts = np.bincount(got, minlength=n)
    sure = np.bincount(np.minimum(lo, n - 1)[lo == hi], minlength=n)
    assert np.all(counts >= sure) and counts.sum() == nh
    if np.all(lo == hi):
        assert np.array_equal(counts, sure)
    # Collision estimate of one-step histories: the step-0 tallies alone.
    w0 = float(norm1) * np.where(v > 0, 1.0, -1.0)
    np.testing.assert_allclose(x, counts * w0 / max(nh, 1), rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [5, 2048, 2049, 16385, 40000])
def test_stratified_counts(ctx, n):
    gen = np.random.default_rng(n)
    A = sp.csr_matrix(0.7 * sp.eye(n))
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP64,
                      rng_mode=capi.RNG_COUNTER, seed=9, history_length=1, sample_ratio=1.5,
                      source_sampling=capi.SOURCE_STRATIFIED)
    v = source("positive_first", n, gen)
    x, nh, tr = dom.mc_trace(v, 4 * n + 4, internal=True)
    f = np.abs(v) * (int(1.5 * n) / np.abs(v).sum())
    want = np.ceil(f).astype(int)
    got = np.bincount(tr["start"], minlength=n)
    near = np.abs(f - np.round(f)) < 1e-9
    assert nh == got.sum() and np.array_equal(got[~near], want[~near])
    assert np.all(np.diff(tr["start"]) <= 0)


# More tiles than one look-back reads (32 at a time) and than run at once.
@pytest.mark.parametrize("n", [32 * 2048, 33 * 2048 + 1, 3_000_001])
@pytest.mark.parametrize("stratified", [False, True])
def test_emission_over_many_tiles(ctx, n, stratified):
    gen = np.random.default_rng(n)
    A = sp.csr_matrix(0.7 * sp.eye(n))
    dom = capi.Domain(ctx, capi.Operator(ctx, A), None, precision=capi.FP64,
                      rng_mode=capi.RNG_COUNTER, seed=9, history_length=1, sample_ratio=1.0,
                      source_sampling=capi.SOURCE_STRATIFIED if stratified
                      else capi.SOURCE_RANDOM)
    v = source("positive_first", n, gen)
    x, nh, tr = dom.mc_trace(v, 4 * n + 4, internal=True)
    got = tr["start"]
    assert got.size == nh and np.all(np.diff(got) <= 0)
    # x = counts * (+-|v|_1) / nh: the counts of the states, from the tally.
    counts = np.bincount(got, minlength=n)
    w0 = np.abs(v).sum() * np.where(v > 0, 1.0, -1.0)
    np.testing.assert_allclose(x, counts * w0 / nh, rtol=1e-10, atol=0)
