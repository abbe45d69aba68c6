"""The FP32 walks on the host, all histories at once (numpy): the counter stream,
24-bit draws, FP32 CDF values and weights, 64-bit sums."""
import numpy as np

U = np.uint64


def splitmix(z):
    z = z + U(0x9E3779B97F4A7C15)
    z = (z ^ (z >> U(30))) * U(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> U(27))) * U(0x94D049BB133111EB)
    return z ^ (z >> U(31))


def xorshift(x):
    x = x ^ (x << U(13))
    x = x ^ (x >> U(7))
    return x ^ (x << U(17))


def streams(kind, count, seed, epoch=0):
    """The first state of each of `count` counter streams (1: draws of the
    source, 2: histories)."""
    with np.errstate(over="ignore"):
        ekey = splitmix(U(seed) ^ splitmix(U(epoch)))
        s = splitmix(ekey ^ splitmix((U(kind) << U(56)) ^ np.arange(count, dtype=np.uint64)))
    return np.where(s == 0, U(0x9E3779B97F4A7C15), s)


class Walk:
    """Transitions of a domain (capi.Domain.export())."""

    def __init__(self, d):
        rp = np.asarray(d["rowptr"], np.int64)
        n, width = rp.size - 1, int(np.diff(rp).max())
        self.n = n
        self.W = np.asarray(d["weights"]).astype(np.float32)
        self.cdf = np.full((n, width), 2.0, np.float32)
        self.col = np.zeros((n, width), np.int64)
        self.neg = np.zeros((n, width), bool)
        row = np.repeat(np.arange(n), np.diff(rp))
        at = np.arange(rp[-1]) - rp[row]
        self.cdf[row, at] = np.asarray(d["cdf"]).astype(np.float32)
        self.col[row, at] = d["col"]
        self.neg[row, at] = ~(np.asarray(d["h"]) > 0)

    def step(self, s, w, r):
        with np.errstate(over="ignore"):
            r = xorshift(r)
        u = (r >> U(40)).astype(np.float32) * np.float32(2.0 ** -24)
        k = (self.cdf[s] < u[:, None]).sum(1)
        w = (w * self.W[s]).astype(np.float32)
        return self.col[s, k], np.where(self.neg[s, k], -w, w), r


def forward(d, src, per, seed, length, epoch=0, cutoff=0.0):
    """Collision estimate of every row by `per` histories, the sum of the terms'
    magnitudes over per, and the steps taken."""
    t = Walk(d)
    c = np.asarray(src).astype(np.float32).astype(np.float64)
    row = np.repeat(np.arange(t.n), per)
    s, w = row.copy(), np.ones(row.size, np.float32)
    r = streams(2, row.size, seed, epoch)
    x, mag, steps = np.zeros(t.n), np.zeros(t.n), 0
    live = np.arange(row.size)
    for _ in range(length):
        term = w.astype(np.float64) * c[s]
        np.add.at(x, row[live], term)
        np.add.at(mag, row[live], np.abs(term))
        s, w, r = t.step(s, w, r)
        steps += live.size
        keep = ~(np.abs(w) < np.float32(cutoff))
        live, s, w, r = live[keep], s[keep], w[keep], r[keep]
    return x / per, mag / per, steps


def adjoint(d, start, sign, norm1, seed, length, epoch=0, cutoff=0.0):
    """Collision estimate by histories from the given states with weights
    sign * norm1, the magnitudes' sum and the steps taken."""
    t = Walk(d)
    s = np.asarray(start, np.int64)
    nh = s.size
    w = (np.asarray(sign) * np.float32(norm1)).astype(np.float32)
    x, mag, steps = np.zeros(t.n), np.zeros(t.n), 0
    np.add.at(x, s, np.asarray(sign) * norm1)
    np.add.at(mag, s, np.full(nh, float(norm1)))
    r = streams(2, nh, seed, epoch)
    wcut = np.float32(cutoff) * np.float32(norm1)
    for k in range(length):
        if k:
            np.add.at(x, s, w.astype(np.float64))
            np.add.at(mag, s, np.abs(w).astype(np.float64))
        s, w, r = t.step(s, w, r)
        steps += s.size
        keep = ~(np.abs(w) < wcut)
        s, w, r = s[keep], w[keep], r[keep]
    return x / nh, mag / nh, steps


def starts(v, nh, seed, epoch=0):
    """Starting states of nh random adjoint histories of the source v (v[0] > 0),
    highest first, and their signs."""
    with np.errstate(over="ignore"):
        x = xorshift(streams(1, nh, seed, epoch))
    u = np.minimum(x.astype(np.float64) * 2.0 ** -64, 1.0 - 2.0 ** -53)
    c = np.cumsum(np.abs(v).astype(np.longdouble))
    c = (c / c[-1]).astype(np.float64)
    c[-1] = 1.0
    at = np.sort(np.searchsorted(c, u, side="left"))[::-1]
    return at, np.where(np.asarray(v)[at] > 0, 1.0, -1.0)
