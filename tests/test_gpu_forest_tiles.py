"""Receiver-forest tile passes and the adjoint at the edges of their tiles:
paths that wind through every pixel of a tile (1023 steps), rivers that
collect every entry of a tile, and random forests, on grids one pixel short
of, on and past a tile, with signed weights (residues over all 64 bits).

Accumulation: the fixed-point scale 2^k1 has max|w| * N * 2^k1 > 2^61, so
rounding N weights is off by at most N * 2^-(k1+1) <= N^2 * 2^-61 * max|w|,
and the result is rounded once to float32 (2^-24 relative).  Adjoint: a sum of
at most N terms in float-float, each addition within 2^-44 of the terms'
magnitude, then rounded once.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DI = np.array([0, 1, 1, 1, 0, -1, -1, -1])
DJ = np.array([1, 1, 0, -1, -1, -1, 0, 1])


def _serpentine(m, n):
    d = np.zeros((m, n), np.uint8)
    for j in range(n):
        down = j % 2 == 0
        d[:, j] = 4 if down else 64  # (i + 1, j) or (i - 1, j)
        d[-1 if down else 0, j] = 1 if j + 1 < n else 0  # (i, j + 1)
    return d


def _river(m, n):
    d = np.full((m, n), 1, np.uint8)  # every row flows right into the last column
    d[:, -1] = 4
    d[-1, -1] = 0
    return d


def _random(m, n, seed):
    """Each pixel drains to a random neighbour of lower random height."""
    rng = np.random.default_rng(seed)
    z = rng.permutation(m * n).reshape(m, n)
    d = np.zeros((m, n), np.uint8)
    for i in range(m):
        for j in range(n):
            lower = [k for k in range(8) if 0 <= i + DI[k] < m and 0 <= j + DJ[k] < n
                     and z[i + DI[k], j + DJ[k]] < z[i, j]]
            if lower:
                d[i, j] = 1 << int(rng.choice(lower))
    return d


def _order(d):
    """Receivers (linear, column-major; -1 without) and pixels, donors first."""
    m, n = d.shape
    r = np.full(m * n, -1)
    f = d.ravel(order="F")
    src = np.nonzero(f)[0]
    k = np.log2(f[src]).astype(int)
    r[src] = (src // m + DJ[k]) * m + src % m + DI[k]
    left = np.bincount(r[src], minlength=m * n)
    order, ready = [], list(np.nonzero(left == 0)[0])
    while ready:
        p = ready.pop()
        order.append(p)
        if r[p] >= 0:
            left[r[p]] -= 1
            if left[r[p]] == 0:
                ready.append(r[p])
    assert len(order) == m * n
    return r, order


@pytest.mark.parametrize("shape", [(1, 1), (1, 70), (31, 33), (32, 32), (33, 31), (64, 65), (97, 40)])
@pytest.mark.parametrize("kind", ["serpentine", "river", "random"])
def test_forest_tiles(gpu, kind, shape):
    from libtopotoolbox_gb300 import api

    m, n = shape
    d = np.asfortranarray({"serpentine": _serpentine, "river": _river}[kind](m, n)
                          if kind != "random" else _random(m, n, m * 100 + n))
    r, order = _order(d)
    rng = np.random.default_rng(m + n)
    N = m * n
    w = rng.normal(0, 1, N).astype(np.float32)
    total, count = w.astype(np.float64), np.ones(N)
    for p in order:
        if r[p] >= 0:
            total[r[p]] += total[p]
            count[r[p]] += count[p]
    acc = api.flow_accumulation(d, w.reshape(shape, order="F")).ravel(order="F")
    bound = N * N * 2.0 ** -61 * np.abs(w).max() + 2.0 ** -24 * np.abs(total) + N * 2.0 ** -52 * 4
    assert np.all(np.abs(acc - total) <= bound)
    assert np.array_equal(api.flow_accumulation(d).ravel(order="F"), count)
    g = rng.normal(0, 1, N).astype(np.float32)
    grad, mag = g.astype(np.float64), np.abs(g).astype(np.float64)
    for p in reversed(order):
        if r[p] >= 0:
            grad[p] += grad[r[p]]
            mag[p] += mag[r[p]]
    got = api.flow_accumulation_backward(d, g.reshape(shape, order="F")).ravel(order="F")
    assert np.all(np.abs(got - grad) <= 2.0 ** -24 * np.abs(grad) + N * 2.0 ** -44 * mag)
