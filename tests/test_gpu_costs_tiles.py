"""Labelling of flats and their costs at the edges of the 32 x 32 tiles:
isolated pixels (the most components a tile can hold), one-pixel columns
and rows, combs and full grids, random masks.  Labels are the smallest pixel
of maximal depth of each 8-connected component, found here by flood fill;
costs follow from them bit for bit (the difference in float, 0.1 added in
double, src/gwdt.c:247-277).  The masks reach the grid's outer ring, which
the reference's costs leave out, so the oracle is compared inside it, where a
component lies inside it as a whole.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mask(kind, m, n, rng):
    f = np.zeros((m, n), bool)
    if kind == "isolated":
        f[::2, ::2] = True
    elif kind == "columns":
        f[:, ::2] = True
    elif kind == "rows":
        f[::2, :] = True
    elif kind == "comb":  # one component of many runs
        f[::2, :] = True
        f[:, 0] = True
    elif kind == "full":
        f[:] = True
    elif kind == "diagonals":
        i, j = np.indices((m, n))
        f = ((i + j) % 5 == 0) | ((i - j) % 7 == 0)
    else:
        f = rng.random((m, n)) < 0.45
    return f


def _labels(f, depth):
    m, n = f.shape
    label = np.zeros((m, n), np.int64)
    seen = np.zeros((m, n), bool)
    for i, j in np.argwhere(f):
        if seen[i, j]:
            continue
        part, stack = [], [(i, j)]
        seen[i, j] = True
        while stack:
            a, b = stack.pop()
            part.append((a, b))
            for c in range(max(a - 1, 0), min(a + 2, m)):
                for d in range(max(b - 1, 0), min(b + 2, n)):
                    if f[c, d] and not seen[c, d]:
                        seen[c, d] = True
                        stack.append((c, d))
        deepest = max(depth[p] for p in part)
        best = min(b * m + a for a, b in part if depth[a, b] == deepest)
        for p in part:
            label[p] = best
    return label


@pytest.mark.parametrize("shape", [(1, 1), (31, 33), (32, 32), (33, 31), (65, 64), (3, 97)])
@pytest.mark.parametrize("kind", ["isolated", "columns", "rows", "comb", "full", "diagonals",
                                  "random"])
def test_costs_at_tile_edges(gpu, port, kind, shape):
    from libtopotoolbox_gb300 import api

    rng = np.random.default_rng(sum(shape))
    f = _mask(kind, *shape, rng)
    flats = np.asfortranarray(f.astype(np.int32))
    filled = np.asfortranarray(np.full(shape, 50, np.float32))
    dem = np.asfortranarray(filled - rng.integers(0, 6, shape).astype(np.float32))  # ties
    costs, labels = api.gwdt_computecosts(flats, dem, filled)
    depth = filled - dem
    want = _labels(f, depth)
    assert np.array_equal(labels, want)
    most = depth.ravel(order="F")[want]
    exact = np.where(f, ((most - depth).astype(np.float64) + 0.1).astype(np.float32),
                     np.float32(0))
    assert np.array_equal(costs, exact)
    inside = f.copy()
    inside[[0, -1], :] = inside[:, [0, -1]] = False
    flats = np.asfortranarray(inside.astype(np.int32))
    assert np.array_equal(api.gwdt_computecosts(flats, dem, filled)[0],
                          port.gwdt_computecosts(flats, dem, filled)[0])
