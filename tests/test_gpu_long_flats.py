"""Labels and costs of flats that reach over many tiles: rows, columns and bands
of one flat, whole grids with tiles cut off at their edges, and random masks on
grids of enough tiles for a warp to take one, two and four of them in the border
pass.  The labels are the smallest pixel of maximal depth of each 8-connected
component, by scipy's labelling; costs follow from them bit for bit (the
difference in float, 0.1 added in double, src/gwdt.c:247-277).

A flat of 2^20 pixels in one row or column takes about twice what it takes in a
square; 25 to 40 times when the unions across tiles walked up to their roots.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(f, depth):
    from scipy import ndimage

    m, n = f.shape
    comp, count = ndimage.label(f, structure=np.ones((3, 3)))
    comp, d, at = comp.ravel(order="F"), depth.ravel(order="F"), np.arange(m * n)
    most = np.full(count + 1, -np.inf, np.float32)
    np.maximum.at(most, comp, d)
    first = np.full(count + 1, m * n, np.int64)
    hit = d == most[comp]
    np.minimum.at(first, comp[hit], at[hit])
    flat = f.ravel(order="F")
    label = np.where(flat, first[comp], 0)
    cost = np.where(flat, ((most[comp] - d).astype(np.float64) + 0.1).astype(np.float32),
                    np.float32(0))
    return label.reshape((m, n), order="F"), cost.reshape((m, n), order="F")


@pytest.mark.parametrize("shape,share", [
    ((1, 5000), 1.0), ((5000, 1), 1.0), ((2, 4097), 1.0), ((33, 3001), 1.0), ((3001, 40), 1.0),
    ((700, 515), 1.0), ((512, 640), 1.0),
    ((700, 515), 0.45), ((300, 303), 0.99),     # a tile a warp
    ((3, 500000), 0.5), ((500000, 2), 0.97),    # two
    ((3, 1000000), 0.5), ((65, 340000), 0.97),  # four
])
def test_labels_and_costs(gpu, shape, share):
    from libtopotoolbox_gb300 import api

    rng = np.random.default_rng(sum(shape))
    f = rng.random(shape) < share
    flats = np.asfortranarray(f.astype(np.int32))
    filled = np.asfortranarray(np.full(shape, 50, np.float32))
    dem = np.asfortranarray(filled - rng.integers(0, 6, shape).astype(np.float32))  # ties
    costs, labels = api.gwdt_computecosts(flats, dem, filled)
    label, cost = _want(f, filled - dem)
    assert np.array_equal(labels, label)
    assert np.array_equal(costs, cost)


def test_depths_that_are_no_numbers(gpu):
    from libtopotoolbox_gb300 import api

    shape = (70, 68)  # tiles inside the flat without any depth, or with NaN among them
    flats = np.ones(shape, np.int32, order="F")
    filled = np.full(shape, 9, np.float32, order="F")
    dem = np.full(shape, np.nan, np.float32, order="F")
    dem[40, 40], dem[50, 33], dem[66, 3] = 4, 4, 8
    _, labels = api.gwdt_computecosts(flats, dem, filled)
    assert np.all(labels == 33 * 70 + 50)


def test_a_row_is_not_slow(gpu):
    torch = gpu
    from libtopotoolbox_gb300.api import dev

    def took(rows, cols):
        flats = torch.ones((cols, rows), dtype=torch.int32, device="cuda")
        dem = torch.rand((cols, rows), device="cuda")
        best = []
        for _ in range(9):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            torch.cuda.synchronize()
            a.record()
            dev.gwdt_computecosts(flats, dem, dem)
            b.record()
            torch.cuda.synchronize()
            best.append(a.elapsed_time(b))
        return min(best)

    square = took(1 << 10, 1 << 10)
    assert took(1, 1 << 20) < 8 * square
    assert took(1 << 20, 1) < 8 * square
