"""Flats and directions on grids of few rows, where a warp walks along several
strips of 4, 8 or 16 lanes: row counts around what such strips put out (8, 24
and 56 rows) and around where the rule between them and whole warps lies, column
counts that leave the last walks of a warp beyond the grid.  Both are whole
numbers and must equal the oracle's (src/identifyflats.c:33-121,
src/flow_routing.c:15-76).

A call on one row of 2^20 pixels takes 2.1 (flats) and 2.4 (directions) times one
on as many in a square; 8.5 and 12 with a strip a warp.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = [1, 2, 4, 7, 8, 9, 12, 23, 24, 25, 28, 55, 56, 57, 60, 72, 73, 76, 120, 121, 128, 144, 145,
        168, 169, 172]


def _dem(m, n, levels):
    rng = np.random.default_rng(7 * m + n)
    z = rng.integers(0, levels, (m, n)).astype(np.float32)
    pick = rng.random((m, n))
    for k, v in enumerate([np.nan, -np.inf, np.inf]):
        z[(pick > 0.01 * k) & (pick < 0.01 * k + 0.004)] = v
    return np.asfortranarray(z)


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("n", [1, 5, 67, 1003])
def test_flats(gpu, port, m, n):
    from libtopotoolbox_gb300 import api

    for levels in (2, 4):
        z = _dem(m, n, levels)
        want, count = port.identifyflats(z)
        got, got_count = api.identifyflats(z)
        assert np.array_equal(got, want) and got_count == count


@pytest.mark.parametrize("m", ROWS)
@pytest.mark.parametrize("n", [1, 5, 67, 1003])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -127])  # the second: walked again with divisions
def test_directions(gpu, port, m, n, scale):
    from libtopotoolbox_gb300 import api

    rng = np.random.default_rng(m * 1000 + n)
    z = (rng.integers(0, 5, (m, n)) * scale).astype(np.float32)
    d = (rng.integers(0, 9, (m, n)) * scale).astype(np.float32)
    pick = rng.random((m, n))
    z[pick < 0.01], d[pick > 0.98] = np.nan, np.inf
    flats = ((rng.random((m, n)) < 0.4) & ~np.isnan(z)).astype(np.int32)
    z, d, flats = (np.asfortranarray(a) for a in (z, d, flats))
    for order in (0, 1):
        _, want = port.flow_routing_d8_carve(z, d, flats, order)
        _, got = api.flow_routing_d8_carve(z, d, flats, order)
        assert np.array_equal(got, want)


def test_one_row_is_not_slow(gpu):
    torch = gpu
    from libtopotoolbox_gb300.api import dev

    def times(rows, cols):
        z = torch.rand((cols, rows), device="cuda").mul_(20).round_()
        flats = torch.zeros((cols, rows), dtype=torch.int32, device="cuda")
        dist = torch.zeros((cols, rows), device="cuda")
        best = []
        for f in (lambda: dev.identifyflats(z),
                  lambda: dev.flow_routing_d8_carve(z, dist, flats, want_node=False)):
            took = []
            for _ in range(9):
                a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                torch.cuda.synchronize()
                a.record()
                f()
                b.record()
                torch.cuda.synchronize()
                took.append(a.elapsed_time(b))
            best.append(min(took))
        return best

    thin, square = times(1, 1 << 20), times(1 << 10, 1 << 10)
    assert thin[0] < 4 * square[0] and thin[1] < 5 * square[1], (thin, square)
