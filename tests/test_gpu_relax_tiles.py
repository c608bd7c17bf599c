"""Tile relaxations (fill, reconstruct, gwdt) at the edges of their 32 x 32
tiles: one pixel short of, on and past one, two and three tiles, so that
sweeps start and end on every position and values cross sides and corners
of tiles, on a DEM whose water winds through all tiles to one outlet pixel.
Bit-exact against the oracle.
"""
import numpy as np
import pytest

from conftest import same_float

pytestmark = pytest.mark.gpu

SIDES = [1, 2, 31, 32, 33, 63, 65, 97]


def _maze(m, n, seed):
    """Flat floors between walls with random gaps, and noise on a few cells:
    a fill level reaches most pixels by a path through many tiles."""
    rng = np.random.default_rng(seed)
    z = np.full((m, n), 2.0, np.float32)
    z[:, ::4] = 9.0
    for j in range(0, n, 4):
        z[rng.integers(0, m), j] = 2.0 + rng.integers(0, 3)
    hit = rng.random((m, n)) < 0.05
    z[hit] += rng.integers(-1, 2, int(hit.sum()))
    if m > 8:  # barriers on the floors, which are three pixels wide
        hole = rng.random((m, n)) < 0.005
        hole[:, ::4] = False
        z[hole] = np.nan
    bc = np.zeros((m, n), np.uint8)
    bc[rng.integers(0, m), rng.integers(0, n)] = 1
    return np.asfortranarray(z), np.asfortranarray(bc)


@pytest.mark.parametrize("m", SIDES)
def test_relax_at_tile_edges(gpu, port, m):
    from libtopotoolbox_gb300 import api

    for n in SIDES:
        z, bc = _maze(m, n, 100 * m + n)
        filled = port.fillsinks(z, bc)
        assert same_float(api.fillsinks(z, bc), filled), (m, n, "fill")
        marker = np.asfortranarray(z - np.float32(1.5))
        assert same_float(api.reconstruct(marker, z), port.reconstruct(marker, z)), (m, n)
        flats, _ = port.identifyflats(filled)
        costs, _ = port.gwdt_computecosts(flats, z, filled)
        assert same_float(api.gwdt(costs, flats), port.gwdt(costs, flats)[0]), (m, n, "gwdt")
        got = api.d8_pipeline(z, bc)
        want = port.pipeline(z, bc)
        for k in ("filled", "dist"):
            assert same_float(got[k], want[k]), (m, n, k)
