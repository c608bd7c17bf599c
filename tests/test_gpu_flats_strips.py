"""Flats, sills and presills at the edges of the strips a warp walks along:
row counts around the 120 rows of a strip and the four of a lane,
column counts around the smallest and the widest run of columns, arrays off a
16-byte boundary.  Elevations tie often and hold NaN, infinities and zeros of
both signs; flags are whole numbers, so they must equal the oracle's
(src/identifyflats.c:33-121).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dem(m, n, levels):
    rng = np.random.default_rng(7 * m + n)
    z = rng.integers(0, levels, (m, n)).astype(np.float32)
    z[z == 0] = rng.choice(np.float32([0.0, -0.0]), (m, n))[z == 0]
    pick = rng.random((m, n))
    for k, v in enumerate([np.nan, -np.inf, np.inf]):
        z[(pick > 0.01 * k) & (pick < 0.01 * k + 0.004)] = v
    return np.asfortranarray(z)


@pytest.mark.parametrize("levels", [2, 4])
@pytest.mark.parametrize("m", [1, 3, 4, 27, 28, 29, 57, 119, 120, 121, 124, 240, 244])
@pytest.mark.parametrize("n", [1, 3, 7, 8, 9, 17])
def test_strip_edges(gpu, port, m, n, levels):
    from libtopotoolbox_gb300 import api

    z = _dem(m, n, levels)
    want, count = port.identifyflats(z)
    got, got_count = api.identifyflats(z)
    assert np.array_equal(got, want) and got_count == count


@pytest.mark.parametrize("m,n", [(4804, 8200), (1001, 7003)])
def test_wide_column_runs(gpu, port, m, n):
    from libtopotoolbox_gb300 import api

    z = _dem(m, n, 3)
    want, count = port.identifyflats(z)
    got, got_count = api.identifyflats(z)
    assert np.array_equal(got, want) and got_count == count


@pytest.mark.parametrize("skip_in,skip_out", [(1, 0), (0, 1), (2, 2), (4, 4)])
def test_arrays_off_a_16_byte_boundary(gpu, port, skip_in, skip_out):
    import torch

    from libtopotoolbox_gb300.api import dev

    m, n = 124, 40
    z = _dem(m, n, 3)
    src = torch.zeros(m * n + 4, device="cuda")
    dem = src[skip_in:skip_in + m * n].view(n, m)
    dem.copy_(torch.from_numpy(np.ascontiguousarray(z.T)))
    dst = torch.full((m * n + 8,), -7, dtype=torch.int32, device="cuda")
    out = dst[skip_out:skip_out + m * n].view(n, m)
    dev.identifyflats(dem, out=out)
    assert np.array_equal(out.cpu().numpy().T, port.identifyflats(z)[0])
    rest = torch.cat([dst[:skip_out], dst[skip_out + m * n:]])
    assert bool((rest == -7).all())  # nothing beside the array is written
