"""Directions where a strip's drops fall below 2^-100, from which on the
quotients by sqrt(2) are divisions, somewhere along its columns: in the first,
in the last, in one of a warp's lanes only.  Whole numbers, equal to the oracle's
(src/flow_routing.c:15-76)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 9), (56, 64), (57, 131), (120, 65), (128, 200), (301, 66)])
@pytest.mark.parametrize("faint", ["first", "last", "one", "half"])
def test_directions(gpu, port, shape, faint):
    from libtopotoolbox_gb300 import api

    m, n = shape
    rng = np.random.default_rng(m + n)
    scale = np.ones(shape)
    if faint == "first":
        scale[:, 0] = 2.0 ** -120
    elif faint == "last":
        scale[:, -1] = 2.0 ** -140
    elif faint == "one":
        scale[m // 2, n // 2] = 2.0 ** -130
    else:
        scale[:, n // 2:] = 2.0 ** -110
    z = np.asfortranarray((rng.integers(0, 9, shape) * scale).astype(np.float32))
    d = np.asfortranarray((rng.integers(0, 9, shape) * scale).astype(np.float32))
    flats = np.asfortranarray((rng.random(shape) < 0.4).astype(np.int32))
    for order in (0, 1):
        _, want = port.flow_routing_d8_carve(z, d, flats, order)
        _, got = api.flow_routing_d8_carve(z, d, flats, order)
        assert np.array_equal(got, want)
