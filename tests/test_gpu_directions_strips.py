"""D8 carve directions at the edges of the strips a warp walks along and at
near ties of slopes: neighbours one and two floats apart across the diagonal
and drops whose diagonal quotients round to the same float, subnormal drops,
infinities and NaN, arrays off a 16-byte boundary.  Directions are whole
numbers and must equal the oracle's (src/flow_routing.c:15-76).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SQ2 = np.float32(np.sqrt(2.0))


def _near_ties(rng, scale):
    x = np.float32(rng.uniform(1, 4) * scale)
    near = [x, (x / SQ2).astype(np.float32)]
    for v in list(near):
        for _ in range(2):
            v = np.nextafter(v, np.float32(0))
            near.append(v)
    return np.array(near, np.float32)


def _grids(m, n, scale):
    """Centres at 0 between neighbours -d; flats on pixels that have an
    elevation, so that no direction can lead around a cycle."""
    rng = np.random.default_rng(m * 1000 + n)
    near = np.concatenate([[np.float32(0)], -_near_ties(rng, scale)])
    z = rng.choice(near, (m, n), p=[0.3] + [0.7 / (len(near) - 1)] * (len(near) - 1))
    d = rng.choice(near, (m, n)) + np.float32(0)
    pick = rng.random((m, n))
    z[pick < 0.01], z[(pick > 0.02) & (pick < 0.025)] = np.nan, np.inf
    d[(pick > 0.03) & (pick < 0.05)] = np.inf
    flats = ((rng.random((m, n)) < 0.4) & ~np.isnan(z)).astype(np.int32)
    return [np.asfortranarray(a) for a in (z.astype(np.float32), d.astype(np.float32), flats)]


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 9), (3, 7), (4, 8), (119, 9), (120, 8), (121, 17),
                                 (124, 3), (240, 24), (244, 25), (1201, 300)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -127, 2.0 ** -148, 2.0 ** 126])
def test_near_ties(gpu, port, m, n, order, scale):
    from libtopotoolbox_gb300 import api

    z, d, flats = _grids(m, n, scale)
    _, want = port.flow_routing_d8_carve(z, d, flats, order)
    _, got = api.flow_routing_d8_carve(z, d, flats, order)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("skips", [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0), (0, 0, 0, 1),
                                   (0, 0, 0, 4)])
def test_arrays_off_their_boundaries(gpu, port, skips):
    import torch

    from libtopotoolbox_gb300 import _native as native
    from libtopotoolbox_gb300.api import dev

    m, n = 124, 40
    z, d, flats = _grids(m, n, 1.0)
    _, want = port.flow_routing_d8_carve(z, d, flats, 0)

    def at(skip, a):
        buf = torch.zeros(m * n + 8, dtype=torch.from_numpy(a).dtype, device="cuda")
        view = buf[skip:skip + m * n].view(n, m)
        view.copy_(torch.from_numpy(np.ascontiguousarray(a.T)))
        return buf, view

    (_, zt), (_, dt), (_, ft) = at(skips[0], z), at(skips[1], d), at(skips[2], flats)
    buf, out = at(skips[3], np.full((m, n), 77, np.uint8))
    buf[:skips[3]] = 77
    buf[skips[3] + m * n:] = 77
    dims, keep = native.dims_arg((m, n))
    native.check(native.lib().tt_cuda_flow_routing_d8_carve_dev(
        None, dev._p(out), dev._p(zt), dev._p(dt), dev._p(ft), dims, 0, dev._stream()),
        "flow_routing_d8_carve_dev")
    assert np.array_equal(out.cpu().numpy().T, want)
    assert bool((buf[:skips[3]] == 77).all() and (buf[skips[3] + m * n:] == 77).all())
