"""List-order edge sweeps through a hub: many edges into one node, then many
out of it, each of which waits for all of the first.  Degrees around the
values a walker reads ahead (8) and the edges it stacks (24); the (+, *) sweep
within 1e-6 of the oracle's FP64 sweep (one float32 rounding is 6e-8), the
(|, &) sweep exact.

The last edge into the hub completes all the edges out of it.  They have to be
spread over the chip: 1500 edges in and out take 4 ms when a further launch sums
them and took 730 ms when that one walker did.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hub(indeg, outdeg):
    """Sources 1 .. indeg into node 0, out of it to indeg + 1 .. ."""
    src = np.concatenate([np.arange(1, indeg + 1), np.zeros(outdeg, np.int64)])
    tgt = np.concatenate([np.zeros(indeg, np.int64), indeg + 1 + np.arange(outdeg)])
    return src, tgt, indeg + outdeg + 1


@pytest.mark.parametrize("indeg", [7, 8, 9, 16, 17, 100])
@pytest.mark.parametrize("outdeg", [1, 24, 26, 90])
def test_hub(gpu, port, indeg, outdeg):
    from libtopotoolbox_gb300 import api

    src, tgt, n = _hub(indeg, outdeg)
    rng = np.random.default_rng(indeg * 100 + outdeg)
    f = rng.uniform(0.2, 1.0, len(src)).astype(np.float32)
    start = rng.uniform(0.0, 1.0, n).astype(np.float32)
    words = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    mask = rng.integers(0, 2**32, len(src), dtype=np.uint64).astype(np.uint32)
    for p in (np.arange(len(src)), rng.permutation(len(src))):
        s, t = src[p], tgt[p]
        got = api.traverse_down_f32_add_mul(start, f, s, t)
        want = port.traverse_down_f32_add_mul(start, f, s, t, f64=True)
        assert np.all(np.abs(got - want) <= 1e-6 * np.abs(want))
        assert np.array_equal(api.traverse_down_u32_or_and(words, mask, s, t),
                              port.traverse_u32_or_and(words, mask, s, t))
        assert np.array_equal(api.traverse_up_u32_or_and(words, mask, s, t),
                              port.traverse_u32_or_and(words, mask, s, t, up=True))


def test_hub_is_not_walked_by_one(gpu):
    torch = gpu
    from libtopotoolbox_gb300.api import dev

    src, tgt, n = _hub(1500, 1500)
    src, tgt = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda()
    f = torch.full((len(src),), 0.5, device="cuda")
    took = []
    for _ in range(3):
        out = torch.ones(n, device="cuda")
        torch.cuda.synchronize()
        t = time.perf_counter()
        dev.traverse_down_f32_add_mul(out, f, src, tgt)
        torch.cuda.synchronize()
        took.append(time.perf_counter() - t)
    assert float(out[0]) == 751.0 and float(out[-1]) == 1 + 0.5 * 751.0
    assert min(took) < 0.06, took
