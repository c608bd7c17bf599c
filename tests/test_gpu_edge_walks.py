"""List-order edge sweeps by how many values an edge waits for: none, one,
two (an exchange), a few and more than a walker reads ahead, along a chain
whose every node has that many in-edges, with side branches out of it, in
topological order, reversed and shuffled; also with NaN, infinite and signed
zero start values.  The (|, &) sweep is exact.  The (+, *) sweep takes the
oracle's FP64 operations in the same order and is rounded once to float32,
so it is within one float32 rounding (2^-24, 6e-8 relative) of the FP64
sweep; 1e-6 leaves room for contraction in the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEN = 70


def _chain(indeg, order, seed):
    """Node k of the chain (0 .. LEN - 1) gets indeg in-edges: one from node
    k - 1, the others from leaves; every third node also feeds a sink."""
    rng = np.random.default_rng(seed)
    src, tgt, leaf = [], [], LEN + 1
    for k in range(LEN):
        feeders = []
        for _ in range(indeg - (k > 0)):
            feeders.append(leaf)
            leaf += 1
        if k > 0:
            feeders.insert(int(rng.integers(0, len(feeders) + 1)), k - 1)
        for u in feeders:
            src.append(u)
            tgt.append(k)
        if k % 3 == 0 and k:
            src.append(k - 1)
            tgt.append(LEN)  # the sink: k - 1 has two out-edges
    src, tgt = np.array(src, np.int64), np.array(tgt, np.int64)
    if order == "reversed":
        src, tgt = src[::-1].copy(), tgt[::-1].copy()
    elif order == "shuffled":
        p = rng.permutation(len(src))
        src, tgt = src[p], tgt[p]
    return src, tgt, leaf, rng


@pytest.mark.parametrize("order", ["topological", "reversed", "shuffled"])
@pytest.mark.parametrize("indeg", [1, 2, 3, 8, 9, 40])
def test_edge_walks(gpu, port, indeg, order):
    from libtopotoolbox_gb300 import api

    src, tgt, n, rng = _chain(indeg, order, 7 * indeg)
    f = rng.uniform(0.2, 1.0, len(src)).astype(np.float32)
    start = rng.uniform(-1.0, 1.0, n).astype(np.float32)
    for special in (False, True):
        if special:
            start[rng.integers(0, n, 3)] = [np.nan, np.inf, -0.0]
        got = api.traverse_down_f32_add_mul(start, f, src, tgt)
        want = port.traverse_down_f32_add_mul(start, f, src, tgt, f64=True)
        fine = np.isfinite(want)
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(got[~fine & ~np.isnan(want)], want[~fine & ~np.isnan(want)])
        size = np.abs(want[fine])
        assert np.all(np.abs(got[fine] - want[fine]) <= 1e-6 * size + 1e-30)
        assert np.array_equal(got, api.traverse_down_f32_add_mul(start, f, src, tgt),
                              equal_nan=True), "run to run"
    words = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    words[rng.random(n) < 0.2] = 0xFFFFFFFF
    mask = rng.integers(0, 2**32, len(src), dtype=np.uint64).astype(np.uint32)
    mask[rng.random(len(src)) < 0.5] = 0xFFFFFFFF
    assert np.array_equal(api.traverse_down_u32_or_and(words, mask, src, tgt),
                          port.traverse_u32_or_and(words, mask, src, tgt))
    assert np.array_equal(api.traverse_up_u32_or_and(words, mask, src, tgt),
                          port.traverse_u32_or_and(words, mask, src, tgt, up=True))
