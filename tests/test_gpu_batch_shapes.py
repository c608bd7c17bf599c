"""Batches of DEMs of few rows or few columns, whose copies to and from the
mosaic go by runs of pixels that end inside columns and span several DEMs:
every output of every DEM equals a separate call's, output families that are
not asked for are left out, and nothing beside an output is written.

64 DEMs of 1 x 8192 pixels take 0.27 of the time of one DEM on the same canvas
(twice their pixels, and flats to cross); with a warp per DEM column 0.72.
"""
import numpy as np
import pytest

from conftest import same_float

pytestmark = pytest.mark.gpu

OUT = ("filled", "flats", "dist", "direction", "acc")
SHAPES = [(1, 1), (1, 37), (37, 1), (3, 3000), (3000, 3), (31, 29), (32, 33), (33, 32), (63, 65),
          (8, 200), (200, 8), (513, 2), (5, 5), (1, 700), (256, 4), (2, 2)]


def _grids(torch, shapes, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dems = [torch.rand((c, r), device="cuda", generator=g).mul_(30).round_() for r, c in shapes]
    bcs = []
    for d in dems:
        b = torch.zeros(d.shape, dtype=torch.uint8, device="cuda")
        b[0, :] = b[-1, :] = b[:, 0] = b[:, -1] = 1
        bcs.append(b)
    return dems, bcs


@pytest.mark.parametrize("pick", [slice(None), slice(1, 2), slice(2, 3), slice(3, 5)])
def test_thin_dems(gpu, pick, tmp_path, monkeypatch):
    torch = gpu
    monkeypatch.setenv("TT_CUDA_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    from libtopotoolbox_gb300.api import dev
    from libtopotoolbox_gb300.batch import Batch

    shapes = SHAPES[pick]
    dems, bcs = _grids(torch, shapes, 5)
    want = [dev.d8_pipeline(d, b) for d, b in zip(dems, bcs)]
    types = {"flats": torch.int32, "direction": torch.uint8}
    for families in (OUT, ("flats", "acc")):
        bufs = {k: torch.full((sum(d.numel() + 3 for d in dems),), 77, device="cuda",
                              dtype=types.get(k, torch.float32)) for k in families}
        out = {k: [] for k in families}
        at = 0
        for d in dems:  # three words between any two outputs
            for k in families:
                out[k].append(bufs[k][at:at + d.numel()].view(d.shape))
            at += d.numel() + 3
        bt = Batch(shapes)
        for _ in range(2):  # the plain run, the graph's replay
            bt.run(dems, bcs, outputs=out)
        bt.close()
        at = 0
        for k, d in enumerate(dems):
            for f in families:
                assert same_float(out[f][k].cpu().numpy(), want[k][f].cpu().numpy()), (shapes[k], f)
                assert bool((bufs[f][at + d.numel():at + d.numel() + 3] == 77).all())
            at += d.numel() + 3


def test_one_row_dems_are_not_slow(gpu, tmp_path, monkeypatch):
    torch = gpu
    monkeypatch.setenv("TT_CUDA_AUTOTUNE_CACHE", str(tmp_path / "tune.json"))
    from libtopotoolbox_gb300.batch import Batch

    def time_of(shapes):
        dems, bcs = _grids(torch, shapes, 9)
        bt = Batch(shapes)
        out = bt.run(dems, bcs)
        took = []
        for _ in range(7):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            bt.run(dems, bcs, outputs=out)
            b.record()
            torch.cuda.synchronize()
            took.append(a.elapsed_time(b))
        info = bt.info()
        bt.close()
        return min(took), info["canvas_rows"], info["canvas_cols"]

    thin, rows, cols = time_of([(1, 8192)] * 64)
    whole, _, _ = time_of([(rows - 2, cols - 2)])  # twice the pixels, on the same canvas
    assert thin < 0.45 * whole, (thin, whole)
