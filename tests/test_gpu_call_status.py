"""Status of whole pipeline calls, which is read once after the last stage:
the iteration cap is reported by the synchronous, deferred and host forms,
the calls after it are exact again, and the visits per tile are reported."""
import numpy as np
import pytest

from conftest import same_float

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (33, 31), (300, 257), (1100, 900)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("form", ["dev", "deferred", "host"])
def test_pipeline_status(gpu, port, form, shape):
    torch = gpu
    import contextlib

    from libtopotoolbox_gb300 import _native, api, dems
    from libtopotoolbox_gb300.api import dev

    dem = dems.pcg4d_dem(shape, 31)
    bc = dems.border_bc(shape)
    d_dem, d_bc = (torch.from_numpy(np.ascontiguousarray(a.T)).cuda() for a in (dem, bc))

    def call():
        if form == "host":
            return api.d8_pipeline(dem, bc)
        with dev.deferred() if form == "deferred" else contextlib.nullcontext():
            o = dev.d8_pipeline(d_dem, d_bc)
        return {k: v.cpu().numpy().T for k, v in o.items()}

    lib = _native.lib()
    if shape[0] > 40:  # enough tiles for two visits a tile to fall short
        lib.tt_cuda_set_max_rounds(1)
        try:
            with pytest.raises(_native.TTCudaError) as e:
                call()
            assert e.value.status == 4
        finally:
            lib.tt_cuda_set_max_rounds(0)
    got, want = call(), port.pipeline(dem, bc)
    for k in ("filled", "flats", "dist", "direction", "acc"):
        assert same_float(got[k], want[k]), (form, shape, k)
    if form == "dev" and shape[0] > 40:
        dev.fillsinks(d_dem, d_bc)
        dev.d8_pipeline(d_dem, d_bc)
        flats = dev.identifyflats(torch.from_numpy(np.ascontiguousarray(want["filled"].T)).cuda())
        costs, _ = dev.gwdt_computecosts(flats, d_dem, torch.from_numpy(
            np.ascontiguousarray(want["filled"].T)).cuda())
        seen = api.last_rounds()
        dev.gwdt(costs, flats)
        assert abs(seen - api.last_rounds()) <= 2, "visits per tile of the last relaxation"
