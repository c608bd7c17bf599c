"""What calls leave behind: the visits per tile of the last relaxation, on
terrain where the fill's and the distances' differ, and the device memory kept
between calls, which is bounded and given back."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


@pytest.mark.parametrize("form", ["dev", "host"])
def test_pipeline_reports_its_last_relaxation(gpu, form):
    """Wide flats everywhere: the fill visits a tile some 4 times, the
    distances 13 times.  A pipeline call reports the latter, whatever the call
    before it reported."""
    torch = gpu
    from libtopotoolbox_gb300 import api
    from libtopotoolbox_gb300.api import dev

    n = 1000
    g = torch.Generator(device="cuda").manual_seed(3)
    dem = torch.rand((n, n), device="cuda", generator=g).mul_(3).round_()
    bc = torch.zeros((n, n), dtype=torch.uint8, device="cuda")
    bc[0, :] = bc[-1, :] = bc[:, 0] = bc[:, -1] = 1
    filled = dev.fillsinks(dem, bc)
    fill = api.last_rounds()
    flats = dev.identifyflats(filled)
    dev.gwdt(dev.gwdt_computecosts(flats, dem, filled)[0], flats)
    gwdt = api.last_rounds()
    assert fill > 0 and gwdt >= fill + 6, (fill, gwdt)  # told apart with +-2 between runs
    dev.fillsinks(dem, bc)
    if form == "dev":
        dev.d8_pipeline(dem, bc)
    else:
        api.d8_pipeline(np.asfortranarray(dem.cpu().numpy().T),
                        np.asfortranarray(bc.cpu().numpy().T))
    assert abs(api.last_rounds() - gwdt) <= 2, (api.last_rounds(), fill, gwdt)


def test_kept_memory_is_bounded_and_given_back(gpu):
    """`reconstruct` takes 8 bytes a pixel from the library's stream-ordered
    pool: 128 MiB stay there for the next call, of 512 MiB at most 256, and
    none after the workspace is released."""
    torch = gpu
    from libtopotoolbox_gb300 import _native
    from libtopotoolbox_gb300.api import dev

    lib = _native.lib()
    grids = {}
    for side in (4096, 8192):
        mask = torch.rand((side, side), device="cuda")
        grids[side] = (mask - 0.5, mask)
    dev.reconstruct(*grids[4096])  # the pool and the kernels exist
    lib.tt_cuda_release_workspace()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = lambda: torch.cuda.mem_get_info()[0]
    before = free()
    slack = 40 * MIB  # the workspace's tile words and granularity
    for side, low, high in ((4096, 128, 128), (8192, 0, 256)):
        dev.reconstruct(*grids[side])
        torch.cuda.synchronize()
        held = before - free()
        assert low * MIB <= held <= high * MIB + slack, (side, held / MIB)
        lib.tt_cuda_release_workspace()
        assert before - free() <= slack, (side, (before - free()) / MIB)
