"""The retry after a buffer of a pass's work space could not be had."""

import numpy as np
import pytest

from rang import core, gridder, synth

pytestmark = pytest.mark.gpu

CELL, NX, NY = 2e-3, 40, 36


def _kernel(supp, single):
    rows = [(abs(r[1] - 2.0), i) for i, r in enumerate(gridder.kernel_table())
            if r[0] == supp and r[5] == 3 and r[6] == single]
    return min(rows)[1]


@pytest.fixture
def limits():
    ext = core.extension()
    yield ext.wgridder_test_limits
    ext.wgridder_test_limits(0, 0, 0)


def _launches(f):
    """f's result and the launches of each stage that it took."""
    ext = core.extension()
    ext.wgridder_profile(1)
    ext.wgridder_profile_read()
    out = f()
    n = {k: v[0] for k, v in ext.wgridder_profile_read().items()}
    ext.wgridder_profile(0)
    return out, n


def _case(supp, nu, nv, single, n=3000):
    rng = np.random.default_rng(100 * supp + nu)
    uvw = np.stack([rng.uniform(-0.5, 0.5, n) / CELL, rng.uniform(-0.5, 0.5, n) / CELL,
                    rng.uniform(-3000.0, 3000.0, n)], axis=1) * (synth.C_LIGHT / 1e9)
    vis = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    wgt = rng.uniform(0.5, 1.5, (n, 1))
    img = rng.standard_normal((NX, NY))
    if single:
        vis, wgt, img = vis.astype(np.complex64), wgt.astype(np.float32), img.astype(np.float32)
    kw = dict(uvw=uvw, freq=np.array([1e9]), wgt=wgt, pixsize_x=CELL, pixsize_y=CELL, epsilon=1e-3, center_x=0.01,
              center_y=-0.02, kernel=(_kernel(supp, single), nu, nv))
    return vis, img, kw


@pytest.mark.parametrize("buffer", [1, 2, 3])
def test_a_buffer_that_cannot_be_had(limits, buffer):
    """The pass asks how much fits, with what it held given back, and gives the
    same results."""
    vis, img, kw = _case(4, 84, 80, True)
    want = gridder.vis2dirty(vis=vis, npix_x=NX, npix_y=NY, **kw), gridder.dirty2vis(dirty=img, **kw)
    limits(0, 0, buffer)
    got, n = _launches(lambda: gridder.vis2dirty(vis=vis, npix_x=NX, npix_y=NY, **kw))
    assert n["grid"] == 1 and np.array_equal(got, want[0])
    limits(0, 0, buffer)
    got, n = _launches(lambda: gridder.dirty2vis(dirty=img, **kw))
    assert n["degrid"] == 1 and np.array_equal(got, want[1])


def test_the_retry_counts_what_it_gave_back(limits):
    """Little memory left: the planes fit at once, though not beside the buffers
    of the attempt that failed."""
    import torch

    from rang import wgrid_torch

    vis, _, kw = _case(4, 4096, 4096, True, n=200)
    wgt, uvw, freq = kw.pop("wgt"), kw.pop("uvw"), kw.pop("freq")
    kw["pixsize_x"] = kw["pixsize_y"] = 2e-5  # a few planes
    plan = wgrid_torch.DevicePlan(torch.from_numpy(uvw).cuda(), freq, npix_x=2048, npix_y=2048,
                                  wgt=torch.from_numpy(wgt).cuda(), **kw)
    planes = plan.info["nplanes"]
    v, w = torch.from_numpy(vis).cuda(), torch.from_numpy(wgt).cuda()
    want = plan.grid(v, w)
    torch.cuda.synchronize()
    assert core.extension().wgridder_release_cached() == 0
    torch.cuda.empty_cache()
    cell, grid, cols = 8, 4096 * 4096, 2048 * 4096
    need = planes * (16 * grid + cell * cols) + cell * grid + 4 * 2048 * 2048
    free, _ = torch.cuda.mem_get_info()
    room = int(need / 0.85) * 2  # half the free memory is the budget
    assert free > room
    held = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        limits(0, 0, 3)  # after the grids, two thirds of the need
        got, n = _launches(lambda: plan.grid(v, w))
    finally:
        del held
        torch.cuda.empty_cache()
    assert n["grid"] == 1 and torch.equal(got, want)
    plan.close()
    assert core.extension().wgridder_release_cached() == 0
