"""Passes that take their w planes in several groups (as where they do not all
fit in memory): every kernel family, direction and the fused residual against
the CPU oracle, with footprints across the groups' edges; and the retry after a
buffer of the work space could not be had."""

import numpy as np
import pytest

import oracle
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


@pytest.mark.parametrize("chunks", [1, 3])
@pytest.mark.parametrize("planes", [1, 2, 5])
@pytest.mark.parametrize("single,supp,nu,nv", [(True, 4, 84, 80), (True, 7, 90, 100), (True, 8, 84, 96),
                                               (False, 4, 84, 80), (False, 8, 90, 100), (False, 11, 96, 84)])
def test_plane_groups_match_the_oracle(limits, monkeypatch, single, supp, nu, nv, planes, chunks):
    monkeypatch.setenv("RANG_WGRIDDER_ROW_CHUNKS", str(chunks))
    vis, img, kw = _case(supp, nu, nv, single)
    total = gridder.plan(vis=vis, npix_x=NX, npix_y=NY, single=single, **kw)["nplanes"]
    assert total > planes + supp
    groups = -(-total // planes)
    tol = 2e-5 if single else 1e-12  # the parity tests' bound; float64 sums of a few thousand terms
    limits(0, planes, 0)
    got, n = _launches(lambda: gridder.vis2dirty(vis=vis, npix_x=NX, npix_y=NY, **kw))
    assert n["grid"] == groups * chunks
    ref = oracle.vis2dirty(vis=vis, npix_x=NX, npix_y=NY, **kw)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    got, n = _launches(lambda: gridder.dirty2vis(dirty=img, **kw))
    assert n["degrid"] == groups * chunks
    ref = oracle.dirty2vis(dirty=img, **kw)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("planes", [1, 3])
@pytest.mark.parametrize("single,supp", [(True, 5), (True, 8), (False, 6)])
def test_residual_in_plane_groups(limits, single, supp, planes):
    import torch

    from rang import wgrid_torch

    vis, img, kw = _case(supp, 84, 90, single)
    wgt = kw.pop("wgt")
    bare = oracle.dirty2vis(dirty=img, **kw)
    ref = oracle.vis2dirty(vis=(vis - bare).astype(vis.dtype), npix_x=NX, npix_y=NY, wgt=wgt, **kw)
    misfit = (wgt.astype(np.float64) * np.abs(vis.astype(np.complex128) - bare) ** 2).sum()
    w = torch.from_numpy(wgt).cuda()
    plan = wgrid_torch.DevicePlan(torch.from_numpy(kw.pop("uvw")).cuda(), kw.pop("freq"), npix_x=NX, npix_y=NY, wgt=w,
                                  single=single, **kw)
    limits(0, planes, 0)
    got, q = plan.residual(torch.from_numpy(vis).cuda(), w, model=torch.from_numpy(img).cuda())
    tol = 4e-5 if single else 1e-12
    assert np.abs(got.cpu().numpy() - ref).max() <= tol * np.abs(ref).max()
    assert abs(float(q) - misfit) <= tol * misfit


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
