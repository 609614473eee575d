"""Copies of pageable host arrays through the pinned buffers: sizes around
the pieces and the limit for staging, several threads at once, and after the
buffers were given back, against the same passes on device tensors."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from cases import meerkat_like
from rang import core, gridder

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvis", [(4 << 17) - 1, 4 << 17, (4 << 17) + 1, (5 << 17) + 77, 3 << 20])
@pytest.mark.parametrize("threads", [1, 3])
def test_host_arrays_give_the_device_tensors_results(nvis, threads):
    import torch

    from rang import wgrid_torch

    uvw, freq = meerkat_like(nant=24, ntime=4, nchan=1, seed=3)
    rows = np.resize(uvw, (nvis, 3)) * np.linspace(0.9, 1.0, nvis)[:, None]
    rng = np.random.default_rng(nvis)
    vis = (rng.standard_normal((nvis, 1)) + 1j * rng.standard_normal((nvis, 1))).astype(np.complex64)  # 8 bytes each
    img = rng.standard_normal((128, 96)).astype(np.float32)
    kw = dict(pixsize_x=4e-5, pixsize_y=4e-5, epsilon=1e-4)
    t = torch.from_numpy(rows).cuda()
    p = wgrid_torch.DevicePlan(t, freq, npix_x=128, npix_y=96, **kw)
    want_vis = p.degrid(torch.from_numpy(img).cuda()).cpu().numpy()
    p.close()
    v = torch.from_numpy(vis).cuda()
    p = wgrid_torch.DevicePlan(t, freq, vis=v, npix_x=128, npix_y=96, **kw)
    want_img = p.grid(v, scanned=True).cpu().numpy()
    p.close()

    def both(_):
        d = gridder.vis2dirty(uvw=rows, freq=freq, vis=vis, npix_x=128, npix_y=96, **kw)
        return d, gridder.dirty2vis(uvw=rows, freq=freq, dirty=img, **kw)

    with ThreadPoolExecutor(threads) as pool:
        for d, y in pool.map(both, range(2 * threads)):
            assert np.array_equal(d, want_img) and np.array_equal(y, want_vis)
    assert core.extension().wgridder_release_cached() == 0
    d, y = both(0)
    assert np.array_equal(d, want_img) and np.array_equal(y, want_vis)


def test_copies_without_pinned_buffers_are_the_drivers():
    uvw, freq = meerkat_like(nant=24, ntime=4, nchan=1, seed=3)
    nvis = (5 << 17) + 77
    rows = np.resize(uvw, (nvis, 3)) * np.linspace(0.9, 1.0, nvis)[:, None]
    rng = np.random.default_rng(1)
    vis = (rng.standard_normal((nvis, 1)) + 1j * rng.standard_normal((nvis, 1))).astype(np.complex64)
    img = rng.standard_normal((128, 96)).astype(np.float32)
    kw = dict(uvw=rows, freq=freq, pixsize_x=4e-5, pixsize_y=4e-5, epsilon=1e-4)
    ext = core.extension()

    def both():
        return gridder.vis2dirty(vis=vis, npix_x=128, npix_y=96, **kw), gridder.dirty2vis(dirty=img, **kw)

    want = both()
    assert ext.wgridder_release_cached() == 0
    ext.wgridder_test_limits(1, 0, 0)
    try:
        got = both()
    finally:
        ext.wgridder_test_limits(0, 0, 0)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
