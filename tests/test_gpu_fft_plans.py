"""The Fourier transforms' plans, which calls of one size share: passes in
flight at the same time on several threads and streams (lengths with a large
prime factor, whose transforms need a work area), against the same passes one
after the other; and how many plans calls with ever other w ranges leave."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle
from rang import core, gridder, synth

pytestmark = pytest.mark.gpu


def _kernel(supp, single):
    rows = [(abs(r[1] - 2.0), i) for i, r in enumerate(gridder.kernel_table())
            if r[0] == supp and r[5] == 3 and r[6] == single]
    return min(rows)[1]


def _case(seed, n, cell, wmax, single):
    rng = np.random.default_rng(seed)
    uvw = np.stack([rng.uniform(-0.45, 0.45, n) / cell, rng.uniform(-0.45, 0.45, n) / cell,
                    rng.uniform(-wmax, wmax, n)], axis=1) * (synth.C_LIGHT / 1e9)
    vis = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    return uvw, vis.astype(np.complex64) if single else vis


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("n", [256, 1018])  # 1018 = 2 x 509
def test_threads_share_plans_but_not_work_areas(single, n):
    cell, freq = 2e-4, np.array([1e9])
    kw = dict(freq=freq, pixsize_x=cell, pixsize_y=cell, epsilon=1e-3, kernel=(_kernel(4, single), n, n))
    cases = [_case(s, 2000, cell, 40.0, single) for s in range(6)]
    imgs = [np.random.default_rng(s).standard_normal((n // 4 * 2, n // 4 * 2)).astype(np.float32 if single else np.float64)
            for s in range(6)]

    def both(k):
        uvw, vis = cases[k]
        return (gridder.vis2dirty(uvw=uvw, vis=vis, npix_x=n // 4 * 2, npix_y=n // 4 * 2, **kw),
                gridder.dirty2vis(uvw=uvw, dirty=imgs[k], **kw))

    want = [both(k) for k in range(6)]
    with ThreadPoolExecutor(6) as pool:
        for _ in range(4):
            for k, (d, v) in enumerate(pool.map(both, range(6))):
                assert np.array_equal(d, want[k][0]) and np.array_equal(v, want[k][1])


def test_streams_share_plans_but_not_work_areas():
    import torch

    from rang import wgrid_torch
    from rang.fista import gaussian_lowpass

    cell, n = 2e-4, 1018
    kw = dict(npix_x=n // 4 * 2, npix_y=n // 4 * 2, pixsize_x=cell, pixsize_y=cell, epsilon=1e-3, kernel=(_kernel(4, True), n, n))
    plans, vis, imgs = [], [], []
    for k in range(4):
        uvw, v = _case(k, 20000, cell, 40.0, True)
        plans.append(wgrid_torch.DevicePlan(torch.from_numpy(uvw).cuda(), np.array([1e9]), **kw))
        vis.append(torch.from_numpy(v).cuda())
        imgs.append(torch.randn(n // 4 * 2, n // 4 * 2, device="cuda"))
    want = [(p.grid(v), p.degrid(i)) for p, v, i in zip(plans, vis, imgs)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in plans]
    for _ in range(5):
        got = []
        for p, v, i, s in zip(plans, vis, imgs, streams):
            with torch.cuda.stream(s):
                got.append((p.grid(v), p.degrid(i)))
        torch.cuda.synchronize()
        for (a, b), (c, d) in zip(got, want):
            assert torch.equal(a, c) and torch.equal(b, d)
    low = [gaussian_lowpass(i, 3.0) for i in imgs]
    torch.cuda.synchronize()
    for _ in range(5):
        got = []
        for i, s in zip(imgs, streams):
            with torch.cuda.stream(s):
                got.append(gaussian_lowpass(i, 3.0))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, low))
    for p in plans:
        p.close()
    assert core.extension().wgridder_release_cached() == 0


@pytest.mark.parametrize("single", [True, False])
def test_plane_counts_share_plans(single):
    """Passes of 4 to 70 planes, whose transforms run together, over sizes rounded
    up: each against the CPU oracle."""
    ext = core.extension()
    assert ext.wgridder_release_cached() == 0
    kept = ext.wgridder_fft_plans()  # of captured graphs, which stay
    cell, n, freq = 2e-3, 32, np.array([1e9])
    planes, sizes = set(), set()
    tol = 2e-5 if single else 1e-12
    for k in range(67):
        uvw, vis = _case(k, 200, cell, 1.0, single)
        uvw[0, 2], uvw[1, 2] = 0.0, (k + 0.5) * 480.0 * synth.C_LIGHT / 1e9
        kw = dict(uvw=uvw, freq=freq, pixsize_x=cell, pixsize_y=cell, epsilon=1e-3, kernel=(_kernel(4, single), 64, 64))
        got = gridder.vis2dirty(vis=vis, npix_x=n, npix_y=n, **kw)
        ref = oracle.vis2dirty(vis=vis, npix_x=n, npix_y=n, **kw)
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
        img = np.random.default_rng(k).standard_normal((n, n)).astype(np.float32 if single else np.float64)
        got = gridder.dirty2vis(dirty=img, **kw)
        ref = oracle.dirty2vis(dirty=img, **kw)
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
        p = int(gridder.plan(vis=vis, npix_x=n, npix_y=n, single=single, **kw)["nplanes"])
        planes.add(p)
        step = max(1, 1 << max(0, (p - 1).bit_length() - 3))
        sizes.add(-(-p // step) * step)
    assert len(planes) >= 60 and min(planes) <= 5 and max(planes) >= 64
    assert ext.wgridder_fft_plans() - kept <= 2 * len(sizes) <= 40
    assert ext.wgridder_release_cached() == 0 and ext.wgridder_fft_plans() == kept


def test_plans_are_bounded():
    ext = core.extension()
    assert ext.wgridder_release_cached() == 0
    kept = ext.wgridder_fft_plans()
    for k in range(40):  # two sizes a call
        uvw, vis = _case(k, 50, 2e-3, 1.0, True)
        gridder.vis2dirty(uvw=uvw, vis=vis, freq=np.array([1e9]), npix_x=16, npix_y=16, pixsize_x=2e-3,
                          pixsize_y=2e-3, epsilon=1e-3, kernel=(_kernel(4, True), 32 + 2 * k, 34 + 2 * k))
    assert kept < ext.wgridder_fft_plans() <= 64
    assert ext.wgridder_release_cached() == 0 and ext.wgridder_fft_plans() == kept


def test_captured_passes_keep_their_plans():
    """A pass captured into a CUDA graph replays after release_cached and after
    more plans than are kept."""
    import torch

    from rang import wgrid_torch

    ext = core.extension()
    uvw, vis = _case(0, 20000, 2e-4, 40.0, True)
    v, img = torch.from_numpy(vis).cuda(), torch.randn(128, 128, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        plan = wgrid_torch.DevicePlan(torch.from_numpy(uvw).cuda(), np.array([1e9]), npix_x=128, npix_y=128,
                                      pixsize_x=2e-4, pixsize_y=2e-4, epsilon=1e-4)
        want = plan.grid(v), plan.degrid(img)
        torch.cuda.synchronize()
        got = torch.empty_like(want[0]), torch.empty_like(want[1])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            plan.grid(v, out=got[0])
            plan.degrid(img, out=got[1])
    torch.cuda.synchronize()
    before = ext.wgridder_fft_plans()
    test_plans_are_bounded()
    assert ext.wgridder_release_cached() == 0 and 2 <= ext.wgridder_fft_plans() <= before
    for _ in range(2):
        for t in got:
            t.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    del graph
    plan.close()
