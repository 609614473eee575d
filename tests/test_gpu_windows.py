"""The moving windows of the tensor-core gridders and degridders: every
support they take, visibility counts around a round and a block of records,
and visibilities spread over the whole grid (sparse bins, tile edges, the
wrap of rows and columns at the grid's edge), against the CPU oracle."""

import numpy as np
import pytest

import oracle
from rang import gridder, synth

pytestmark = pytest.mark.gpu


def _kernel(supp, single):
    """A w-gridding kernel row of support `supp` whose oversampling is near 2."""
    rows = [(abs(r[1] - 2.0), i) for i, r in enumerate(gridder.kernel_table())
            if r[0] == supp and r[5] == 3 and r[6] == single]
    return min(rows)[1]


def _uv(n, nu, nv, cell, seed):
    """`n` rows whose u, v cover the grid evenly with clusters at a tile corner
    and at the grid's edge, and a few w."""
    rng = np.random.default_rng(seed)
    u, v = rng.uniform(-0.5, 0.5, n), rng.uniform(-0.5, 0.5, n)
    k = n // 4
    u[:k], v[:k] = 0.5 - rng.uniform(0, 4.0 / nu, k), rng.uniform(-2.0, 2.0, k) / nv
    u[k:2 * k], v[k:2 * k] = (32 + rng.uniform(-4, 4, k)) / nu, (32 + rng.uniform(-4, 4, k)) / nv
    uvw = np.stack([u / cell, v / cell, rng.uniform(-40.0, 40.0, n)], axis=1)
    return uvw * (synth.C_LIGHT / 1e9)  # wavelengths at 1 GHz


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("supp", [4, 5, 6, 7, 8])
@pytest.mark.parametrize("n", [1, 33, 64, 65, 1025, 40000])
def test_windows_match_the_oracle(single, supp, n):
    nx, ny, cell = 96, 64, 2e-4
    nu, nv = 216, 150  # neither a multiple of the tile
    uvw = _uv(n, nu, nv, cell, 17 * supp + n)
    freq = np.array([1e9])
    rng = np.random.default_rng(n)
    vis = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    img = rng.standard_normal((nx, ny))
    wgt = rng.uniform(0.5, 1.5, (n, 1))
    if single:
        vis, img, wgt = vis.astype(np.complex64), img.astype(np.float32), wgt.astype(np.float32)
    kw = dict(uvw=uvw, freq=freq, wgt=wgt, pixsize_x=cell, pixsize_y=cell, epsilon=1e-3,
              kernel=(_kernel(supp, single), nu, nv))
    got = gridder.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw)
    ref = oracle.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw)
    # Factors in 23 bits (single: the parity tests' bound) or float64 throughout, random
    # signs, no wide-field correction at this field.
    tol = 2e-5 if single else 1e-12
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    got = gridder.dirty2vis(dirty=img, **kw)
    ref = oracle.dirty2vis(dirty=img, **kw)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("supp", [9, 13, 16])
def test_wider_supports_far_from_the_centre(supp):
    """The tile kernels' phases: a field off the centre and long baselines, tens
    of turns each."""
    n, nx, ny, cell = 3000, 48, 40, 2e-4
    uvw = _uv(n, 216, 150, cell, supp)
    uvw[:, 2] *= 50.0
    freq = np.array([1e9])
    rng = np.random.default_rng(supp)
    vis = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    img = rng.standard_normal((nx, ny))
    kw = dict(uvw=uvw, freq=freq, pixsize_x=cell, pixsize_y=cell, epsilon=1e-9, center_x=0.03, center_y=-0.02,
              kernel=(_kernel(supp, False), 216, 150))
    # Both sides' phases in float64; the oracle's angle is rounded before it is
    # reduced, 2^-53 of 100 turns (1e-13).
    for got, ref in ((gridder.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw),
                      oracle.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw)),
                     (gridder.dirty2vis(dirty=img, **kw), oracle.dirty2vis(dirty=img, **kw))):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("supp,nu,nv,nx,ny", [(4, 4, 4, 2, 2), (4, 4, 14, 2, 6), (4, 6, 4, 2, 2), (5, 6, 6, 2, 2),
                                              (5, 8, 6, 4, 2), (6, 6, 8, 2, 4), (7, 8, 8, 4, 2), (8, 8, 10, 4, 4)])
def test_grids_smaller_than_a_window(single, supp, nu, nv, nx, ny):
    """The smallest grids an explicit kernel may have, around which a window of 8
    cells would wrap twice: the tile kernels' (with the first sizes that are not)."""
    n, cell = 300, 2e-3
    rng = np.random.default_rng(supp + nu)
    uvw = np.stack([rng.uniform(-0.5, 0.5, n) / cell, rng.uniform(-0.5, 0.5, n) / cell,
                    rng.uniform(-40.0, 40.0, n)], axis=1) * (synth.C_LIGHT / 1e9)
    vis = rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))
    img = rng.standard_normal((nx, ny))
    if single:
        vis, img = vis.astype(np.complex64), img.astype(np.float32)
    kw = dict(uvw=uvw, freq=np.array([1e9]), pixsize_x=cell, pixsize_y=cell, epsilon=1e-3,
              kernel=(_kernel(supp, single), nu, nv))
    tol = 2e-5 if single else 1e-12
    got = gridder.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw)
    ref = oracle.vis2dirty(vis=vis, npix_x=nx, npix_y=ny, **kw)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    got = gridder.dirty2vis(dirty=img, **kw)
    ref = oracle.dirty2vis(dirty=img, **kw)
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("nu,nv", [(4, 6), (8, 8)])
def test_residual_on_the_smallest_grids(nu, nv):
    import torch

    from rang import wgrid_torch

    n, cell = 300, 2e-3
    rng = np.random.default_rng(nu)
    uvw = np.stack([rng.uniform(-0.5, 0.5, n) / cell, rng.uniform(-0.5, 0.5, n) / cell,
                    rng.uniform(-40.0, 40.0, n)], axis=1) * (synth.C_LIGHT / 1e9)
    vis = (rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))).astype(np.complex64)
    img = rng.standard_normal((2, 2)).astype(np.float32)
    kw = dict(uvw=uvw, freq=np.array([1e9]), pixsize_x=cell, pixsize_y=cell, epsilon=1e-3,
              kernel=(_kernel(4, True), nu, nv))
    ref = oracle.vis2dirty(vis=vis - oracle.dirty2vis(dirty=img, **kw), npix_x=2, npix_y=2, **kw)
    plan = wgrid_torch.DevicePlan(torch.from_numpy(uvw).cuda(), kw["freq"], npix_x=2, npix_y=2, pixsize_x=cell,
                                  pixsize_y=cell, epsilon=1e-3, kernel=kw["kernel"])
    got, _ = plan.residual(torch.from_numpy(vis).cuda(), model=torch.from_numpy(img).cuda())
    assert np.abs(got.cpu().numpy() - ref).max() <= 2e-5 * np.abs(ref).max()


def test_bin_offsets_past_one_level_of_tile_sums():
    """Supports of 8 on a 4096^2 grid: 33 M bins, whose offsets are scanned in
    two levels."""
    n, nx, nu, cell = 5000, 64, 4096, 2e-4
    uvw = _uv(n, nu, nu, cell, 5)
    rng = np.random.default_rng(6)
    vis = (rng.standard_normal((n, 1)) + 1j * rng.standard_normal((n, 1))).astype(np.complex64)
    kw = dict(uvw=uvw, freq=np.array([1e9]), pixsize_x=cell, pixsize_y=cell, epsilon=1e-3,
              kernel=(_kernel(8, True), nu, nu))
    got = gridder.vis2dirty(vis=vis, npix_x=nx, npix_y=nx, **kw)
    ref = oracle.vis2dirty(vis=vis, npix_x=nx, npix_y=nx, **kw)
    assert np.abs(got - ref).max() <= 2e-5 * np.abs(ref).max()
