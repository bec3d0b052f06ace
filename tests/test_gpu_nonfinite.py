"""Values that are no numbers: what does not touch them is as without them."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, wrt

pytestmark = pytest.mark.gpu

TOL_L2 = 1e-5  # the FP32 tolerance of every parity test


def _volume(n, at):
    v = np.random.default_rng(n).standard_normal((n, n, n)).astype(np.float32)
    for x in at:
        v[x] = np.nan
    return v


VOLUMES = [(40, [(20, 21, 5)]), (40, [(0, 0, 7)]), (33, [(3, 30, 16), (12, 2, 31)])]
GRID = (20, 16, 60)


@pytest.mark.parametrize("sampler", [O.TRILINEAR, O.NEAREST])
@pytest.mark.parametrize("n,at", VOLUMES)
def test_planes(ctx, sampler, n, at):
    v = _volume(n, at).astype(np.float64)
    ref = O.radon_forward(v, *GRID, sampler=sampler, half_extent=n)
    clear = np.isfinite(ref)
    assert 0.2 < clear.mean() < 1.0
    got = ctx.radon_grid(v, *GRID, sampler=sampler, half_extent=n)
    assert rel_l2(got[clear], ref[clear]) < TOL_L2


def test_planes_batched_and_served_equal_alone(ctx):
    n, at = VOLUMES[0]
    vols = [_volume(n, a) for a in (at, [], [(0, 0, 7)])]
    alone = []
    for v in vols:
        vol = wrt.Volume(ctx, n)
        vol.upload(v)
        g = wrt.Grid(ctx, *GRID)
        out = wrt.DeviceBuffer(ctx, g.nplanes * 8)
        wrt.radon_forward_device(ctx, vol, g, out.ptr, half_extent=n)
        alone.append((vol, g, out, out.download(np.empty(g.nplanes))))
    wrt.radon_forward_batch(ctx, [(v, g, o.ptr, n) for v, g, o, _ in alone])
    for _, g, out, x in alone:
        assert np.array_equal(x, out.download(np.empty(g.nplanes)), equal_nan=True)
    with wrt.Server(0, budget_bytes=1 << 30) as srv:
        outs = [np.zeros((GRID[2], GRID[0], GRID[1])) for _ in vols]
        ids = [srv.submit_forward(v, *GRID, o, half_extent=n) for v, o in zip(vols, outs)]
        for i in ids:
            assert srv.wait(i, 120_000).status == 0
    for (_, _, _, x), o in zip(alone, outs):
        assert np.array_equal(x, o.ravel(), equal_nan=True)


@pytest.mark.parametrize("n,nslices", [(40, 40), (33, 33), (40, 7)])  # vector loads, scalar, layer pairs
def test_rays(ctx, n, nslices):
    v = _volume(n, [(0, 0, 3), (0, 0, n - 2)]).astype(np.float64)
    ref = O.ray_forward(v, nslices, 41, 18)
    clear = np.isfinite(ref)
    assert 0.2 < clear.mean() < 1.0
    got = ctx.ray_grid(v, nslices, 41, 18)
    assert rel_l2(got[clear], ref[clear]) < TOL_L2


@pytest.mark.parametrize("n,nphi,ntheta,nshift,at", [
    (20, 96, 47, 61, [(30, 7, 20)]), (20, 33, 31, 257, [(0, 4, 9), (200, 4, 9), (40, 5, 9)]),
])
def test_backprojection(ctx, n, nphi, ntheta, nshift, at):
    # a line with such a value has none that is a number; voxels beyond its ends are free of it
    radon = np.random.default_rng(n).standard_normal((nshift, nphi, ntheta))
    for x in at:
        radon[x] = np.nan
    got = ctx.radon3d_adjoint(radon, n)
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    iz, ix, iy = (a.ravel() for a in np.meshgrid(np.arange(n), np.arange(n), np.arange(n), indexing="ij"))
    phi, theta, _, _ = O.radon_grid(nphi, ntheta, nshift)
    clear = np.ones(n ** 3, bool)
    for _, ip, it in at:
        s = (np.sin(theta[it]) * (np.cos(phi[ip]) * x[ix] + np.sin(phi[ip]) * x[iy])
             + np.cos(theta[it]) * x[iz])
        clear &= np.abs(s) > 1.0
    assert 0.005 < clear.mean() < 1.0
    assert np.isnan(got.ravel()[~clear]).all()
    clean = radon.copy()
    clean[:, [a[1] for a in at], [a[2] for a in at]] = 0.0
    pick = np.flatnonzero(clear)
    ref = O.adjoint_points(clean, x[ix[pick]], x[iy[pick]], x[iz[pick]])
    assert rel_l2(got.ravel()[pick], ref) < TOL_L2
