"""Sums of the staged reduction, of the merged backprojection and of the plane
transforms against the FP64 oracle: no further from it than the kernels that took every sample and direction on
its own, whose errors on this data are the bounds (FP64 sums of FP32 samples; adding
up to eight samples in FP32 first was 1.2 to 1.5 times as far off)."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, wrt  # noqa: F401 (loads the package)
from wrt_b200.phantom import ellipsoid_phantom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ngrid,nsr,nphi,nshift,ntheta,bound", [
    (64, 40, 33, 100, 16, 1.2e-8), (100, 17, 20, 64, 30, 8e-9)])
def test_reduction(ctx, ngrid, nsr, nphi, nshift, ntheta, bound):
    z = np.linspace(-1.0, 1.0, ngrid)[:, None, None]
    s = np.linspace(-1.0, 1.0, nsr)[None, :, None]
    r = np.random.default_rng(3)
    rays = np.clip(1.0 - z ** 2 - (s - r.uniform(-0.2, 0.2, (1, 1, nphi))) ** 2, 0.0, None)
    rays = rays * (1.0 + 0.1 * r.standard_normal((ngrid, nsr, nphi)))
    got = ctx.radon_reduction(rays, nshift, ntheta)
    err = rel_l2(got, O.reduction_forward(rays, nshift, ntheta))
    print(f"reduction {err:.2e}")
    assert err < bound


def test_backprojection(ctx):
    n, nphi, ntheta, nshift = 32, 128, 64, 256
    r = np.random.default_rng(4)
    s = np.linspace(-1.0, 1.0, nshift)[:, None, None]
    radon = np.clip(1.0 - ((s - r.uniform(-0.3, 0.3, (1, nphi, ntheta))) / 0.7) ** 2, 0.0, None)
    radon = np.ascontiguousarray(radon + 0.05 * r.standard_normal((nshift, nphi, ntheta)))
    got = ctx.radon3d_adjoint(radon, n)
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    pick = r.integers(0, n, (4000, 3))
    ref = O.adjoint_points(radon, x[pick[:, 1]], x[pick[:, 2]], x[pick[:, 0]])
    err = rel_l2(got[pick[:, 0], pick[:, 1], pick[:, 2]], ref)
    print(f"backprojection {err:.2e}")
    assert err < 6.4e-9


@pytest.mark.parametrize("sampler,n,grid,bound", [
    (O.NEAREST, 24, (16, 8, 32), 1.86e-8), (O.TRILINEAR, 12, (16, 12, 40), 4.3e-8),
    (O.TRILINEAR, 64, (32, 16, 64), 1.2e-8)])
def test_planes(ctx, sampler, n, grid, bound):
    vol = ellipsoid_phantom(n, 12, 0, dtype=np.float32).astype(np.float64)
    got = ctx.radon_grid(vol, *grid, sampler=sampler, half_extent=n)
    err = rel_l2(got, O.radon_forward(vol, *grid, sampler=sampler, half_extent=n))
    print(f"planes {n} {err:.2e}")
    assert err < bound
