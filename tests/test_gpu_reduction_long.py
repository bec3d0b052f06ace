"""The ray-to-Radon reduction of many layers and few offsets (long lines of the staged
kernel), and of few layers and many offsets, against the FP64 oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, wrt  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ngrid,nshift_ray,nphi,nshift,ntheta", [
    (256, 60, 4, 65, 9), (600, 30, 5, 33, 12), (2000, 8, 3, 65, 7), (3, 2000, 4, 64, 9),
])
def test_long_lines_match_oracle(ctx, ngrid, nshift_ray, nphi, nshift, ntheta):
    z = np.linspace(-1.0, 1.0, ngrid)[:, None, None]
    s = np.linspace(-1.0, 1.0, nshift_ray)[None, :, None]
    r = np.random.default_rng(ngrid)
    rays = (1.5 - z ** 2 - s ** 2) * (1.0 + 0.1 * r.standard_normal((ngrid, nshift_ray, nphi)))
    got = ctx.radon_reduction(rays, nshift, ntheta)
    assert rel_l2(got, O.reduction_forward(rays, nshift, ntheta)) < 1e-5
