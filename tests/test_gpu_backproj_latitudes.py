"""Backprojection of many latitudes with few shifts: up to where the latitudes of the
merged splines' build fit shared memory (csrc/k_backproj.cu), and beyond, where the
direct kernel serves."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nphi,ntheta,nshift", [(8, 16, 3980, 9), (8, 16, 3990, 9), (8, 16, 4500, 9)])
def test_many_latitudes(ctx, n, nphi, ntheta, nshift):
    radon = np.random.default_rng(n).standard_normal((nshift, nphi, ntheta))
    got = ctx.radon3d_adjoint(radon, n)
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    pick = np.random.default_rng(2).integers(0, n, (60, 3))
    ref = O.adjoint_points(radon, x[pick[:, 1]], x[pick[:, 2]], x[pick[:, 0]])
    assert rel_l2(got[pick[:, 0], pick[:, 1], pick[:, 2]], ref) < 1e-5
