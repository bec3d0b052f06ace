"""Rows of the row-sum profiles (csrc/k_profile.cu) whose t is the border of two
units: an odd number of latitudes has theta = pi/2, where all rows of a plane have
one t, and at these shift counts that is a border for part of the planes."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, rel_max, wrt

pytestmark = pytest.mark.gpu

# the FP32 tolerance of every plane kernel's parity test
TOL_L2, TOL_MAX = 1e-5, 1e-4


@pytest.mark.parametrize("sampler,n,grid", [
    (O.NEAREST, 64, (10, 3, 65)), (O.NEAREST, 64, (7, 1, 129)), (O.NEAREST, 128, (6, 1, 129)),
    (O.TRILINEAR, 64, (10, 3, 127)), (O.TRILINEAR, 128, (6, 1, 255)), (O.TRILINEAR, 96, (5, 1, 191)),
])
def test_rows_on_the_border_of_two_units(ctx, sampler, n, grid):
    vol = np.random.default_rng(n).standard_normal((n, n, n)).astype(np.float32).astype(np.float64)
    wrt.set_plane_kernel_config(ctx, len(wrt.plane_kernel_configs()) - 1)
    try:
        got = ctx.radon_grid(vol, *grid, sampler=sampler, half_extent=n)
        assert np.array_equal(got, ctx.radon_grid(vol, *grid, sampler=sampler, half_extent=n))
    finally:
        wrt.set_plane_kernel_config(ctx, -1)
    ref = O.radon_forward(vol, *grid, sampler=sampler, half_extent=n)
    assert rel_l2(got, ref) < TOL_L2
    assert rel_max(got, ref) < TOL_MAX
