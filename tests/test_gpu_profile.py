"""Plane integrals by the row-sum profiles (csrc/k_profile.cu) against the FP64
oracle, at the sizes where their rules change: the smallest edge, odd and even
edges (a sample line on a cell boundary for phis on an axis), edges around the
one from which phi and phi + pi share tables, phis on and off the axes, one
latitude (every row of a plane at one t), lattices that end inside the cube,
volumes that reach its faces, several units of t and groups of layers."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, rel_max, wrt
from wrt_b200.phantom import ellipsoid_phantom

pytestmark = pytest.mark.gpu

# the FP32 tolerance of every plane kernel's parity test
TOL_L2, TOL_MAX = 1e-5, 1e-4

CASES = [  # n, (nphi, ntheta, nshift), L, volume
    (8, (8, 4, 9), 8, "noise"), (9, (6, 3, 33), 18, "noise"),
    (9, (4, 1, 5), 9, "noise"), (24, (7, 5, 31), 24, "noise"),
    (33, (12, 5, 40), 33, "phantom"), (39, (8, 3, 32), 39, "noise"),
    (40, (8, 3, 32), 40, "noise"), (41, (10, 3, 21), 41, "phantom"),
    (41, (8, 5, 21), 20, "noise"), (64, (6, 4, 65), 128, "noise"),
    (65, (8, 3, 17), 65, "phantom"), (97, (4, 2, 9), 97, "noise"),
]


def _volume(kind, n):
    if kind == "phantom":
        return ellipsoid_phantom(n, 8, 100 + n)
    return np.random.default_rng(n).standard_normal((n, n, n)).astype(np.float32).astype(np.float64)


@pytest.fixture()
def profiles(ctx):
    wrt.set_plane_kernel_config(ctx, len(wrt.plane_kernel_configs()) - 1)
    yield ctx
    wrt.set_plane_kernel_config(ctx, -1)


@pytest.mark.parametrize("sampler", [O.TRILINEAR, O.NEAREST])
@pytest.mark.parametrize("n,grid,L,kind", CASES)
def test_matches_oracle(profiles, n, grid, L, kind, sampler):
    vol = _volume(kind, n)
    got = profiles.radon_grid(vol, *grid, sampler=sampler, half_extent=L)
    ref = O.radon_forward(vol, *grid, sampler=sampler, half_extent=L)
    assert rel_l2(got, ref) < TOL_L2
    assert rel_max(got, ref) < TOL_MAX
    again = profiles.radon_grid(vol, *grid, sampler=sampler, half_extent=L)
    assert np.array_equal(got, again)


def test_batch_and_bf16_equal_alone(profiles):
    reqs, keep = [], []
    for k, (n, grid, L, kind) in enumerate(CASES[4:9]):
        v = wrt.Volume(profiles, n, storage=wrt.STORAGE_BF16 if k % 2 else wrt.STORAGE_F32)
        v.upload(_volume(kind, n))
        g = wrt.Grid(profiles, *grid)
        out = wrt.DeviceBuffer(profiles, g.nplanes * 8)
        keep.append((v, g, out, L))
        reqs.append((v, g, out.ptr, L))
    wrt.radon_forward_batch(profiles, reqs)
    profiles.synchronize()
    batched = [out.download(np.empty(g.nplanes)) for (_, g, out, _) in keep]
    for (v, g, out, L), got in zip(keep, batched):
        wrt.radon_forward_device(profiles, v, g, out.ptr, half_extent=L)
        assert np.array_equal(got, out.download(np.empty(g.nplanes)))


def test_batch_of_both_kernels(ctx):
    # sizes on either side of the rule: the profiles run beside the staged kernel
    sizes = [(16, (16, 8, 40), 16), (40, (8, 3, 32), 40), (24, (16, 8, 32), 24),
             (65, (30, 15, 50), 65), (9, (6, 3, 33), 9), (31, (15, 9, 61), 31)]
    reqs, keep = [], []
    for n, grid, L in sizes:
        v = wrt.Volume(ctx, n)
        v.upload(_volume("noise", n))
        g = wrt.Grid(ctx, *grid)
        out = wrt.DeviceBuffer(ctx, g.nplanes * 8)
        keep.append((v, g, out))
        reqs.append((v, g, out.ptr, L))
    got = []
    for _ in range(2):
        wrt.radon_forward_batch(ctx, reqs)
        ctx.synchronize()
        got.append([out.download(np.empty(g.nplanes)) for _, g, out in keep])
    for (n, grid, L), a, b in zip(sizes, *got):
        ref = O.radon_forward(_volume("noise", n), *grid, sampler=O.TRILINEAR, half_extent=L)
        assert np.array_equal(a, b)
        assert rel_l2(a, ref.ravel()) < TOL_L2
        assert rel_max(a, ref.ravel()) < TOL_MAX


def test_tight_budget_takes_the_staged_kernel():
    vol = ellipsoid_phantom(48, 8, 5)
    with wrt.Context(0, budget_bytes=12 << 20) as c:
        got = c.radon_grid(vol, 32, 16, 64, sampler=wrt.TRILINEAR, half_extent=48)
    ref = O.radon_forward(vol, 32, 16, 64, sampler=O.TRILINEAR, half_extent=48)
    assert rel_l2(got, ref) < TOL_L2


@pytest.mark.parametrize("n,grid", [(64, (8, 16, 64)), (31, (12, 9, 70)), (45, (4, 33, 40))])
def test_nearest_in_little_memory(n, grid):
    # the tables of phis on an axis in several groups of cells
    vol = _volume("noise", n)
    with wrt.Context(0, budget_bytes=24 << 20) as c:
        got = c.radon_grid(vol, *grid, sampler=wrt.NEAREST, half_extent=n)
    ref = O.radon_forward(vol, *grid, sampler=O.NEAREST, half_extent=n)
    assert rel_l2(got, ref) < TOL_L2
    assert rel_max(got, ref) < TOL_MAX


# ---- backprojection from merged splines (csrc/k_backproj.cu): just beyond the
# sizes of the allocation-free path; odd longitudes (nothing merged), longitudes
# not a multiple of 32, odd latitudes, one voxel tile and several, few knots
# with many longitudes
@pytest.mark.parametrize("n,nphi,ntheta,nshift", [
    (5, 64, 32, 129), (20, 33, 31, 257), (17, 130, 64, 33), (33, 96, 47, 61), (48, 70, 35, 110),
])
def test_backprojection_matches_oracle(ctx, n, nphi, ntheta, nshift):
    radon = np.random.default_rng(n).standard_normal((nshift, nphi, ntheta))
    got = ctx.radon3d_adjoint(radon, n)
    assert np.array_equal(got, ctx.radon3d_adjoint(radon, n))
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    pick = np.random.default_rng(1).integers(0, n, (400, 3))
    ref = O.adjoint_points(radon, x[pick[:, 1]], x[pick[:, 2]], x[pick[:, 0]])
    assert rel_l2(got[pick[:, 0], pick[:, 1], pick[:, 2]], ref) < TOL_L2


# the spline solve takes 16 elements at a time: the shortest line, and lines of one
# element less than a whole number of groups, of a whole number and of one more
@pytest.mark.parametrize("n,nphi,ntheta,nshift", [
    (9, 300, 300, 3), (9, 98, 160, 17), (10, 96, 160, 18), (11, 96, 160, 19), (12, 96, 90, 34),
])
def test_backprojection_short_lines_match_oracle(ctx, n, nphi, ntheta, nshift):
    radon = np.random.default_rng(n).standard_normal((nshift, nphi, ntheta))
    got = ctx.radon3d_adjoint(radon, n)
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    pick = np.random.default_rng(2).integers(0, n, (200, 3))
    ref = O.adjoint_points(radon, x[pick[:, 1]], x[pick[:, 2]], x[pick[:, 0]])
    assert rel_l2(got[pick[:, 0], pick[:, 1], pick[:, 2]], ref) < TOL_L2


def test_tables_make_room():
    # the tables' buffer may fill the budget; what is allocated next still fits
    with wrt.Context(0, budget_bytes=96 << 20) as c:
        v = wrt.Volume(c, 64)
        v.upload(_volume("noise", 64))
        g = wrt.Grid(c, 32, 16, 64)
        out = wrt.DeviceBuffer(c, g.nplanes * 8)
        wrt.radon_forward_device(c, v, g, out.ptr, half_extent=64)
        c.synchronize()
        first = out.download(np.empty(g.nplanes))
        big = wrt.DeviceBuffer(c, 80 << 20)
        wrt.radon_forward_device(c, v, g, out.ptr, half_extent=64)
        c.synchronize()
        again = out.download(np.empty(g.nplanes))
        del big
    assert rel_l2(first, again) < TOL_L2
    ref = O.radon_forward(_volume("noise", 64), 32, 16, 64, sampler=O.TRILINEAR, half_extent=64)
    assert rel_l2(first, ref.ravel()) < TOL_L2
