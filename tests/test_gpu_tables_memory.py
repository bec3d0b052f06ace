"""The working memory that only makes calls faster (csrc/api.cu, tables_get): it makes
room for what is allocated next and is taken again once that is freed."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, wrt

pytestmark = pytest.mark.gpu


def _planes(c):
    v = wrt.Volume(c, 64)
    x = np.random.default_rng(64).standard_normal((64, 64, 64)).astype(np.float32)
    v.upload(x)
    g = wrt.Grid(c, 32, 16, 64)
    out = wrt.DeviceBuffer(c, g.nplanes * 8)
    ref = O.radon_forward(x.astype(np.float64), 32, 16, 64, sampler=O.TRILINEAR, half_extent=64)
    return lambda: wrt.radon_forward_device(c, v, g, out.ptr, half_extent=64), out, ref


def _adjoint(c):
    radon = np.random.default_rng(5).standard_normal((110, 70, 35))
    src = wrt.DeviceBuffer(c, radon.nbytes)
    src.upload(radon)
    g = wrt.Grid(c, 70, 35, 110)
    out = wrt.DeviceBuffer(c, 8 * 48 ** 3)
    return (lambda: wrt.radon3d_adjoint_device(c, src.ptr, g, 48, out.ptr), out,
            O.adjoint_forward(radon, 48))


@pytest.mark.parametrize("op", [_planes, _adjoint])
@pytest.mark.parametrize("left", [24, 64])  # MB beside the other buffer
def test_tables_come_back(op, left):
    with wrt.Context(0, budget_bytes=512 << 20) as c:
        call, out, ref = op(c)
        call()
        c.synchronize()
        first, full = out.download(np.empty(out.nbytes // 8)), c.bytes_in_use
        big = wrt.DeviceBuffer(c, (512 - left) << 20)
        call()
        c.synchronize()
        tight = out.download(np.empty(out.nbytes // 8))
        assert c.bytes_in_use <= 512 << 20
        big.close()
        call()
        c.synchronize()
        # nothing allocated on the way stays behind but what the staged and direct kernels keep
        assert c.bytes_in_use >= full
        assert np.array_equal(first, out.download(np.empty(out.nbytes // 8)))
    assert rel_l2(first, ref.ravel()) < 1e-5
    assert rel_l2(tight, ref.ravel()) < 1e-5


def test_batch_equals_alone_in_a_tight_budget():
    # the large requests' tables do not fit, the small ones' do, whatever else is in the batch
    sizes = [(64, (32, 16, 64)), (24, (16, 8, 40)), (16, (8, 4, 9)), (72, (30, 15, 70)), (30, (16, 8, 50))]
    with wrt.Context(0, budget_bytes=28 << 20) as c:
        reqs, keep = [], []
        for n, grid in sizes:
            v = wrt.Volume(c, n)
            v.upload(np.random.default_rng(n).standard_normal((n, n, n)).astype(np.float32))
            g = wrt.Grid(c, *grid)
            out = wrt.DeviceBuffer(c, g.nplanes * 8)
            keep.append((v, g, out))
            reqs.append((v, g, out.ptr, n))
        wrt.radon_forward_batch(c, reqs)
        batched = [out.download(np.empty(g.nplanes)) for _, g, out in keep]
        for (n, _), (v, g, out), got in zip(sizes, keep, batched):
            wrt.radon_forward_device(c, v, g, out.ptr, half_extent=n)
            assert np.array_equal(got, out.download(np.empty(g.nplanes))), n


def test_nearest_bits_do_not_depend_on_the_memory():
    n, grid = 45, (8, 33, 64)
    vol = np.random.default_rng(n).standard_normal((n, n, n))
    got = []
    for mb in (0, 48, 32, 24, 20):  # all of them room for the least
        with wrt.Context(0, budget_bytes=mb << 20) as c:
            got.append(c.radon_grid(vol, *grid, sampler=wrt.NEAREST, half_extent=n))
    for x in got[1:]:
        assert np.array_equal(got[0], x)
