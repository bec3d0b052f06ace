"""Rays of the z-slices through a volume of more than 2^31 nodes: a linear function,
whose samples are those of the reference's interpolation in closed form, against
their sums along the rays."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2, wrt

pytestmark = pytest.mark.gpu


def _sampled(x, n):
    """Where the reference's interpolation takes a coordinate to be: cell by truncation,
    fraction by fmod (radon_grid/src/interp.c:32-53), which differ on a node."""
    h = 2.0 / (n - 1)
    i = np.trunc((x + 1.0) / h)
    c = np.fmod(x + 1.0, h) / h
    last = i == n - 1
    return -1.0 + (np.where(last, i - 1, i) + np.where(last, 1.0, c)) * h


@pytest.mark.parametrize("n,nslices", [(1300, 1300), (1301, 7)])  # rows in 16-byte loads, and not
def test_columns_beyond_two_to_the_31(n, nslices):
    import torch

    nshift, nphi = 9, 5
    c = (1.0, 0.5, -0.25, 0.125)
    x = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda").float()
    f = c[0] + c[1] * x[:, None, None] + c[2] * x[None, :, None] + c[3] * x[None, None, :]
    torch.cuda.synchronize()
    with wrt.Context(0) as ctx:
        vol = wrt.Volume(ctx, n)
        ctx.check(wrt.lib().wrt_volume_upload_device(vol.handle, C.c_void_p(f.data_ptr())), "upload")
        ctx.synchronize()
        del f
        torch.cuda.empty_cache()
        out = wrt.DeviceBuffer(ctx, 8 * nslices * nshift * nphi)
        wrt.ray_forward_device(ctx, vol, nslices, nshift, nphi, out.ptr)
        got = out.download(np.empty((nslices, nshift, nphi)))
    s = -1.0 + np.arange(nshift) * (2.0 / (nshift - 1))
    z = -1.0 + np.arange(nslices) * (2.0 / (nslices - 1))
    delta = (2.0 / (n - 1)) / 2.0
    k = np.arange(-2 * n, 2 * n + 1)
    ref = np.empty_like(got)
    for ip in range(nphi):
        phi = 2 * np.pi / nphi * ip
        # the reference's order of operations decides which samples lie inside
        # (ray_grid/src/integral.c:32-44); rays along a face are left out below
        px = s[:, None] * np.cos(phi) + (delta * np.cos(phi + np.pi / 2)) * k
        py = s[:, None] * np.sin(phi) + (delta * np.sin(phi + np.pi / 2)) * k
        inside = (np.abs(px) <= 1.0) & (np.abs(py) <= 1.0)
        layer = (inside * (c[0] + c[1] * _sampled(px, n) + c[2] * _sampled(py, n))).sum(1)
        ref[:, :, ip] = delta * (layer[None] + c[3] * _sampled(z, n)[:, None] * inside.sum(1)[None])
    assert rel_l2(got[:, 1:-1], ref[:, 1:-1]) < 1e-5
