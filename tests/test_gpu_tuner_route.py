"""The autotuner chooses among the staged kernel's tiles; which kernel a request takes
stays a matter of its sizes, so results of other requests keep their bits."""
import numpy as np
import pytest

from conftest import wrt

pytestmark = pytest.mark.gpu


def test_tuning_does_not_move_other_requests():
    with wrt.Context(0) as c:
        runs = []
        for n, grid in ((48, (32, 16, 64)), (30, (8, 4, 20)), (24, (16, 8, 32))):
            v = wrt.Volume(c, n)
            v.upload(np.random.default_rng(n).standard_normal((n, n, n)).astype(np.float32))
            g = wrt.Grid(c, *grid)
            out = wrt.DeviceBuffer(c, g.nplanes * 8)
            runs.append((v, g, out, n))

        def results():
            got = []
            for v, g, out, n in runs:
                wrt.radon_forward_device(c, v, g, out.ptr, half_extent=n)
                got.append(out.download(np.empty(g.nplanes)))
            return got

        before = results()
        for v, g, out, n in runs[:2]:  # one that takes the row-sum profiles, one that does not
            best, ms = wrt.tune_plane_kernel(c, v, g, out.ptr, half_extent=n)
            assert wrt.plane_kernel_configs()[best][0] > 0 and ms > 0
            for x, y in zip(before, results()):
                assert np.array_equal(x, y)
