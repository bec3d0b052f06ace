"""Two threads, each with a context of its own, run the same kernels at sizes with
different amounts of shared memory: a kernel's limit belongs to the kernel, and
neither thread may lower it under the other's launch."""
import threading

import numpy as np
import pytest

from conftest import wrt

pytestmark = pytest.mark.gpu

SIZES = {  # for each thread
    "reduction": [(100, 150, 2, 16, 4), (128, 200, 2, 16, 4)],  # 130 and 218 KB
    "adjoint": [(4, 640, 20, 24), (4, 16, 210, 200)],           # 14 and 200 KB
}


@pytest.mark.parametrize("op", ["reduction", "adjoint"])
def test_two_contexts_on_two_threads(op):
    errors, results = [], [[], []]

    def work(k):
        try:
            rng = np.random.default_rng(k)
            with wrt.Context(0) as c:
                if op == "reduction":
                    ngrid, nsr, nphi, nshift, ntheta = SIZES[op][k]
                    data = rng.standard_normal((ngrid, nsr, nphi))
                    g = wrt.Grid(c, nphi, ntheta, nshift)
                    nout = g.nplanes
                else:
                    ngrid, nphi, ntheta, nshift = SIZES[op][k]
                    data = rng.standard_normal((nshift, nphi, ntheta))
                    g = wrt.Grid(c, nphi, ntheta, nshift)
                    nout = ngrid ** 3
                src, out = wrt.DeviceBuffer(c, data.nbytes), wrt.DeviceBuffer(c, 8 * nout)
                src.upload(data)
                for i in range(2000):
                    if op == "reduction":
                        wrt.radon_reduction_device(c, src.ptr, ngrid, nsr, g, out.ptr)
                    else:
                        wrt.radon3d_adjoint_device(c, src.ptr, g, ngrid, out.ptr)
                    if i % 100 == 0:
                        results[k].append(out.download(np.empty(nout)))
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors, errors
    for r in results:
        assert all(np.array_equal(r[0], x) for x in r)
