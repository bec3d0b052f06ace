"""A server's budget bounds its device memory, the tables that make requests faster
among it, and a request that has no room beside them is still served."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_l2, wrt
from wrt_b200.phantom import ellipsoid_phantom

pytestmark = pytest.mark.gpu

WAIT_MS = 120_000


def test_device_memory_stays_within_the_budget(ctx):
    import torch

    vol = ellipsoid_phantom(48, 6, 1).astype(np.float32)
    ctx.radon_grid(vol.astype(np.float64), 16, 8, 40, sampler=wrt.TRILINEAR)  # modules loaded
    budget, slack = 4 << 30, 256 << 20  # slack: batch tables, graphs, streams
    for slots in (2, 8):
        before = torch.cuda.mem_get_info()[0]
        with wrt.Server(0, budget_bytes=budget, max_inflight=slots) as srv:
            out = np.zeros((40, 16, 8))
            assert srv.wait(srv.submit_forward(vol, 16, 8, 40, out), WAIT_MS).status == 0
            assert before - torch.cuda.mem_get_info()[0] <= budget + slack
            assert srv.stats().bytes_peak <= budget


def test_a_request_without_room_beside_the_tables(ctx):
    # 160 MB: 20 MB of tables for each of two launches; 8 x 250^3 bytes need 125 MB
    budget, n = 160 << 20, 250
    radon = np.random.default_rng(3).standard_normal((20, 12, 6))
    vols = [ellipsoid_phantom(24, 6, k).astype(np.float32) for k in range(6)]
    small = np.random.default_rng(4).standard_normal((61, 96, 47))
    direct = []
    for v in vols:
        vol = wrt.Volume(ctx, 24)
        vol.upload(v)
        g = wrt.Grid(ctx, 16, 8, 32)
        buf = wrt.DeviceBuffer(ctx, g.nplanes * 8)
        wrt.radon_forward_device(ctx, vol, g, buf.ptr, half_extent=24)
        direct.append(buf.download(np.empty(g.nplanes)))
    with wrt.Server(0, budget_bytes=budget) as srv:
        outs = [np.zeros((32, 16, 8)) for _ in vols]
        big = [np.zeros((n, n, n)) for _ in range(2)]
        adj = [np.zeros((10, 10, 10)) for _ in range(2)]
        ids = []
        for k in range(2):  # small ones before, between and after the large ones
            ids += [srv.submit_forward(v, 16, 8, 32, o, half_extent=24)
                    for v, o in zip(vols[3 * k:3 * k + 3], outs[3 * k:3 * k + 3])]
            ids.append(srv.submit_adjoint(radon, n, big[k]))
            ids.append(srv.submit_adjoint(small, 10, adj[k]))
        for i in ids:
            assert srv.wait(i, WAIT_MS).status == 0
        st = srv.stats()
        assert st.bytes_peak <= budget and st.failed == 0
    for o, d in zip(outs, direct):
        assert np.array_equal(o.ravel(), d)
    assert np.array_equal(adj[0], adj[1])
    assert rel_l2(adj[0], O.adjoint_forward(small, 10)) < 1e-5
    assert np.array_equal(big[0], big[1])
    x = -1.0 + (2.0 * np.arange(n) + 1.0) / n
    pick = np.random.default_rng(1).integers(0, n, (300, 3))
    ref = O.adjoint_points(radon, x[pick[:, 1]], x[pick[:, 2]], x[pick[:, 0]])
    assert rel_l2(big[0][pick[:, 0], pick[:, 1], pick[:, 2]], ref) < 1e-5
