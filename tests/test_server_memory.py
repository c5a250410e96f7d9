"""Device memory of a serving pass against what it was admitted with, from the
high-water mark of the device's memory pool."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

USED_MEM_CURRENT, USED_MEM_HIGH = 7, 8
SLACK = 4 << 20


class Pool:
    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, self.pool = C.c_int(), C.c_void_p()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def get(self, attr):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def reset(self):
        v = C.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_MEM_HIGH, C.byref(v)) == 0


def pendants(n34, hubs, leaves):
    r = np.random.default_rng(1)
    i, j = np.triu_indices(hubs, 1)
    keep = r.random(len(i)) < 0.3
    leaf = np.arange(hubs, hubs + leaves)
    return n34.graph_from_edges(np.concatenate([i[keep], leaf]).astype(np.uint32),
                                np.concatenate([j[keep], r.integers(0, hubs, leaves)]).astype(np.uint32))


@pytest.mark.parametrize("hubs,leaves", [(60, 1000000), (300, 1500000)])
def test_triangle_poor_pass_stays_within_its_admission(n34, hubs, leaves):
    """Edges that lie on no triangle cost the lists no more than the estimate's 40
    bytes (44 with the vertices of degree 1, which it leaves out); the rows take
    72 to 100."""
    g = pendants(n34, hubs, leaves)
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_HOST_LOOP, n_quds=0)
    est = n34.server_estimate(g, 1 << 40)["ondemand_bytes"]
    pool = Pool()
    with n34.Server(workers=1, mem_budget_bytes=8 << 30, route=n34.ROUTE_ONDEMAND) as srv:
        before = pool.get(USED_MEM_CURRENT)
        pool.reset()
        rid = srv.submit(g)
        info = srv.wait(rid, timeout_ms=120000)
        assert np.array_equal(srv.copy_k(rid, info["triangle_count"]), want.k)
        used = pool.get(USED_MEM_HIGH) - before
    assert used <= max(est + SLACK, want.result["peak_device_bytes"]) + (1 << 20), (used, est)


@pytest.mark.parametrize("case", [("rmat", 8, 8, 2), ("rmat", 14, 16, 1), ("rgg", 50000, 30, 1), ("ws", 30000, 10, 4)])
def test_triangle_rich_pass_keeps_the_rows(n34, capfd, case):
    s, t = (n34.gen_ws(case[1], case[2], 0.1, case[3]) if case[0] == "ws" else
            getattr(n34, "gen_" + case[0])(*case[1:]))
    g = n34.graph_from_edges(s, t)
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY, n_quds=0)
    capfd.readouterr()
    with n34.Server(workers=1, mem_budget_bytes=8 << 30, route=n34.ROUTE_ONDEMAND,
                    flags=n34.OPT_PROFILE_PEEL) as srv:
        rid = srv.submit(g)
        info = srv.wait(rid, timeout_ms=120000)
        assert np.array_equal(srv.copy_k(rid, info["triangle_count"]), want.k)
    line = [x for x in capfd.readouterr().err.splitlines() if x.startswith("[peel-profile]")]
    assert len(line) == 1 and "scans=" in line[0], line
