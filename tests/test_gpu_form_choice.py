"""Which form a call takes, told from the peel's profile line, and that its result
is the same: rows where they are the less work, incidence lists on graphs whose
rows are long and nearly empty or that hold few triangles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense(n, p, seed):
    i, j = np.triu_indices(n, 1)
    keep = np.random.default_rng(seed).random(len(i)) < p
    return i[keep].astype(np.uint32), j[keep].astype(np.uint32)


def hubs(n34):
    # 400 hubs, 7e6 vertices of one edge: in-rows of 550 words, mostly empty
    a, b = dense(400, 0.3, 1)
    t = np.random.default_rng(1).integers(0, 400, 7000000).astype(np.uint32)
    leaf = np.arange(400, 7000400, dtype=np.uint32)
    return n34.graph_from_edges(np.concatenate([a, leaf]), np.concatenate([b, t]))


def long_rows(n34):
    # vertex 0 points at all others: rows of 625 words, 60 bits each
    n, r = 20000, np.random.default_rng(5)
    s, t = r.integers(1, n, (2, 30 * n))
    s, t = np.minimum(s, t), np.maximum(s, t)
    key = np.unique(np.concatenate([s << 32 | t, np.arange(1, n)])[np.concatenate([s != t, np.ones(n - 1, bool)])])
    D = np.bincount(key >> 32, minlength=n).astype(np.uint32)
    O = np.concatenate([[0], np.cumsum(D)]).astype(np.uint32)
    return n34.HostGraph(n, len(key), O, D, (key & 0xffffffff).astype(np.uint32))


def grid(n34):
    # 3100 x 3100 grid with 1 % of the diagonals, and a clique: 1.9e7 edges
    w = 3100
    i = np.arange(w * w, dtype=np.uint32).reshape(w, w)
    d = np.random.default_rng(2).random((w - 1, w - 1)) < 0.01
    a, b = dense(12, 1.0, 1)
    return n34.graph_from_edges(np.concatenate([i[:, :-1].ravel(), i[:-1].ravel(), i[:-1, :-1][d], a + w * w]),
                                np.concatenate([i[:, 1:].ravel(), i[1:].ravel(), i[1:, 1:][d], b + w * w]))


def rmat(n34):
    return n34.graph_from_edges(*n34.gen_rmat(12, 16, 1))


def rgg(n34):
    return n34.graph_from_edges(*n34.gen_rgg(200000, 5, 1))


@pytest.mark.parametrize("make,rows", [(hubs, False), (long_rows, False), (grid, False), (rmat, True), (rgg, True)])
def test_on_demand(n34, capfd, make, rows):
    g = make(n34)
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY, n_quds=0)
    capfd.readouterr()
    d = n34.decompose(g, variant="ondemand", flags=n34.OPT_PROFILE_PEEL, n_quds=0)
    line = [x for x in capfd.readouterr().err.splitlines() if x.startswith("[peel-profile]")]
    assert len(line) == 1 and ("scans=" in line[0]) == rows, line
    assert d.result["four_clique_count"] == want.result["four_clique_count"] > 0
    assert d.result["sum_te_sq"] == want.result["sum_te_sq"]
    assert np.array_equal(d.k, want.k)


@pytest.mark.parametrize("make", [hubs, long_rows, grid, rgg])
def test_direct(n34, make):
    g = make(n34)
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY, n_quds=0)
    d = n34.decompose(g, variant="direct", n_quds=0)
    assert d.result["four_clique_count"] == want.result["four_clique_count"]
    assert d.result["sum_te_sq"] == want.result["sum_te_sq"]
    assert np.array_equal(d.k, want.k)
