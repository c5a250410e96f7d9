"""Memory budgets that the incidence lists of a graph need and its bit rows
exceed: the call keeps to the lists there and returns the same result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense(n, p, seed):
    i, j = np.triu_indices(n, 1)
    keep = np.random.default_rng(seed).random(len(i)) < p
    return i[keep].astype(np.uint32), j[keep].astype(np.uint32)


def oriented_by_id(n34, s, t, n):
    s, t = np.minimum(s, t).astype(np.int64), np.maximum(s, t).astype(np.int64)
    key = np.unique((s << 32 | t)[s != t])
    D = np.bincount(key >> 32, minlength=n).astype(np.uint32)
    O = np.concatenate([[0], np.cumsum(D)]).astype(np.uint32)
    return n34.HostGraph(n, len(key), O, D, (key & 0xffffffff).astype(np.uint32))


def pendants(n34):
    # 60 hubs, 1e6 vertices of one edge
    a, b = dense(60, 0.3, 1)
    t = np.random.default_rng(1).integers(0, 60, 1000000).astype(np.uint32)
    leaf = np.arange(60, 1000060, dtype=np.uint32)
    return n34.graph_from_edges(np.concatenate([a, leaf]), np.concatenate([b, t]))


def long_rows(n34):
    # vertex 0 points at all others: 8000 rows of 250 words
    r = np.random.default_rng(5)
    s, t = r.integers(1, 8000, (2, 40000))
    return oriented_by_id(n34, np.concatenate([s, np.zeros(7999, np.int64)]),
                          np.concatenate([t, np.arange(1, 8000)]), 8000)


@pytest.mark.parametrize("variant", ["ondemand", "direct"])
@pytest.mark.parametrize("make", [pendants, long_rows])
def test_listing_room(n34, oracle, make, variant):
    """Triangle-poor graphs, where the listing's words are the peak: a column
    word, a row word and its prefix (12 bytes) per word, the CSR and its sources
    (8m + 4n), counts and offsets per edge (12m) and per vertex (8n), and the
    triangles."""
    g = make(n34)
    o = oracle.decompose(g, quds_cap=0)
    D = g.D[: g.n].astype(np.int64)
    words = int((D * ((D + 31) // 32)).sum())
    budget = 12 * words + 20 * g.m + 12 * g.n + 12 * o.T + (1 << 19)
    d = n34.decompose(g, variant=variant, mem_budget_bytes=budget, n_quds=0)
    assert np.array_equal(d.k, o.k) and np.array_equal(d.tris, o.tris)
    assert d.result["peak_device_bytes"] <= budget


def test_death_rounds_room(n34, oracle):
    """Budgets from the memory-lean lists' need to that of the rows with every
    table, with the death rounds kept: a graph of 10 triangles and 12 words an
    edge, where the rows need more without death rounds than the lists with
    them."""
    g = n34.graph_from_edges(*dense(3000, 0.1, 2))
    o = oracle.decompose(g, quds_cap=0)
    full, low = (n34.decompose(g, variant="ondemand", flags=n34.OPT_VERIFIABLE | fl, n_quds=0)
                 .result["peak_device_bytes"] for fl in (0, n34.OPT_LEAN_MEMORY))
    assert low < full
    for i in range(33):
        budget = low + (full - low) * i // 32 + (1 << 20)
        with n34.Context(mem_budget_bytes=budget, flags=n34.OPT_VERIFIABLE) as ctx:
            ctx.upload(g)
            r = ctx.run("ondemand")
            assert r["peak_device_bytes"] <= budget
            assert np.array_equal(ctx.copy_k(r["triangle_count"]), o.k)
