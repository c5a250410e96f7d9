"""The bit-matrix form of the on-demand variant (support count and peel) against
the oracle and against the list form (NUCLEUS34_OPT_LEAN_MEMORY), at the sizes
where its words, batches and claims have edges. All results are integers and
must be equal."""
import numpy as np
import pytest

import graphs

pytestmark = pytest.mark.gpu


def dense(n, p, seed, offset=0):
    i, j = np.triu_indices(n, 1)
    keep = np.random.default_rng(seed).random(len(i)) < p
    return (i[keep] + offset).astype(np.uint32), (j[keep] + offset).astype(np.uint32)


def same_as_oracle(d, o):
    r = d.result
    assert (r["triangle_count"], r["four_clique_count"]) == (o.T, o.Q)
    assert np.array_equal(d.tris, o.tris) and np.array_equal(d.k, o.k)
    if o.Q:
        assert (r["k_max"], r["k_avg"], r["unpeeled_count"]) == (o.k_max, o.k_avg, 0)


# out-degrees around the 32-bit words of a row: one, two and three words, full
# and with one bit over; a lone triangle; cliques sharing and not sharing sources
@pytest.mark.parametrize("n", [3, 4, 31, 32, 33, 34, 64, 65, 66, 97])
@pytest.mark.parametrize("p", [1.0, 0.7])
def test_row_words(n34, oracle, n, p):
    g = n34.graph_from_edges(*dense(n, p, n))
    same_as_oracle(n34.decompose(g, variant="ondemand"), oracle.decompose(g, quds_cap=0))


# frontiers from fewer triangles than warps to many per warp, with ordering
@pytest.mark.parametrize("case", [("rmat", 11, 20, 2), ("rgg", 40000, 40, 3), ("ws", 30000, 20, 4)])
@pytest.mark.parametrize("shift", [1, 12, 0xffffffff])
def test_frontier_order_and_claims(n34, oracle, case, shift):
    s, t = (n34.gen_ws(case[1], case[2], 0.1, case[3]) if case[0] == "ws" else
            getattr(n34, "gen_" + case[0])(*case[1:]))
    g = n34.graph_from_edges(s, t)
    o = oracle.decompose(g, quds_cap=0)
    with n34.Context() as ctx:
        ctx.upload(g)
        ctx.set_tune({"sort_shift": shift})
        r = ctx.run("ondemand")
        assert np.array_equal(ctx.copy_k(r["triangle_count"]), o.k)
        assert r["four_clique_count"] == o.Q and r["k_max"] == o.k_max and r["k_avg"] == o.k_avg


# frontiers put in id order: graphs of 2^24 triangles and more, with the
# threshold at its lowest, at its default and off
def test_ordered_frontiers_match_the_list_form(n34):
    g = n34.graph_from_edges(*n34.gen_rgg(200003, 32, 9))
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY)
    assert want.result["triangle_count"] >= 2 ** 24
    with n34.Context() as ctx:
        ctx.upload(g)
        for shift in (31, 12, 0xffffffff):
            ctx.set_tune({"sort_shift": shift})
            r = ctx.run("ondemand")
            assert r["peeling_iterations"] == want.result["peeling_iterations"]
            assert np.array_equal(ctx.copy_k(r["triangle_count"]), want.k)


# an acyclic orientation that is not by degree: every source's list is long
@pytest.mark.parametrize("seed", [1, 2])
def test_other_orientations(n34, seed):
    s, t = dense(160, 0.35, seed)
    order = np.argsort(s.astype(np.int64) * 1000 + t, kind="stable")
    s, t = s[order], t[order]
    n = 160
    D = np.bincount(s, minlength=n).astype(np.uint32)
    O = np.concatenate([[0], np.cumsum(D)]).astype(np.uint32)
    g = n34.HostGraph(n, len(s), O, D, t.copy())
    want = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY)
    got = n34.decompose(g, variant="ondemand")
    for key in ("triangle_count", "four_clique_count", "k_max", "k_avg", "sum_te_sq", "peeling_iterations"):
        assert got.result[key] == want.result[key], key
    assert np.array_equal(got.k, want.k) and np.array_equal(got.tris, want.tris)


# budgets from the list form's need to the bit form's with all its tables: the
# optional tables go first, then the whole form
def test_budgets(n34, oracle):
    g = n34.graph_from_edges(*n34.gen_rgg(60000, 36, 7))
    o = oracle.decompose(g, quds_cap=0)
    full = n34.decompose(g, variant="ondemand").result["peak_device_bytes"]
    lean = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY).result["peak_device_bytes"]
    assert lean < full
    peaks = set()
    for i in range(9):
        budget = int(lean + (full - lean) * i / 8) + (1 << 20)
        d = n34.decompose(g, variant="ondemand", mem_budget_bytes=budget)
        same_as_oracle(d, o)
        assert d.result["peak_device_bytes"] <= budget
        peaks.add(d.result["peak_device_bytes"])
    assert len(peaks) >= 3


def test_rounds_and_work_measure_match_the_list_form(n34):
    g = n34.graph_from_edges(*graphs.union(graphs.clique(40), graphs.clique(7, offset=38), dense(90, 0.5, 5, 60)))
    a = n34.decompose(g, variant="ondemand").result
    b = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY).result
    for key in ("peeling_iterations", "sum_te_sq", "four_clique_count", "k_max"):
        assert a[key] == b[key], key


# in-rows on both sides of two words per edge (with and without live counts)
@pytest.mark.parametrize("hubs", [1, 40, 200])
def test_in_row_widths(n34, oracle, hubs):
    n, rng = 400, np.random.default_rng(hubs)
    hub = np.arange(hubs, dtype=np.uint32) + n
    i, j = dense(n, 0.08, hubs)
    k = rng.random((n, hubs)) < 0.5
    s = np.concatenate([i, np.repeat(np.arange(n, dtype=np.uint32), hubs)[k.ravel()]])
    t = np.concatenate([j, np.tile(hub, n)[k.ravel()]])
    a, b = dense(hubs, 0.5, 3, offset=n)
    g = n34.graph_from_edges(np.concatenate([s, a]), np.concatenate([t, b]))
    same_as_oracle(n34.decompose(g, variant="ondemand"), oracle.decompose(g, quds_cap=0))
