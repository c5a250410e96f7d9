"""The direct variant's clique list from the listing's bit matrices against the
oracle and against brute force, at the sizes where its words and its owner masks
have edges, on both sides of the choice of the peel and down to the memory where
the incidence lists take over. All results are integers and must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ALL = 1 << 28


def dense(n, p, seed):
    i, j = np.triu_indices(n, 1)
    keep = np.random.default_rng(seed).random(len(i)) < p
    return i[keep].astype(np.uint32), j[keep].astype(np.uint32)


def same_as_oracle(d, o):
    r = d.result
    assert (r["triangle_count"], r["four_clique_count"]) == (o.T, o.Q)
    assert np.array_equal(d.tris, o.tris) and np.array_equal(d.k, o.k)
    assert np.array_equal(d.quds, o.quds)


# out-degrees around the 32-bit words of a row, under labels in every direction
# against the degree order: fourth vertices below and above the source
@pytest.mark.parametrize("n", [4, 5, 31, 33, 34, 64, 66, 97])
@pytest.mark.parametrize("p", [1.0, 0.6])
@pytest.mark.parametrize("labels", ["same", "reversed", "shuffled"])
def test_row_words(n34, oracle, n, p, labels):
    s, t = dense(n, p, n)
    name = {"same": np.arange(n), "reversed": np.arange(n)[::-1],
            "shuffled": np.random.default_rng(n).permutation(n)}[labels].astype(np.uint32)
    g = n34.graph_from_edges(name[s], name[t])
    same_as_oracle(n34.decompose(g, variant="direct", n_quds=ALL), oracle.decompose(g, quds_cap=ALL))


# an acyclic orientation that follows no order of the labels
@pytest.mark.parametrize("seed", [1, 2])
def test_other_orientations(n34, seed):
    n = 130
    s, t = dense(n, 0.4, seed)
    name = np.random.default_rng(seed).permutation(n).astype(np.uint32)
    s, t = name[s], name[t]
    order = np.argsort(s.astype(np.int64) * 1000 + t, kind="stable")
    s, t = s[order], t[order]
    D = np.bincount(s, minlength=n).astype(np.uint32)
    O = np.concatenate([[0], np.cumsum(D)]).astype(np.uint32)
    g = n34.HostGraph(n, len(s), O, D, t.copy())
    d = n34.decompose(g, variant="direct", n_quds=ALL)
    # triangles are {vertex of the tail, source, head} of edges a = u -> w, b = u -> v
    of = {}
    for i, (a, b, _) in enumerate(d.tris):
        of[frozenset((int(s[a]), int(t[a]), int(t[b])))] = i
    adj = np.zeros((n, n), bool)
    adj[s, t] = adj[t, s] = True
    want = []
    for key, i in of.items():
        u, v, w = key
        for x in np.flatnonzero(adj[u] & adj[v] & adj[w]):
            ids = sorted([of[frozenset((u, v, x))], of[frozenset((u, w, x))], of[frozenset((v, w, x))]])
            if i < ids[0]:
                want.append((i, x, *ids))
    want = np.array([(w[0], *w[2:]) for w in sorted(want)], np.uint32)
    assert np.array_equal(d.quds, want)


# both sides of the clique count that decides between the two peels
@pytest.mark.parametrize("n", [50000, 70000])
def test_both_peels(n34, oracle, n):
    s, t = n34.gen_rgg(n, 30, 5)
    g = n34.graph_from_edges(s, t)
    d = n34.decompose(g, variant="direct", n_quds=ALL)
    o = n34.decompose(g, variant="ondemand")
    assert (d.result["four_clique_count"] > 1 << 24) == (n == 70000)
    for key in ("four_clique_count", "k_max", "k_avg", "peeling_iterations", "unpeeled_count"):
        assert d.result[key] == o.result[key], key
    assert np.array_equal(d.k, o.k)
    assert np.array_equal(d.quds, oracle.decompose(g, quds_cap=ALL).quds)


# budgets down to a refusal: with few cliques the incidence lists need less than
# the rows and take over, with many the clique list decides
@pytest.mark.parametrize("case,forms", [(("rgg", 30000, 30), 1), (("ws", 100000, 8, 0.3), 2)])
def test_budgets(n34, oracle, case, forms):
    g = n34.graph_from_edges(*getattr(n34, "gen_" + case[0])(*case[1:], 7))
    o = oracle.decompose(g, quds_cap=ALL)
    full = n34.decompose(g, variant="direct").result["peak_device_bytes"]
    peaks, refused = set(), 0
    for i in range(10, 0, -1):
        budget = full * i // 10 + (1 << 20)
        try:
            d = n34.decompose(g, variant="direct", n_quds=ALL, mem_budget_bytes=budget)
        except n34.Nucleus34Error as e:
            assert e.code == n34.E_OOM_BUDGET
            refused += 1
            continue
        assert not refused  # less memory never helps
        same_as_oracle(d, o)
        assert d.result["peak_device_bytes"] <= budget
        peaks.add(d.result["peak_device_bytes"])
    assert refused and len(peaks) >= forms
