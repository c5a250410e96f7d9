"""CSRs whose orientation is not acyclic: triangles and cliques are those with
a source at every step (u -> v, u -> w, v -> w), so three vertices that form a
directed cycle are no triangle and no part of a clique. The bit rows would take a
cycle above a common source for one, and do not tell u -> v from v -> u."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def csr(n34, edges):
    e = np.unique(np.array([u << 32 | v for u, v in edges], np.int64))
    n = int(max(max(u, v) for u, v in edges)) + 1
    D = np.bincount(e >> 32, minlength=n).astype(np.uint32)
    O = np.concatenate([[0], np.cumsum(D)]).astype(np.uint32)
    return n34.HostGraph(n, len(e), O, D, (e & 0xffffffff).astype(np.uint32))


def same_as_oracle(n34, oracle, g):
    o = oracle.decompose(g, quds_cap=1 << 20)
    for variant in ("ondemand", "direct"):
        d = n34.decompose(g, variant=variant, n_quds=o.Q)
        assert (d.result["triangle_count"], d.result["four_clique_count"]) == (o.T, o.Q)
        assert np.array_equal(d.tris, o.tris) and np.array_equal(d.k, o.k)
        if variant == "direct":
            assert np.array_equal(d.quds, o.quds)
    assert o.Q > 0


@pytest.mark.parametrize("cycles", [1, 4, 5])
def test_cycles_above_a_source(n34, oracle, cycles):
    edges = list(itertools.combinations(range(12), 2))
    for i in range(cycles):
        u, v, w, x = range(12 + 4 * i, 16 + 4 * i)
        edges += [(u, v), (u, w), (u, x), (v, w), (w, x), (x, v)]
    same_as_oracle(n34, oracle, csr(n34, edges))


@pytest.mark.parametrize("seed", [1, 2])
def test_edges_in_both_directions(n34, oracle, seed):
    """Pairs u <-> v below one w, apart from the cliques."""
    r = np.random.default_rng(seed)
    edges = list(itertools.combinations(range(10), 2))
    for i in range(int(r.integers(1, 6))):
        u, v, w = (10 + 3 * i + r.permutation(3)).tolist()
        edges += [(u, v), (v, u), (u, w), (v, w)]
    same_as_oracle(n34, oracle, csr(n34, edges))
