"""Frontiers put in id order by the one-launch peel on graphs below 2^24 triangles,
where a pinned sort_shift asks for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the ordering bitmap at triangle counts that end inside a word, on skewed and even
# graphs: pinned thresholds act below 2^24 triangles too
@pytest.mark.parametrize("case", [("rmat", 13, 16, 2), ("rgg", 40001, 40, 3), ("rgg", 30011, 20, 5), ("ws", 30000, 20, 4)])
@pytest.mark.parametrize("shift", [31, 20])
def test_ordered_small_frontiers(n34, oracle, capfd, case, shift):
    s, t = (n34.gen_ws(case[1], case[2], 0.1, case[3]) if case[0] == "ws" else
            getattr(n34, "gen_" + case[0])(*case[1:]))
    g = n34.graph_from_edges(s, t)
    o = oracle.decompose(g, quds_cap=0)
    with n34.Context(flags=n34.OPT_PROFILE_PEEL) as ctx:
        ctx.upload(g)
        ctx.set_tune({"sort_shift": shift})
        capfd.readouterr()
        r = ctx.run("ondemand")
        line = [x for x in capfd.readouterr().err.splitlines() if "ordered=" in x]
        assert len(line) == 1 and " ordered=0 " not in line[0], line
        assert np.array_equal(ctx.copy_k(r["triangle_count"]), o.k)
        assert r["four_clique_count"] == o.Q and r["k_max"] == o.k_max
