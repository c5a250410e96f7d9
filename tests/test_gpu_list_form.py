"""The list form in its regular layout and default schedule, which graphs take whose
matrices are not kept: every tuning setting, the device loop and the direct variant
against the oracle. A cap on the listing's chunk (read at every call) keeps the
matrices from being kept without choosing a layout or a schedule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SETTINGS = [
    {"lane_max": 8},
    {"lane_max": 32},
    {"compact_div": 1},
    {"compact_div": "never"},
    {"sort_shift": 1},
    {"sort_shift": 31},
    {"sort_shift": "never"},
    {"rounds_per_replay": 1},
    {"rounds_per_replay": 64},
    {"lane_max": 32, "compact_div": "never", "sort_shift": "never", "rounds_per_replay": 3},
]


def chunked(monkeypatch, g):
    D = g.D[: g.n].astype(np.int64)
    monkeypatch.setenv("NUCLEUS34_LIST_CHUNK_WORDS", str(int((D * ((D + 31) // 32)).sum()) // 2 + 1))


@pytest.fixture(scope="module")
def rmat(n34, oracle):
    g = n34.graph_from_edges(*n34.gen_rmat(12, 16, 1))
    return g, oracle.decompose(g, quds_cap=0)


@pytest.mark.parametrize("settings", SETTINGS, ids=[str(s) for s in SETTINGS])
def test_settings_in_the_regular_layout(n34, rmat, monkeypatch, settings):
    g, o = rmat
    chunked(monkeypatch, g)
    with n34.Context() as ctx:
        ctx.upload(g)
        ctx.set_tune(settings)
        r = ctx.run("ondemand")
        assert r["four_clique_count"] == o.Q
        assert np.array_equal(ctx.copy_k(r["triangle_count"]), o.k)


def test_the_cap_selects_the_lists(n34, rmat, monkeypatch, capfd):
    g, o = rmat
    for cap in (False, True):
        if cap:
            chunked(monkeypatch, g)
        capfd.readouterr()
        d = n34.decompose(g, variant="ondemand", flags=n34.OPT_PROFILE_PEEL, n_quds=0)
        line = [x for x in capfd.readouterr().err.splitlines() if x.startswith("[peel-profile]")]
        assert len(line) == 1 and ("compactions=" in line[0]) == cap, line
        assert np.array_equal(d.k, o.k)


@pytest.mark.parametrize("case", [("rmat", 13, 16, 3), ("rgg", 30000, 40, 9), ("ws", 5000, 16, 4)])
@pytest.mark.parametrize("variant", ["ondemand", "direct"])
def test_default_schedule(n34, oracle, monkeypatch, case, variant):
    s, t = (n34.gen_ws(case[1], case[2], 0.1, case[3]) if case[0] == "ws" else
            getattr(n34, "gen_" + case[0])(*case[1:]))
    g = n34.graph_from_edges(s, t)
    o = oracle.decompose(g, quds_cap=1 << 26)
    rounds = n34.decompose(g, variant="ondemand", n_quds=0).result["peeling_iterations"]
    chunked(monkeypatch, g)
    d = n34.decompose(g, variant=variant, n_quds=1 << 26)
    assert np.array_equal(d.tris, o.tris) and np.array_equal(d.k, o.k)
    assert d.result["four_clique_count"] == o.Q and d.result["peeling_iterations"] == rounds
    if variant == "direct":
        assert np.array_equal(d.quds, o.quds)
