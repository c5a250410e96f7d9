"""Which form the tuning settings act on, told from the peel's profile lines: the
autotuner times the list form, whose settings they are, and sort_shift on the bit
form where that reads it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lines(capfd):
    out = [x for x in capfd.readouterr().err.splitlines() if x.startswith("[peel-profile]")]
    rows = [x for x in out if "scans=" in x]
    assert all("compactions=" in x for x in out if x not in rows)
    return len(rows), len(out) - len(rows)


def test_autotune_times_the_list_form(n34, oracle, capfd, tmp_path):
    g = n34.graph_from_edges(*n34.gen_rmat(10, 16, 1))
    o = oracle.decompose(g, quds_cap=0)
    with n34.Context(flags=n34.OPT_PROFILE_PEEL) as ctx:
        ctx.upload(g)
        capfd.readouterr()
        out = ctx.autotune(str(tmp_path / "t"))
        rows, lists = lines(capfd)
        # the first run tells the form; 16 candidates differ from the defaults
        assert rows == 1 and lists >= 2 + 16
        assert 0 < out["tuned_sec"] <= out["default_sec"]
        r = ctx.run("ondemand")
        assert lines(capfd) == (1, 0)
        assert np.array_equal(ctx.copy_k(r["triangle_count"]), o.k)


def test_autotune_orders_frontiers_on_the_rows(n34, capfd):
    g = n34.graph_from_edges(*n34.gen_rgg(200003, 32, 9))
    with n34.Context(flags=n34.OPT_PROFILE_PEEL) as ctx:
        ctx.upload(g)
        capfd.readouterr()
        ctx.autotune()
        rows, lists = lines(capfd)
        assert rows >= 3 + 5 and lists >= 2 + 11
        assert ctx.run("ondemand")["triangle_count"] >= 2 ** 24


def test_autotune_without_room_for_the_lists(n34, capfd):
    """A budget that holds the rows and not the lists, in either layout."""
    i, j = np.triu_indices(1500, 1)
    keep = (i % 3 != j % 3) & (np.random.default_rng(3).random(len(i)) < 0.6)
    a, b = np.triu_indices(12, 1)
    g = n34.graph_from_edges(np.concatenate([i[keep], a + 1500]).astype(np.uint32),
                             np.concatenate([j[keep], b + 1500]).astype(np.uint32))
    lean = n34.decompose(g, variant="ondemand", flags=n34.OPT_LEAN_MEMORY, n_quds=0)
    budget = lean.result["peak_device_bytes"] - (40 << 20)
    with n34.Context(mem_budget_bytes=budget, flags=n34.OPT_PROFILE_PEEL) as ctx:
        ctx.upload(g)
        capfd.readouterr()
        out = ctx.autotune()
        rows, lists = lines(capfd)
        assert rows >= 3 and lists == 0
        assert 0 < out["tuned_sec"] <= out["default_sec"]
        r = ctx.run("ondemand")
        assert np.array_equal(ctx.copy_k(r["triangle_count"]), lean.k)
