"""Performance cases: (3,4)-nucleus decompositions as programs run them.

Every case goes through the public Python face of the library (the same C
entry points a C/C++ caller uses) and returns everything the caller asked
for: counts, K_max, K_avg and k of every triangle, and the triangle list where
the entry point hands it out with k.

Inputs are seeded synthetic edge lists of the three families the repository's
own workloads use (R-MAT with a, b, c = 0.57, 0.19, 0.19; random geometric
graphs in the unit square; Watts-Strogatz), raw: with repeats, self-loops and
in random order, as a reader would deliver them. The seed relabels the vertices
in a way that keeps the family (R-MAT: which corner of each level is the dense
one; geometric: any order of the points; Watts-Strogatz: where the ring
starts) and shuffles the pairs; the structure is the case's own, so that every
seed has the same number of triangles.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "gpu-nucleus34_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import nucleus34 as n34  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------ cases ----

def listed():
    return [
        # The smallest call: one graph in host memory, one call of the drop-in
        # entry point, results back (a small Watts-Strogatz graph of the
        # batched workload's range). All latency.
        {"name": "oneshot_ws", "mode": "oneshot", "variant": "ondemand", "kind": "ws", "n": 2000, "deg": 10},
        # The same call of the direct variant on a small skewed graph, with the
        # first four-cliques of its list.
        {"name": "oneshot_direct", "mode": "oneshot", "variant": "direct", "kind": "rmat", "scale": 10, "ef": 16},
        # The plain small configuration (R-MAT scale 12): a resident graph
        # decomposed again and again, on demand.
        {"name": "resident_rmat12", "mode": "resident", "variant": "ondemand", "kind": "rmat", "scale": 12, "ef": 16},
        # An ordinary graph with the clique list materialised.
        {"name": "direct_rmat14", "mode": "resident", "variant": "direct", "kind": "rmat", "scale": 14, "ef": 16},
        # An ordinary flat graph, direct, odd size.
        {"name": "direct_rgg", "mode": "resident", "variant": "direct", "kind": "rgg", "n": 50021, "deg": 24},
        # An ordinary skewed graph, on demand.
        {"name": "resident_rmat16", "mode": "resident", "variant": "ondemand", "kind": "rmat", "scale": 16, "ef": 16},
        # The largest skewed graph that a pass here affords (the headline
        # benchmark is the same family at scale 20).
        {"name": "resident_rmat18", "mode": "resident", "variant": "ondemand", "kind": "rmat", "scale": 18, "ef": 16},
        # A new edge list every time: built into a resident CSR on the device,
        # decomposed, k read back.
        {"name": "edges_rgg", "mode": "edges", "variant": "ondemand", "kind": "rgg", "n": 200003, "deg": 32},
        # The largest flat graph: the 4M-point configuration of the benchmark,
        # an eighth of its points.
        {"name": "resident_rgg", "mode": "resident", "variant": "ondemand", "kind": "rgg", "n": 500000, "deg": 48},
        # The same family under the same memory cap per point (40 GB for 4M
        # points), which the regular layout of the on-demand variant exceeds.
        {"name": "capped_rgg", "mode": "resident", "variant": "ondemand", "kind": "rgg", "n": 200000, "deg": 48,
         "budget": 2_000_000_000},
        # Many independent graphs in one call (the batched workload's mix).
        {"name": "batch_mixed", "mode": "batch", "kind": "mixed", "count": 56, "scale": 13, "nmax": 20000},
        # A burst of requests to the serving loop, waited for together.
        {"name": "serve_burst", "mode": "serve", "kind": "mixed_rgg", "count": 24, "scale": 14, "nmax": 50000},
    ]


def draw(rng):
    pick = rng.choice(["oneshot", "oneshot", "resident", "resident", "resident", "direct", "direct", "edges", "capped",
                       "batch", "serve"])

    def graph(t_max):
        """One family with sizes spread over the logarithm, about t_max triangles at most."""
        while True:
            kind = rng.choice(["rmat", "rmat", "rgg", "ws"])
            if kind == "rmat":
                c = {"kind": "rmat", "scale": rng.randint(8, 18), "ef": rng.randint(8, 24)}
            elif kind == "rgg":
                c = {"kind": "rgg", "n": int(math.exp(rng.uniform(math.log(500), math.log(500000)))),
                     "deg": rng.randint(12, 64)}
            else:
                c = {"kind": "ws", "n": int(math.exp(rng.uniform(math.log(500), math.log(500000)))),
                     "deg": 2 * rng.randint(4, 10)}
            if _size(c)[2] <= t_max:
                return c

    if pick == "oneshot":
        return {"mode": "oneshot", "variant": rng.choice(["ondemand", "direct"]), **graph(2e6)}
    if pick == "resident":
        return {"mode": "resident", "variant": "ondemand", **graph(7.5e7)}
    if pick == "direct":
        return {"mode": "resident", "variant": "direct", **graph(6e6)}
    if pick == "edges":
        return {"mode": "edges", "variant": "ondemand", **graph(3e7)}
    if pick == "capped":
        n = int(math.exp(rng.uniform(math.log(20000), math.log(200000))))
        return {"mode": "resident", "variant": "ondemand", "kind": "rgg", "n": n, "deg": 48, "budget": n * 10000}
    if pick == "batch":
        return {"mode": "batch", "kind": "mixed", "count": rng.randint(8, 56), "scale": rng.randint(9, 13),
                "nmax": rng.randint(2000, 20000)}
    return {"mode": "serve", "kind": "mixed_rgg", "count": rng.randint(4, 24), "scale": rng.randint(10, 14),
            "nmax": rng.randint(2000, 50000)}


# ----------------------------------------------------------------- inputs ----

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rmat(scale, ef, seed):
    g = _gen(seed)
    m = ef << scale
    s = torch.zeros(m, dtype=torch.int64, device=DEV)
    d = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        r = torch.rand(m, generator=g, device=DEV, dtype=torch.float64)
        s = 2 * s + (r >= 0.76)
        d = 2 * d + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    return s, d


def _rgg(n, deg, seed):
    g = _gen(seed)
    p = torch.rand(n, 2, generator=g, device=DEV, dtype=torch.float64)
    r = math.sqrt(deg / (math.pi * n))
    side = max(1, int(1.0 / r))
    cell = (p * side).long().clamp_(max=side - 1)
    key = cell[:, 1] * side + cell[:, 0]
    key, order = key.sort()
    pos, cx, cy = p[order], cell[order, 0], cell[order, 1]
    start = torch.searchsorted(key, torch.arange(side * side + 1, device=DEV))
    ids = torch.arange(n, device=DEV)
    src, dst = [], []
    for dx, dy in ((0, 0), (1, 0), (-1, 1), (0, 1), (1, 1)):
        x, y = cx + dx, cy + dy
        ok = (x >= 0) & (x < side) & (y < side)
        k = torch.where(ok, y * side + x, torch.zeros_like(x))
        lo = start[k]
        cnt = torch.where(ok, start[k + 1] - lo, torch.zeros_like(lo))
        a = torch.repeat_interleave(ids, cnt)
        first = torch.cumsum(cnt, 0) - cnt
        b = torch.arange(a.numel(), device=DEV) - first[a] + lo[a]
        keep = ((pos[a] - pos[b]) ** 2).sum(1) <= r * r
        if (dx, dy) == (0, 0):
            keep &= a < b
        src.append(order[a[keep]])
        dst.append(order[b[keep]])
    return torch.cat(src), torch.cat(dst)


def _ws(n, deg, seed):
    g = _gen(seed)
    i = torch.arange(n, device=DEV).repeat(deg // 2)
    j = torch.arange(1, deg // 2 + 1, device=DEV).repeat_interleave(n)
    far = torch.randint(0, n, (i.numel(),), generator=g, device=DEV)
    move = torch.rand(i.numel(), generator=g, device=DEV) < 0.1
    return i, torch.where(move, far, (i + j) % n)


def _edges(c, seed):
    """The raw edge list of a one-graph case, relabelled and shuffled, as uint32 arrays."""
    rng = random.Random(seed)
    if c["kind"] == "rmat":
        s, d = _rmat(c["scale"], c["ef"], c.get("structure", 1))
        mask = rng.randrange(1 << c["scale"])
        s, d = s ^ mask, d ^ mask
    elif c["kind"] == "rgg":
        s, d = _rgg(c["n"], c["deg"], c.get("structure", 1))
        label = torch.randperm(c["n"], generator=_gen(rng.randrange(1 << 30)), device=DEV)
        s, d = label[s], label[d]
    else:
        s, d = _ws(c["n"], c["deg"], c.get("structure", 1))
        turn = rng.randrange(c["n"])
        s, d = (s + turn) % c["n"], (d + turn) % c["n"]
    p = torch.randperm(s.numel(), generator=_gen(rng.randrange(1 << 30)), device=DEV)
    return s[p].cpu().numpy().astype(np.uint32), d[p].cpu().numpy().astype(np.uint32)


def _members(c, seed):
    """The member graphs of a batch or a burst."""
    sizes, rng = random.Random(c["count"]), random.Random(seed)
    out = []
    for i in range(c["count"]):
        if i % 2 == 0:
            m = {"kind": "rmat", "scale": sizes.randint(8, c["scale"]), "ef": sizes.randint(8, 24)}
        else:
            n = int(math.exp(sizes.uniform(math.log(500), math.log(c["nmax"]))))
            m = {"kind": "ws", "n": n, "deg": 10} if c["kind"] == "mixed" else \
                {"kind": "rgg", "n": n, "deg": sizes.randint(16, 64)}
        out.append(({**m, "structure": i + 1}, rng.randrange(1 << 30)))
    return out


def prepare(case, seed):
    mode = case["mode"]
    if mode in ("batch", "serve"):
        graphs = [n34.graph_from_edges(*_edges(m, s)) for m, s in _members(case, seed)]
        state = {"case": case, "graphs": graphs}
        if mode == "serve":
            state["server"] = n34.Server(mem_budget_bytes=20_000_000_000)
        return state
    s, d = _edges(case, seed)
    if mode == "oneshot":
        return {"case": case, "graph": n34.graph_from_edges(s, d)}
    ctx = n34.Context(mem_budget_bytes=case.get("budget", 0))
    if mode == "edges":
        return {"case": case, "ctx": ctx, "src": s, "dst": d}
    ctx.upload_edges(s, d)
    return {"case": case, "ctx": ctx}


# -------------------------------------------------------------------- run ----

def _counts(r):
    return {"triangles": int(r["triangle_count"]), "cliques": int(r["four_clique_count"]), "k_max": int(r["k_max"]),
            "k_avg": float(r["k_avg"])}


def _many(summaries, ks):
    """Results of many graphs: one array per count, one k array per graph."""
    rows = [_counts(r) for r in summaries]
    return {**{f: np.array([r[f] for r in rows]) for f in ("triangles", "cliques", "k_max", "k_avg")}, "k": ks}


def run(state):
    c = state["case"]
    mode = c["mode"]
    if mode == "oneshot":
        d = n34.decompose(state["graph"], variant=c["variant"])
        out = {**_counts(d.result), "k": d.k, "tris": d.tris}
        if d.quds is not None:
            out["quds"] = d.quds
        return out
    if mode == "batch":
        with n34.batch_decompose(state["graphs"]) as b:
            return _many([b.summary(i) for i in range(b.count)], [b.copy_k(i) for i in range(b.count)])
    if mode == "serve":
        srv = state["server"]
        ids = [srv.submit(g) for g in state["graphs"]]
        infos, ks = [], []
        for i in ids:
            infos.append(srv.wait(i))
            ks.append(srv.copy_k(i, int(infos[-1]["triangle_count"])))
            srv.release(i)
        return _many(infos, ks)
    ctx = state["ctx"]
    if mode == "edges":
        ctx.upload_edges(state["src"], state["dst"])
    r = ctx.run(c["variant"])
    return {**_counts(r), "k": ctx.copy_k(int(r["triangle_count"]))}


# ------------------------------------------------------------------- work ----

def _size(c):
    """(vertices, edges, triangles, four-cliques) of a one-graph case, from the
    families' densities (triangles and cliques per edge measured on seeds)."""
    if c["kind"] == "rmat":
        s, ef = c["scale"], c["ef"]
        return (2 ** s, 0.85 * ef * 2 ** s, 2.8e6 * 5.5 ** ((s - 14) / 2) * (ef / 16) ** 1.9,
                3.5e7 * 8.1 ** ((s - 14) / 2) * (ef / 16) ** 2.8)
    if c["kind"] == "rgg":
        n, d = c["n"], c["deg"]
        return n, n * d / 2, 0.0972 * n * d ** 2, 0.01137 * n * d ** 3
    n, d = c["n"], c["deg"]
    return n, n * d / 2, 0.073 * n * d ** 2, 0.0053 * n * d ** 3


def work(case):
    """Bytes: the oriented CSR (or the pairs) in, k (and the triangles) out.
    Operations: every four-clique found once and its four supports updated."""
    parts = [m for m, _ in _members(case, 0)] if case["mode"] in ("batch", "serve") else [case]
    byts = ops = 0
    for p in parts:
        n, m, t, q = _size(p)
        byts += 8 * m if case["mode"] == "edges" else 4 * (n + m)
        byts += 16 * t if case["mode"] == "oneshot" else 4 * t
        ops += 4 * q
    return {"bytes": int(byts), "flops": int(ops)}


# ------------------------------------------------------------------ exact ----

def _pairs_in_groups(key):
    """All index pairs (i, j) with key[i] == key[j] and i < j, key ascending."""
    n = key.numel()
    _, cnt = torch.unique_consecutive(key, return_counts=True)
    end = torch.repeat_interleave(torch.cumsum(cnt, 0), cnt)
    more = end - torch.arange(n, device=key.device) - 1
    i = torch.repeat_interleave(torch.arange(n, device=key.device), more)
    first = torch.cumsum(more, 0) - more
    j = torch.arange(i.numel(), device=key.device) - first[i] + i + 1
    return i, j


def _find(keys, q):
    p = torch.searchsorted(keys, q).clamp_(max=keys.numel() - 1)
    return p, keys[p] == q


def exact(case, seed):
    """The decomposition in plain torch with 64-bit integers: list triangles
    and four-cliques by joining sorted keys, then peel level by level. For
    graphs small enough to hold every four-clique with 64-bit members."""
    if case["mode"] in ("batch", "serve") or _size(case)[3] > 5e7:
        return None
    s, d = _edges(case, seed)
    s = torch.from_numpy(s.astype(np.int64)).to(DEV)
    d = torch.from_numpy(d.astype(np.int64)).to(DEV)
    keep = s != d
    s, d = s[keep], d[keep]
    n = int(torch.maximum(s, d).max()) + 1
    lo, hi = torch.minimum(s, d), torch.maximum(s, d)
    und = torch.unique(lo * n + hi)
    lo, hi = und // n, und % n
    deg = torch.bincount(lo, minlength=n) + torch.bincount(hi, minlength=n)
    flip = (deg[lo] > deg[hi])  # equal degrees keep the lower id first
    a, b = torch.where(flip, hi, lo), torch.where(flip, lo, hi)
    E = torch.sort(a * n + b).values  # oriented edges (u, v) by u, then v
    eu, ev = E // n, E % n
    # triangles: two out-edges of u, closed by v -> w in either direction
    i, j = _pairs_in_groups(eu)
    c1, f1 = _find(E, ev[i] * n + ev[j])
    c2, f2 = _find(E, ev[j] * n + ev[i])
    ta = torch.cat([j[f1], i[f2]])  # edge u -> w, the head of the closing edge
    tb = torch.cat([i[f1], j[f2]])
    tc = torch.cat([c1[f1], c2[f2]])
    m = E.numel()
    key, order = torch.sort(ta * m + tb)
    ta, tb, tc = ta[order], tb[order], tc[order]
    T = key.numel()
    # four-cliques, each once: triangles (u, v, w) and (u, v, x) with edge
    # u -> v as b in both (v below w and x), closed by w -> x or x -> w
    bo = torch.sort(tb, stable=True).indices
    i, j = _pairs_in_groups(tb[bo])
    i, j = bo[i], bo[j]
    w, x = ev[ta[i]], ev[ta[j]]
    quads = []
    for p, q, h, t in ((i, j, x, w), (j, i, w, x)):  # closing edge t -> h, q the triangle of h
        cl, f = _find(E, t * n + h)
        p, q, cl = p[f], q[f], cl[f]
        third, _ = _find(key, ta[q] * m + ta[p])  # (u, t, h): a = u -> h, b = u -> t
        top, _ = _find(key, tc[q] * m + tc[p])    # (v, t, h): a = v -> h, b = v -> t
        quads.append(torch.stack([p, q, third, top], 1))
    quads = torch.cat(quads)
    Q = quads.shape[0]
    S = torch.bincount(quads.reshape(-1), minlength=T)
    K = torch.zeros(T, dtype=torch.int64, device=DEV)
    alive = torch.ones(T, dtype=torch.bool, device=DEV)
    level = 0
    live = quads
    while True:
        if not bool(alive.any()):
            break
        die = alive & (S <= level)
        if not bool(die.any()):
            level = int(S[alive].min())
            continue
        K[die] = level
        alive &= ~die
        gone = die[live].any(1)
        S -= torch.bincount(live[gone].reshape(-1), minlength=T)
        live = live[~gone]
    k = K.to(torch.int32).cpu().numpy()
    out = {"triangles": T, "cliques": Q, "k_max": int(K.max()) if T and Q else 0,
           "k_avg": float(int(K.sum())) / T if T and Q else 0.0, "k": k}
    if case["mode"] == "oneshot":
        out["tris"] = torch.stack([ta, tb, tc], 1).cpu().numpy().astype(np.uint32)
        if case["variant"] == "direct":
            # by lowest member, then by the vertex outside it; members ascending
            mem = torch.sort(quads, 1).values
            tri_v = torch.stack([eu[tb], ev[tb], ev[ta]], 1)
            rest = tri_v[mem[:, 1:]].reshape(Q, -1)
            base = tri_v[mem[:, 0]]
            outside = rest.sum(1) - 2 * base.sum(1)  # the fourth vertex occurs three times
            fourth = outside // 3
            o = torch.sort(fourth, stable=True).indices
            o = o[torch.sort(mem[o, 0], stable=True).indices]
            out["quds"] = mem[o[:5]].cpu().numpy().astype(np.uint32)
    return out
