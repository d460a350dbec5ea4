"""Timed cases of the library's work: single-source BFS, connected components,
multi-source BFS, multi-graph plans and the query server, each through its
public entry points, on the graph families and sizes of the benchmark
workloads and tests (RMAT, Erdos-Renyi, grids; 2^10 to 2^22 vertices).

A case names a graph (family, vertices, edges) and what is asked of it; the
seed draws the graph's edges and the source vertices. Graphs are generated
on the GPU, handed over as host arrays (Csc.from_arrays) and made resident
(Graph.from_csc) before the timed pass, as a program that loads a graph and
then answers queries does.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import blest_b200 as B
from blest_b200.server import Server

UNREACHED = -1  # 0xFFFFFFFF as int32


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # The smallest call: one query on a graph of the smallest multi-graph
        # batch size, where launches, barriers and host work are all there is.
        _bfs("bfs_small", "rmat", 1024, 16, k=1, mode="device"),
        # The plain single-source configuration, RMAT scale 16, reordered.
        _bfs("bfs_rmat16", "rmat", 1 << 16, 16, k=1, mode="device", order="jaccard", window=4096),
        # A directed graph of odd size with the parent option (its pull lists
        # are the transpose).
        _bfs("bfs_directed_parents", "directed", 300_007, 12, k=1, mode="parents"),
        # The plain Python call with its results on the host.
        _bfs("bfs_host_rmat18", "rmat", 1 << 18, 16, k=1, mode="host"),
        # A query stream on a large skewed graph: asynchronous calls, settled
        # at the end (the way the throughput benchmark runs).
        _bfs("bfs_stream_rmat22", "rmat", 1 << 22, 16, k=16, mode="stream"),
        # High diameter: one query on a grid with odd sides and shortcuts.
        _bfs("bfs_grid", "grid", 2901 * 2801, 2, k=1, mode="device", width=2901),
        # Low skew: uniform degree 32, every level dense, odd vertex count.
        _bfs("bfs_er", "er", 2_000_003, 16, k=4, mode="stream"),
        # Components of a skewed graph and of a grid.
        _cc("cc_rmat20", "rmat", 1 << 20, 16),
        _cc("cc_grid", "grid", 2048 * 2047, 2, width=2048),
        # Many sources on one graph (two full 128-source groups).
        _mbfs("mbfs_rmat20", "rmat", 1 << 20, 16, k=256, group=128),
        # Many uneven graphs in one captured launch, 8 sources each.
        _plan("plan_48_graphs", count=48, median=1 << 14, k=8, group=32),
        # A burst of mixed queries to the server over three resident graphs.
        _serve("serve_burst", n=1 << 18, requests=96),
    ]


def _named(name, case):
    return {"name": name, **case} if name else case


def _bfs(name, family, n, ef, *, k, mode, order="natural", window=0, width=0):
    return _named(name, {"kind": "bfs", "family": family, "n": n, "ef": ef, "k": k, "mode": mode, "order": order,
                         "window": window, "width": width})


def _cc(name, family, n, ef, *, width=0):
    return _named(name, {"kind": "cc", "family": family, "n": n, "ef": ef, "order": "natural", "window": 0,
                         "width": width})


def _mbfs(name, family, n, ef, *, k, group, width=0):
    return _named(name, {"kind": "mbfs", "family": family, "n": n, "ef": ef, "k": k, "group": group,
                         "order": "natural", "window": 0, "width": width})


def _plan(name, *, count, median, k, group):
    return _named(name, {"kind": "plan", "count": count, "median": median, "k": k, "group": group})


def _serve(name, *, n, requests):
    return _named(name, {"kind": "serve", "n": n, "requests": requests})


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["bfs", "bfs", "bfs", "cc", "cc", "mbfs", "plan", "serve"])
    if kind == "plan":
        return _plan(None, count=rng.randint(4, 48), median=_log_int(rng, 1 << 11, 1 << 14),
                     k=_log_int(rng, 1, 32), group=rng.choice([32, 64, 128]))
    if kind == "serve":
        return _serve(None, n=_log_int(rng, 1 << 12, 1 << 18), requests=_log_int(rng, 1, 96))
    family = rng.choice(["rmat", "er", "grid"] + (["directed"] if kind != "cc" else []))
    width = 0
    if family == "grid":
        width = _log_int(rng, 32, 2048)
        n, ef = width * _log_int(rng, 32, 2048), 2
    else:
        n = _log_int(rng, 1 << 10, 1 << 21)
        ef = _log_int(rng, 4, min(32, (1 << 25) // n))
    if kind == "bfs":
        mode = rng.choice(["device", "stream", "host", "parents"])
        order, window = "natural", 0
        if family == "rmat" and n <= 1 << 17 and rng.random() < 0.5:
            order, window = "jaccard", 1024
        return _bfs(None, family, n, ef, k=_log_int(rng, 2, 16) if mode == "stream" else 1, mode=mode, order=order,
                    window=window, width=width)
    if kind == "cc":
        return _cc(None, family, n, ef, width=width)
    k = _log_int(rng, 8, max(8, min(512, (1 << 28) // n)))
    return _mbfs(None, family, n, ef, k=k, group=rng.choice([32, 64, 128]), width=width)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _edges(family: str, n: int, ef: int, width: int, seed: int):
    """Directed edge endpoints (before symmetrising) as int64 CUDA tensors."""
    g = _gen(seed)
    if family in ("grid", "er"):
        # as in measured data, one vertex in 200 has no edge
        gone = torch.zeros(n, dtype=torch.bool, device="cuda")
        gone[torch.randperm(n, generator=g, device="cuda")[: n // 200 + 2]] = True
    if family == "grid":
        ids = torch.arange(n, device="cuda")
        src = torch.cat([ids[ids % width != width - 1], ids[: n - width]])
        dst = torch.cat([ids[ids % width != width - 1] + 1, ids[: n - width] + width])
        keep = torch.rand(src.numel(), generator=g, device="cuda") >= 0.05
        m = src.numel() // 1000
        far = torch.randint(0, n, (2, m), generator=g, device="cuda")
        src, dst = torch.cat([src[keep], far[0]]), torch.cat([dst[keep], far[1]])
        there = ~(gone[src] | gone[dst])
        return src[there], dst[there]
    m = n * ef
    if family == "er":
        e = torch.randint(0, n, (2, m), generator=g, device="cuda")
        e = e[:, ~(gone[e[0]] | gone[e[1]])]
        return e[0], e[1]
    # RMAT with quadrant probabilities 0.57 / 0.19 / 0.19 / 0.05; ids beyond n
    # are folded back for sizes that are no power of two; ids permuted
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=g, device="cuda")
        src = src * 2 + (r >= 0.76)
        dst = dst * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(n, generator=g, device="cuda")
    return perm[src % n], perm[dst % n]


def _columns(n: int, src, dst):
    """Sorted, de-duplicated columns of the edges src -> dst."""
    key = torch.sort(src * n + dst).values
    key = key[torch.cat([torch.ones(1, dtype=torch.bool, device="cuda"), key[1:] != key[:-1]])]
    ptr = torch.searchsorted(key, torch.arange(n + 1, device="cuda") * n)
    return ptr.to(torch.int32).cpu().numpy().view(np.uint32), (key % n).to(torch.int32).cpu().numpy().view(np.uint32)


def _directed_edges(case: dict, seed: int):
    """All directed edges of the case's graph, self loops dropped."""
    src, dst = _edges(case["family"], case["n"], case["ef"], case.get("width", 0), seed)
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if case["family"] != "directed":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    return src, dst


def _graph(case: dict, seed: int):
    """The resident graph and its inverse ordering (old id -> new id), or
    None when the vertices keep their ids."""
    n = case["n"]
    src, dst = _directed_edges(case, seed)
    csc = B.Csc.from_arrays(n, *_columns(n, src, dst))
    if case["family"] == "directed":
        return B.Graph.from_csc(csc, B.Csc.from_arrays(n, *_columns(n, dst, src))), None
    inv = None
    if case.get("order", "natural") != "natural":
        inv = csc.reorder(case["order"], window=case["window"])
    return B.Graph.from_csc(csc), inv


def _sources(case: dict, seed: int, k: int, src) -> np.ndarray:
    """k distinct vertices with an out-edge (original ids)."""
    has = torch.unique(src)
    pick = torch.randperm(has.numel(), generator=_gen(seed + 7919), device="cuda")[:k]
    return has[pick].cpu().numpy().astype(np.uint32)


def _plan_cases(case: dict):
    """Lognormal vertex counts between 2^10 and 2^18, edge factors 4 to 32
    (the sizes belong to the case; the seed draws the edges)."""
    r = random.Random(case["count"] * 1000003 + case["median"])
    out = []
    for _ in range(case["count"]):
        n = int(case["median"] * math.exp(r.gauss(0.0, 1.0)))
        out.append({"family": "rmat", "n": max(1 << 10, min(1 << 18, n)), "ef": r.randint(4, 32)})
    return out


def _serve_cases(case: dict):
    n = case["n"]
    side = max(32, math.isqrt(n))
    return [{"family": "rmat", "n": n, "ef": 16}, {"family": "grid", "n": side * side, "ef": 2, "width": side},
            {"family": "er", "n": max(1024, n // 2 + 1), "ef": 8}]


def _serve_requests(case: dict):
    """(graph, is_cc) of each request: graphs in turn, one in five asks for
    components."""
    return [(i % 3, i % 5 == 4) for i in range(case["requests"])]


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "plan":
        items, outs, graphs = [], [], []
        for i, c in enumerate(_plan_cases(case)):
            src, _ = _directed_edges(c, seed * 4099 + i)
            g, _ = _graph(c, seed * 4099 + i)
            s = _sources(c, seed + i, case["k"], src)
            out = torch.empty((s.size, c["n"]), dtype=torch.int32, device="cuda")
            graphs.append(g)
            outs.append(out)
            items.append((g, s, out.data_ptr()))
        torch.cuda.synchronize()
        return {"case": case, "graphs": graphs, "outs": outs, "plan": B.MbfsPlan(items, group_width=case["group"])}
    if kind == "serve":
        srv = Server(lanes=4)
        cs = _serve_cases(case)
        gids, pools = [], []
        for i, c in enumerate(cs):
            src, _ = _directed_edges(c, seed * 4099 + i)
            gids.append(srv.add_graph(_graph(c, seed * 4099 + i)[0]))
            pools.append(_sources(c, seed + i, 256, src))
        reqs = [(g, cc, int(pools[g][i % pools[g].size])) for i, (g, cc) in enumerate(_serve_requests(case))]
        outs = [torch.empty((max(1, sum(r[0] == g for r in reqs)), c["n"]), dtype=torch.int32, device="cuda").fill_(0)
                for g, c in enumerate(cs)]
        torch.cuda.synchronize()
        return {"case": case, "server": srv, "gids": gids, "requests": reqs, "outs": outs}
    graph, inv = _graph(case, seed)
    n = case["n"]
    st = {"case": case, "graph": graph}
    if kind == "cc":
        st["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
        st["ws"] = B.Workspace(graph)
        st["stream"] = torch.cuda.Stream()
        return st
    s = _sources(case, seed, case["k"], _directed_edges(case, seed)[0])
    if inv is not None:
        s = inv[s]
    st["sources"] = s if kind == "mbfs" else [int(x) for x in s]
    if kind == "mbfs" or case["mode"] != "host":
        st["out"] = torch.empty((s.size, n), dtype=torch.int32, device="cuda")
    if kind == "mbfs" or case["mode"] in ("stream", "parents"):
        st["ws"] = B.Workspace(graph)
        st["stream"] = torch.cuda.Stream()
    if kind == "bfs" and case["mode"] == "parents":
        st["parents"] = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "bfs":
        return _run_bfs(st, case)
    if kind == "cc":
        stats = st["ws"].cc(st["out"].data_ptr(), stream=st["stream"].cuda_stream)
        return {"labels": st["out"], "components": stats.no_components}
    if kind == "mbfs":
        out = st["out"]
        st["ws"].mbfs_rows(st["sources"], [out[i].data_ptr() for i in range(out.shape[0])],
                           group_width=case["group"], stream=st["stream"].cuda_stream)
        return out
    if kind == "plan":
        st["plan"].run()
        return st["outs"]
    srv, rows = st["server"], [0, 0, 0]
    tickets = []
    for g, cc, source in st["requests"]:
        out = st["outs"][g][rows[g]]
        rows[g] += 1
        tickets.append(srv.submit_cc(st["gids"][g], out) if cc else srv.submit_bfs(st["gids"][g], source, out))
    for t in tickets:
        t.result()
        srv.release(t.id)
    return st["outs"]


def _run_bfs(st, case):
    mode, g = case["mode"], st["graph"]
    if mode == "host":
        levels, _, stats = g.bfs(st["sources"][0])
        return {"levels": levels.view(np.int32), "visited": stats.no_visited}
    out = st["out"]
    if mode == "stream":
        ws, stream = st["ws"], st["stream"].cuda_stream
        for i, s in enumerate(st["sources"]):
            ws.bfs_async(s, out[i].data_ptr(), stream)
        ws.sync()
        return out
    if mode == "device":
        stats = g.bfs_device(st["sources"][0], out.data_ptr())
        return {"levels": out, "visited": stats.no_visited, "depth": stats.total_levels}
    # Which of a vertex's valid parents is recorded is up to the run; every
    # one of them lies on the level before, so the level of the parent is
    # what two runs have in common (the source is its own parent).
    parents = st["parents"]
    with torch.cuda.stream(st["stream"]):
        st["ws"].bfs_async(st["sources"][0], out.data_ptr(), st["stream"].cuda_stream, parents.data_ptr())
        stats = st["ws"].sync()
        of_parent = torch.where(parents >= 0, out[0][parents.clamp(min=0).long()], parents)
    return {"levels": out, "level_of_parent": of_parent, "visited": stats.no_visited}


# --------------------------------------------------------------------------
# what a pass cannot do without, and its exact result
# --------------------------------------------------------------------------
def work(case: dict) -> dict:
    """Per traversed vertex its list bound and one edge (8 bytes) read, per
    result 4 bytes written; traversals of one call that share a pass share
    the reads."""
    kind = case["kind"]
    if kind == "bfs":
        per = 16 if case["mode"] == "parents" else 12
        return {"bytes": float(per * case["n"] * case["k"]), "flops": 0.0}
    if kind == "cc":
        return {"bytes": 12.0 * case["n"], "flops": 0.0}
    if kind == "mbfs":
        return {"bytes": case["n"] * (8.0 + 4.0 * case["k"]), "flops": 0.0}
    if kind == "plan":
        n = case["count"] * case["median"] * math.exp(0.5)  # mean of the lognormal
        return {"bytes": n * (8.0 + 4.0 * case["k"]), "flops": 0.0}
    n = sum(c["n"] for c in _serve_cases(case))
    return {"bytes": n * (8.0 + 4.0 * case["requests"] / 3), "flops": 0.0}


def _levels(n: int, src, dst, source: int):
    """BFS levels by whole-edge-list passes."""
    lev = torch.full((n,), UNREACHED, dtype=torch.int32, device="cuda")
    lev[source] = 0
    d = 0
    while True:
        hit = dst[lev[src] == d]
        hit = hit[lev[hit] == UNREACHED]
        if hit.numel() == 0:
            return lev, d + 1
        d += 1
        lev[hit] = d


def _labels(n: int, src, dst):
    """Smallest vertex id of each component: minimum over the edges and
    pointer jumping until nothing changes."""
    lab = torch.arange(n, device="cuda")
    while True:
        new = lab.scatter_reduce(0, dst, lab[src], "amin")
        new = torch.minimum(new, new[new])
        if torch.equal(new, lab):
            return lab.to(torch.int32)
        lab = new


def _size(case: dict) -> int:
    return case["n"] * case["ef"] * case.get("k", 1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("plan", "serve", "mbfs") or _size(case) > 1 << 28:
        return None
    n = case["n"]
    src, dst = _directed_edges(case, seed)
    if kind == "cc":
        lab = _labels(n, src, dst)
        ids = torch.arange(n, device="cuda", dtype=torch.int32)
        return {"labels": lab, "components": int((lab == ids).sum())}
    if case["order"] != "natural":  # ids are those of the library's own ordering
        return None
    s = _sources(case, seed, case["k"], src)
    rows, depths = zip(*(_levels(n, src, dst, int(x)) for x in s))
    out = torch.stack(rows)
    visited = int((out[0] >= 0).sum())
    if case["mode"] == "host":
        return {"levels": out[0].cpu().numpy(), "visited": visited}
    if case["mode"] == "stream":
        return out
    if case["mode"] == "device":
        return {"levels": out, "visited": visited, "depth": depths[0]}
    return {"levels": out, "level_of_parent": (out[0] - 1).clamp(min=UNREACHED).where(out[0] != 0, out[0]),
            "visited": visited}
