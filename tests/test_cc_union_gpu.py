"""Components by union-find (symmetric graphs) and the check that chooses it:
edges of the grid and warp sizes, several large components with lists over
one piece, orders that make long chains, and graphs that must not take it."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph
from graphs import edges_graph, random_directed

pytestmark = pytest.mark.gpu


def both_ways(csc):
    """The graph with its pull lists passed and checked, and without them."""
    yield Graph(Bvss.build(csc), csc.transpose())
    yield Graph.from_csc(csc)


def check(csc):
    want = O.cc_csc(csc.n, csc.col_ptrs, csc.rows)
    for g in both_ways(csc):
        for _ in range(2):
            lab, st = g.cc()
            np.testing.assert_array_equal(lab, want)
            assert st.no_components == np.unique(want).size


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 511, 512, 513, 2049, 100_003])
@pytest.mark.parametrize("per_vertex", [0.4, 1.0, 3.0])
def test_sizes(gpu, n, per_vertex):
    rng = np.random.default_rng(n)
    e = rng.integers(0, n, (int(n * per_vertex), 2))
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], axis=1), axis=0)
    check(edges_graph(n, e))


def test_several_large_components(gpu):
    """Four hubs of 3000 (lists cut in pieces, none of them in a majority)
    joined in pairs by single low-degree edges, and a clique."""
    perm = np.random.default_rng(7).permutation(4 * 3000 + 100)
    e = [(h * 3000, h * 3000 + i) for h in range(4) for i in range(1, 3000)]
    e += [(2999, 5999), (6001, 9001)]
    e += [(12000 + i, 12000 + j) for i in range(90) for j in range(i + 1, 90)]
    check(edges_graph(perm.size, [(perm[a], perm[b]) for a, b in e]))


@pytest.mark.parametrize("order", ["up", "down", "random"])
def test_long_path(gpu, order):
    n = 20_001
    ids = {"up": np.arange(n), "down": np.arange(n)[::-1], "random": np.random.default_rng(1).permutation(n)}[order]
    check(edges_graph(n, [(ids[i], ids[i + 1]) for i in range(n - 1) if i != n // 2]))


@pytest.mark.parametrize("lists", ["transpose", "own"])
def test_directed_keeps_reachability_labels(gpu, lists):
    """Directed edges (also when the caller passes the out-lists as pull
    lists): labels are the smallest id that reaches a vertex."""
    csc = random_directed(3001, 9000, 5)
    g = Graph(Bvss.build(csc), csc.transpose() if lists == "transpose" else csc)
    lab, _ = g.cc()
    np.testing.assert_array_equal(lab, O.cc_csc(csc.n, csc.col_ptrs, csc.rows))


def test_one_missing_reverse_edge(gpu):
    csc = Csc.rmat(10, 8, seed=2)
    src = np.repeat(np.arange(csc.n), csc.degrees())
    dst = csc.rows.astype(np.int64)
    keep = np.ones(src.size, bool)
    keep[src.size // 2] = False
    d = Csc.from_edges(csc.n, src[keep], dst[keep])
    lab, _ = Graph(Bvss.build(d), d.transpose()).cc()
    np.testing.assert_array_equal(lab, O.cc_csc(d.n, d.col_ptrs, d.rows))


def test_calls_back_to_back(gpu):
    """Runs leave their counters clean for the next, on any stream, with BFS
    and multi-source runs in between and with results on either side."""
    import torch

    from blest_b200 import Workspace
    csc = Csc.rmat(11, 4, seed=6, permute_seed=2)
    want = O.cc_csc(csc.n, csc.col_ptrs, csc.rows)
    g = Graph.from_csc(csc)
    ws = Workspace(g)
    streams = [torch.cuda.Stream() for _ in range(2)]
    out = torch.empty(csc.n, dtype=torch.int32, device="cuda")
    lev = torch.empty(csc.n, dtype=torch.int32, device="cuda")
    for i in range(40):
        out.fill_(-5)
        torch.cuda.synchronize()
        st = ws.cc(out.data_ptr(), stream=streams[i % 2].cuda_stream)
        assert st.no_components == np.unique(want).size and st.time > 0
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)
        if i % 3 == 0:
            ws.bfs_async(i, lev.data_ptr(), streams[1].cuda_stream)
            ws.sync()
        if i % 3 == 1:
            ws.mbfs_rows([i], [lev.data_ptr()], stream=streams[0].cuda_stream)
        np.testing.assert_array_equal(g.cc()[0], want)
