"""Single-source BFS over adjacency lists where its forms change: list lengths
around one piece, levels that move between one block and the whole grid,
blocks whose discovery buffer overflows, long runs of one-block levels,
frontiers that change between queue and bitmap, and directed graphs whose
out-lists are derived from the tiles. Levels equal the oracle's, parents form
a valid tree."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, bfs_params
from graphs import edges_graph, path, random_directed

pytestmark = pytest.mark.gpu


def check(csc, sources, g=None, **kw):
    csr = csc.transpose()
    g = g or Graph(Bvss.build(csc), csr)
    deg = np.diff(csr.col_ptrs.astype(np.int64))
    for direction in ("auto", "push", "pull"):
        p = bfs_params(direction, **kw)
        for s in sources:
            want = O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s)
            reached = want != O.UNREACHED
            for parents in (False, True):
                lv, par, st = g.bfs(s, parents=parents, params=p)
                np.testing.assert_array_equal(lv, want, err_msg=f"{direction} source {s} parents {parents}")
                assert st.no_visited == int(reached.sum())
                assert st.total_levels == int(want[reached].max()) + 1
                assert st.push_levels + st.pull_levels == st.total_levels
                assert st.reached_degree_sum == int(deg[reached].sum())
                if parents:
                    assert O.check_parents(csc.n, csc.col_ptrs, csc.rows, s, lv, par) == 0


@pytest.mark.parametrize("leaves", [1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 2047, 2048, 2049, 5000])
def test_list_lengths(gpu, leaves):
    """A chain of three hubs of that many leaves each (the source is a leaf of
    the first): each level's pieces and discoveries cross the limits of a
    piece, of one-block levels and of the discovery buffer."""
    hubs = [0, leaves + 1, 2 * leaves + 2]
    e = [(h, h + i) for h in hubs for i in range(1, leaves + 1)]
    e += [(h + 1, h + leaves + 1) for h in hubs[:2]]
    check(edges_graph(3 * leaves + 3, e), [1, 0])


@pytest.mark.parametrize("threads", [32, 512])
def test_buffer_overflow(gpu, threads):
    """One level of 600 k discoveries: with 32-thread blocks far more per
    block than its buffer holds, some with long lists of their own."""
    n = 600_000
    e = np.stack([np.zeros(n - 1, np.int64), np.arange(1, n)], 1)
    more = np.stack([np.repeat(np.arange(1, 40), 300), np.random.default_rng(2).integers(100, n, 39 * 300)], 1)
    e = np.unique(np.concatenate([e, more]), axis=0)
    both = np.concatenate([e, e[:, ::-1]])
    check(Csc.from_edges(n, both[:, 0], both[:, 1]), [0, 5], threads_per_block=threads, blocks_per_sm=1)


@pytest.mark.parametrize("n", [600, 3001])
def test_long_path(gpu, n):
    check(path(n), [0, n // 2])


def test_wide_and_narrow_levels(gpu):
    """Levels of 1 and of 3000 vertices in turn (diamonds in a row)."""
    e, at = [], 0
    for _ in range(6):
        e += [(at, at + i) for i in range(1, 3001)] + [(at + i, at + 3001) for i in range(1, 3001)]
        at += 3001
    check(edges_graph(at + 1, e), [0, at // 2])


@pytest.mark.parametrize("n,m", [(1, 0), (2, 1), (33, 40), (4097, 30_000), (50_001, 700_000)])
def test_directed(gpu, n, m):
    csc = random_directed(n, m, 9)
    check(csc, [0, n // 2, n - 1])
    g = Graph.from_csc(csc, csc.transpose())
    check(csc, [n // 3], g=g)


def test_directed_out_hub(gpu):
    """Out-degrees and in-degrees that differ by orders of magnitude."""
    n = 30_000
    rng = np.random.default_rng(4)
    e = np.concatenate([np.stack([np.full(n - 2, 1), np.arange(2, n)], 1),
                        np.stack([rng.integers(2, n, 60_000), rng.integers(0, 50, 60_000)], 1), [[0, 1]]])
    e = np.unique(e[e[:, 0] != e[:, 1]], axis=0)
    check(Csc.from_edges(n, e[:, 0], e[:, 1]), [0, 1, 17])


def test_uniform_dense_levels(gpu):
    """A level whose edges outnumber n / 4 (marked first, swept after)."""
    check(Csc.er(100_003, 1_600_000, seed=3), [0, 777])


def test_pull_then_push_queues_its_finds(gpu):
    """A dense core (pulled) with tails hanging off it: the pull level that
    finds the tails' ends queues them for the push levels that follow, a few
    and several thousand (more than a block's buffer), with and without the
    grid's cap."""
    for tails, spread in ((5, 1), (3000, 1), (9000, 2)):
        core = Csc.er(20_000, 400_000, seed=tails)
        src = np.repeat(np.arange(core.n), core.degrees()).astype(np.int64)
        dst = core.rows.astype(np.int64)
        at = core.n + np.arange(tails * 3).reshape(tails, 3)
        base = (np.arange(tails) * spread) % core.n
        a = np.concatenate([base, at[:, 0], at[:, 1]])
        b = np.concatenate([at[:, 0], at[:, 1], at[:, 2]])
        csc = Csc.from_edges(core.n + tails * 3, np.concatenate([src, a, b]), np.concatenate([dst, b, a]))
        check(csc, [0, csc.n - 1])
        check(csc, [7], threads_per_block=32, blocks_per_sm=1)


def test_calls_back_to_back_and_between_other_kernels(gpu):
    """The counters that one run leaves clean serve the next, whatever ran in
    between on the workspace and whichever stream the next call takes."""
    import torch

    from blest_b200 import Workspace
    csc = Csc.rmat(12, 8, seed=3, permute_seed=4)
    g = Graph(Bvss.build(csc), csc.transpose())
    ws = Workspace(g)
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [torch.empty(csc.n, dtype=torch.int32, device="cuda") for _ in range(12)]
    want = [O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s) for s in range(12)]
    labels = torch.empty(csc.n, dtype=torch.int32, device="cuda")
    for rep in range(20):
        for i, out in enumerate(outs):
            out.fill_(7)
            torch.cuda.synchronize()
            ws.bfs_async(i, out.data_ptr(), streams[i % 3].cuda_stream)
            st = ws.sync()
            assert st.source_vertex == i and st.no_visited == int((want[i] != O.UNREACHED).sum())
            if i % 4 == 1:
                ws.cc(labels.data_ptr(), stream=streams[0].cuda_stream)
            if i % 4 == 2:
                ws.mbfs_rows([0, i], [outs[0].data_ptr(), labels.data_ptr()], stream=streams[1].cuda_stream)
            if i % 4 == 3:
                g.bfs(i, params=bfs_params("auto", "mma"))
            np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want[i])
