"""Long runs of one-block levels in single-source BFS, repeated. A block's
discoveries are counted in shared memory; every warp reads that count and one
warp starts the next level's from zero, so a warp that read it late would leave
the run of levels alone. Levels and counts equal the oracle's in every call."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, bfs_params

pytestmark = pytest.mark.gpu


def bands(width, depth):
    """`depth` bands of `width` vertices; each vertex is joined to two of the next band."""
    at = np.arange(width * (depth - 1))
    nxt = (at // width + 1) * width
    src = np.concatenate([at, at])
    dst = np.concatenate([nxt + at % width, nxt + (at + 1) % width])
    pairs = np.unique(np.concatenate([np.stack([src, dst], 1), np.stack([dst, src], 1)]), axis=0)
    return Csc.from_edges(width * depth, pairs[:, 0], pairs[:, 1])


@pytest.mark.parametrize("width", [1, 2, 31, 32, 33, 200])  # at and around one warp's lanes
@pytest.mark.parametrize("threads", [32, 64, 512])
def test_long_runs_of_small_levels(gpu, width, threads):
    csc = bands(width, 300)
    g = Graph(Bvss.build(csc), csc)
    sources = [0, csc.n // 2, csc.n - 1]
    want = [O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s) for s in sources]
    for call in range(60):
        i = call % len(sources)
        lv, _, st = g.bfs(sources[i], params=bfs_params("auto", threads_per_block=threads))
        np.testing.assert_array_equal(lv, want[i])
        assert st.no_visited == csc.n
        assert st.total_levels == int(want[i].max()) + 1
        assert st.reached_degree_sum == csc.nnz


@pytest.mark.parametrize("test", ["cuda_core", "mma"])
@pytest.mark.parametrize("leaves,reached", [(40_000, 1), (40_000, 7), (40_000, 39_000), (300_000, 2)])
def test_long_lists_found_by_several_pieces(gpu, test, leaves, reached):
    """Three hubs that share all their leaves are reached in one pull level
    through the first, the last or nearly all of their list's pieces at once;
    pieces of the same list stop when another has found the vertex."""
    hubs = leaves + 1 + np.arange(3)
    # the source sees `reached` leaves, spread evenly over the ids
    seen = 1 + np.linspace(0, leaves - 1, reached).astype(np.int64)
    a = np.concatenate([np.zeros(reached, np.int64), np.repeat(hubs, leaves)])
    b = np.concatenate([seen, np.tile(np.arange(1, leaves + 1), 3)])
    csc = Csc.from_edges(leaves + 4, np.concatenate([a, b]), np.concatenate([b, a]))
    g = Graph(Bvss.build(csc), csc)
    want = O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, 0)
    for call in range(20):
        lv, par, st = g.bfs(0, parents=call % 2 == 1, params=bfs_params("pull", test))
        np.testing.assert_array_equal(lv, want)
        assert st.no_visited == csc.n and st.reached_degree_sum == csc.nnz
        if par is not None:
            assert O.check_parents(csc.n, csc.col_ptrs, csc.rows, 0, lv, par) == 0
