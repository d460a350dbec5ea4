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
