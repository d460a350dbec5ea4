"""Directed single-source BFS whose frontiers have few in-edges and many
out-edges (or the other way): which levels one block runs alone, look before
they claim, or mark first is a matter of out-edges."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, bfs_params

pytestmark = pytest.mark.gpu


def fans(hubs, leaves, depth, back):
    """`depth` layers of `hubs` vertices; each points to `leaves` leaves of its
    own, the first of which points to the hub of the next layer; with `back`
    every leaf also has that many in-edges from a last, unreached vertex set."""
    per = hubs * (1 + leaves)
    n = per * depth + 64
    h = (np.arange(depth)[:, None] * per + np.arange(hubs)).ravel()
    leaf = (h // per * per + hubs + (h % per) * leaves)[:, None] + np.arange(leaves)
    e = [np.stack([np.repeat(h, leaves), leaf.ravel()], 1)]
    e.append(np.stack([leaf[:-hubs, 0], h[hubs:]], 1) if depth > 1 else np.zeros((0, 2), np.int64))
    e.append(np.stack([np.full(hubs, n - 1), np.arange(hubs)], 1))  # the source sees the first layer
    if back:
        r = np.random.default_rng(1)
        e.append(np.stack([r.integers(per * depth, n - 1, back * leaf.size), np.repeat(leaf.ravel(), back)], 1))
    e = np.unique(np.concatenate(e), axis=0)
    return Csc.from_edges(n, e[:, 0], e[:, 1]), n - 1


# out-edges of a layer at and around what one block takes (2048 edges, 512
# pieces), what is looked up first (131072) and a quarter of the vertices
@pytest.mark.parametrize("hubs,leaves,depth,back", [
    (16, 128, 6, 0), (16, 129, 6, 0), (4, 512, 6, 0), (4, 513, 6, 0), (512, 4, 6, 0), (513, 4, 6, 0),
    (500, 128, 5, 0), (512, 128, 5, 0), (20, 3000, 5, 0), (512, 257, 3, 0), (64, 64, 40, 0), (30, 100, 6, 3)])
def test_fans(gpu, hubs, leaves, depth, back):
    csc, src = fans(hubs, leaves, depth, back)
    csr = csc.transpose()
    g = Graph(Bvss.build(csc), csr)
    want = O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, src)
    indeg = np.diff(csr.col_ptrs.astype(np.int64))
    for direction in ("auto", "push", "pull"):
        for parents in (False, True):
            lv, par, st = g.bfs(src, parents=parents, params=bfs_params(direction))
            np.testing.assert_array_equal(lv, want)
            assert st.reached_degree_sum == int(indeg[want != O.UNREACHED].sum())
            assert st.push_levels + st.pull_levels == st.total_levels == 2 * depth + 1
            if parents:
                assert O.check_parents(csc.n, csc.col_ptrs, csc.rows, src, lv, par) == 0
