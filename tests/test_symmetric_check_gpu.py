"""Graphs made with their pull lists passed: the edge-by-edge check that tells
symmetric graphs from directed ones at creation. A graph taken for symmetric
gets components by union-find and BFS over its pull lists, so what comes out
tells what the check found."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph

pytestmark = pytest.mark.gpu


def check(csc, sources=()):
    csr = csc.transpose()
    want = O.cc_csc(csc.n, csc.col_ptrs, csc.rows)
    for g in (Graph(Bvss.build(csc), csr), Graph.from_csc(csc, csr)):
        labels, _ = g.cc()
        np.testing.assert_array_equal(labels, want)
        for s in (0, csc.n // 2, csc.n - 1, *sources):
            lv, _, _ = g.bfs(s)
            np.testing.assert_array_equal(lv, O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s))


def from_pairs(n, src, dst):
    pairs = np.unique(np.stack([src, dst], 1), axis=0)
    return Csc.from_edges(n, pairs[:, 0], pairs[:, 1])


@pytest.mark.parametrize("n", [2, 3, 31, 257, 100_003])
def test_directed_cycle(gpu, n):
    """In- and out-degrees agree everywhere; no edge has its reverse (n > 2)."""
    v = np.random.default_rng(n).permutation(n)
    check(from_pairs(n, v, np.roll(v, -1)))


def symmetric_pairs(n, m, seed):
    r = np.random.default_rng(seed)
    a, b = r.integers(0, n, m), r.integers(0, n, m)
    a, b = a[a != b], b[a != b]
    return np.concatenate([a, b]), np.concatenate([b, a])


@pytest.mark.parametrize("n,m", [(1, 0), (9, 12), (64, 400), (5001, 40_000), (60_000, 900_000)])
def test_symmetric(gpu, n, m):
    check(from_pairs(n, *symmetric_pairs(n, m, 7)))


@pytest.mark.parametrize("at", [0, 0.5, 1])
def test_one_edge_without_its_reverse(gpu, at):
    """Symmetric up to one directed 3-cycle between new vertices of equal
    degree, at the front, in the middle or at the end of the ids."""
    n = 20_001
    src, dst = symmetric_pairs(n - 3, 200_000, 11)
    x = int(at * (n - 3))
    src, dst = src + 3 * (src >= x), dst + 3 * (dst >= x)
    check(from_pairs(n, np.append(src, [x, x + 1, x + 2]), np.append(dst, [x + 1, x + 2, x])), sources=(x, x + 1))


def test_hub_sets(gpu):
    """Every vertex joined to a few hubs whose columns share one set."""
    n = 120_000
    r = np.random.default_rng(3)
    hubs = np.arange(8)
    a = np.concatenate([np.repeat(hubs, n - 8), r.integers(8, n, n)])
    b = np.concatenate([np.tile(np.arange(8, n), 8), r.integers(8, n, n)])
    a, b = a[a != b], b[a != b]
    check(from_pairs(n, np.concatenate([a, b]), np.concatenate([b, a])))
    # the same with one hub's edges turned one way
    check(from_pairs(n, np.concatenate([a, b[a != 5]]), np.concatenate([b, a[a != 5]])))


@pytest.mark.parametrize("to_hub", [False, True])
@pytest.mark.parametrize("lists", ["transpose", "same"])
def test_one_direction_of_one_edge(gpu, to_hub, lists):
    """One edge between a hub and a leaf of its own lacks its reverse. With the
    out-lists passed as pull lists (which describe the same edges then, but the
    wrong way) only the missing reverse tells; components read the tiles."""
    n = 5000
    src, dst = symmetric_pairs(n - 1, 20_000, 13)
    hub_src = np.append(src, np.full(1500, 7))
    hub_dst = np.append(dst, np.arange(100, 1600))
    both = (np.append(hub_src, np.arange(100, 1600)), np.append(hub_dst, np.full(1500, 7)))
    one = (n - 1, 7) if to_hub else (7, n - 1)
    csc = from_pairs(n, np.append(both[0], one[0]), np.append(both[1], one[1]))
    g = Graph(Bvss.build(csc), csc if lists == "same" else csc.transpose())
    labels, _ = g.cc()
    np.testing.assert_array_equal(labels, O.cc_csc(csc.n, csc.col_ptrs, csc.rows))
    if lists == "transpose":
        for s in (7, n - 1, 0):
            lv, _, _ = g.bfs(s)
            np.testing.assert_array_equal(lv, O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s))
