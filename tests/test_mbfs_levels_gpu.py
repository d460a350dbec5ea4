"""Multi-source BFS where a level's course changes: levels that are one half
only (pulling graphs without long lists), more levels than history slots and
than fit the byte write-out, lists around one pull piece and one id quad, row
counts around a byte group, and plans with more graphs than a block keeps
modes for. Every row equals the single-source oracle BFS."""
import numpy as np
import pytest
import torch

import oracle as O
from blest_b200 import Bvss, Csc, Graph, MbfsPlan, Workspace
from graphs import edges_graph, path, random_directed, star

pytestmark = pytest.mark.gpu


def check(csc, sources, levels):
    for i, s in enumerate(sources):
        np.testing.assert_array_equal(levels[i], O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, int(s)), err_msg=f"#{i} {s}")


@pytest.mark.parametrize("width", [32, 64, 128])
@pytest.mark.parametrize("pull_fraction", [0.0, 1e-9, 2.0])  # default, always pull, always push
@pytest.mark.parametrize("side", [9, 70, 150])
def test_grids(gpu, width, pull_fraction, side):
    csc = Csc.grid(side, side + 1, 0.05, 0.0, seed=side)
    g = Graph.from_csc(csc)
    sources = np.random.default_rng(side).integers(0, csc.n, 2 * width + 5)
    for _ in range(2):
        levels, _ = g.mbfs(sources, group_width=width, pull_fraction=pull_fraction)
        check(csc, sources[:6], levels)
        check(csc, sources[-3:], levels[-3:])


@pytest.mark.parametrize("n", [62, 63, 64, 65, 66, 129, 300])
def test_levels_around_the_slots(gpu, n):
    """Paths: 63 to 300 levels, written out at once or as slots run out."""
    csc = path(n)
    g = Graph.from_csc(csc)
    sources = [0, n - 1, n // 2, 0, 1]
    for pf in (0.0, 1e-9, 2.0):
        levels, _ = g.mbfs(sources, group_width=32, pull_fraction=pf)
        check(csc, sources, levels)


@pytest.mark.parametrize("k", [1, 3, 4, 5, 31, 32, 33, 63, 65, 127, 128, 129, 200, 257])
def test_row_counts(gpu, k):
    csc = Csc.rmat(11, 8, seed=4, permute_seed=1)
    g = Graph(Bvss.build(csc), csc.transpose())
    sources = np.random.default_rng(k).integers(0, csc.n, k)
    ws = Workspace(g)
    for width in (32, 128):
        levels, _ = g.mbfs(sources, group_width=width)
        check(csc, sources, levels)
        rows = torch.empty((k, csc.n), dtype=torch.int32, device="cuda")
        ws.mbfs_rows(sources, [rows[i].data_ptr() for i in range(k)], group_width=width)
        np.testing.assert_array_equal(rows.cpu().numpy().view(np.uint32), levels)


@pytest.mark.parametrize("leaves", [1, 2, 3, 4, 5, 62, 63, 64, 65, 127, 128, 129, 1000])
def test_list_lengths(gpu, leaves):
    """Hubs whose lists end at every place of an id quad and around a piece,
    joined in a chain, pulled and pushed."""
    hubs = [0, leaves + 1, 2 * leaves + 2]
    e = [(h, h + i) for h in hubs for i in range(1, leaves + 1)] + [(h + 1, h + leaves + 1) for h in hubs[:2]]
    csc = edges_graph(3 * leaves + 3, e)
    g = Graph.from_csc(csc)
    sources = [0, 1, csc.n - 1, leaves]
    for pf in (1e-9, 2.0):
        for width in (32, 64, 128):
            levels, _ = g.mbfs(sources, group_width=width, pull_fraction=pf)
            check(csc, sources, levels)


def test_plan_of_many_small_graphs(gpu):
    """1100 graphs, pulling and pushing side by side, some directed."""
    kinds = [path(33), star(70), random_directed(40, 100, 3), Csc.grid(6, 7, 0.0, 0.0, seed=1)]
    graphs = [Graph(Bvss.build(c), c.transpose()) for c in kinds]
    items, outs = [], []
    for i in range(1100):
        c, g = kinds[i % 4], graphs[i % 4]
        src = np.array([i % c.n, (7 * i) % c.n], dtype=np.uint32)
        outs.append((c, src, torch.empty((2, c.n), dtype=torch.int32, device="cuda")))
        items.append((g, src, outs[-1][2].data_ptr()))
    plan = MbfsPlan(items)
    for _ in range(2):
        plan.run()
        for c, src, out in outs[:40] + outs[-40:]:
            check(c, src, out.cpu().numpy().view(np.uint32))
