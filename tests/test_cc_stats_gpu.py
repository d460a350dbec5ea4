"""What a components call reports beside the labels: passes over edges (of
union-find on symmetric graphs, of label propagation on others) and device time."""
import numpy as np
import pytest

from blest_b200 import Bvss, Csc, Graph
from graphs import path, random_directed, star

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [lambda: path(2), lambda: path(5000), lambda: star(3000), lambda: Csc.rmat(13, 8, seed=1),
                                  lambda: Csc.grid(300, 301, 0.05, 0.001, seed=2)])
def test_symmetric(gpu, make):
    csc = make()
    g = Graph(Bvss.build(csc), csc)
    for _ in range(5):
        labels, st = g.cc()
        # one sampling pass, 1 to 12 rounds, one linking pass
        assert 3 <= st.iterations <= 14
        assert st.no_components == np.unique(labels).size
        assert 0 < st.time < 1


def test_rounds_are_counted(gpu):
    """Long chains take more than one round of hooks."""
    csc = Csc.grid(700, 701, 0.05, 0.001, seed=2)
    _, st = Graph.from_csc(csc).cc()
    assert st.iterations > 3


@pytest.mark.parametrize("n", [1, 2, 4097])
def test_no_edges(gpu, n):
    csc = Csc.from_arrays(n, np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32))
    _, st = Graph(Bvss.build(csc), csc).cc()
    assert st.iterations == 0 and st.no_components == n


def test_directed(gpu):
    csc = random_directed(3000, 20_000, 2)
    _, st = Graph(Bvss.build(csc), csc.transpose()).cc()
    assert 1 <= st.iterations <= csc.n and st.time > 0
