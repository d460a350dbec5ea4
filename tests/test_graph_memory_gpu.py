"""A graph that fits the device only without what BFS over lists adds to it
(a directed graph's out-lists, the list heads, the wider queues) is made without
it, and answers the same."""
import gc

import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, Workspace, bfs_params
from graphs import random_directed

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free_bytes():
    import torch
    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("directed,short", [(True, 12), (True, 36), (False, 8), (False, 16)])
def test_graph_without_room_for_lists(gpu, directed, short):
    """`short` MB less than the whole graph and its workspace take. Directed, n
    = 2^20 and 8 M edges: out-lists 36 MB, heads 16, queues 9 more; symmetric:
    heads 16 and queues 10 (16 M edges)."""
    import torch
    n = 1 << 20
    csc = random_directed(n, 8 << 20, 5) if directed else Csc.er(n, 8 << 20, seed=5)
    csr = csc.transpose() if directed else csc
    bvss = Bvss.build(csc, full_padding=False)  # (else the upload of the padding takes the most)
    sources = [0, n // 3, n - 1]
    lv = [O.bfs_csc(n, csc.col_ptrs, csc.rows, s) for s in sources]
    cc = O.cc_csc(n, csc.col_ptrs, csc.rows)

    def answers(g):
        for s, want in zip(sources, lv):
            for parents in (False, True):
                got, par, _ = g.bfs(s, parents=parents, params=bfs_params("auto"))
                np.testing.assert_array_equal(got, want)
                if parents:
                    assert O.check_parents(n, csc.col_ptrs, csc.rows, s, got, par) == 0
        np.testing.assert_array_equal(g.cc()[0], cc)

    before = free_bytes()
    g = Graph(bvss, csr)
    whole = before - free_bytes()
    bytes_whole = g.info().device_bytes_graph + g.info().device_bytes_workspace
    answers(g)
    g.bfs(0, params=bfs_params("auto", "mma"))
    g.close()
    before = free_bytes()
    hold = torch.empty(before - (whole - short * MB), dtype=torch.uint8, device="cuda")
    try:
        g = Graph(bvss, csr)
        assert g.info().device_bytes_graph + g.info().device_bytes_workspace <= bytes_whole - short * MB
        answers(g)
        g.close()
    finally:
        del hold
        free_bytes()
    # with room again: the whole graph, and a workspace that finds none for its queues
    g = Graph(bvss, csr)
    assert g.info().device_bytes_graph + g.info().device_bytes_workspace == bytes_whole
    answers(g)
    before = free_bytes()
    ws = Workspace(g)
    w = before - free_bytes()  # with the allocator's rounding
    ws.close()
    hold = torch.empty(free_bytes() - (w - 4 * MB), dtype=torch.uint8, device="cuda")
    ws = Workspace(g)
    del hold
    free_bytes()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    for s, want in zip(sources, lv):
        ws.bfs_async(s, out.data_ptr(), stream.cuda_stream)
        ws.sync()
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)
    ws.close()
    g.close()
