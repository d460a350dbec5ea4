"""Device memory of one workspace: bitmaps (four of n bits), one scratch array
(16 bytes a queued vertex and long-list piece), two level-sized outputs, the
long-list queue, and what does not grow with the graph."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, Workspace, bfs_params

pytestmark = pytest.mark.gpu

FIXED = 512 * 1024  # level trace (4096 records of 56 bytes), summaries, counters, rounding


@pytest.mark.parametrize("make", [lambda: Csc.rmat(18, 16, seed=1), lambda: Csc.grid(700, 701, 0.05, 0.001, seed=1),
                                  lambda: Csc.er(200_003, 400_000, seed=1)])
def test_bytes_per_vertex(gpu, make):
    csc = make()
    info = Graph(Bvss.build(csc), csc).info()
    bitmaps = 4 * csc.n / 8
    scratch = 16 * (csc.n + csc.nnz / 128)
    outputs = 8 * csc.n
    heavy = 16 * csc.nnz / 1024
    assert info.device_bytes_workspace <= bitmaps + scratch + outputs + heavy + FIXED


@pytest.mark.parametrize("directed", [False, True])
def test_kernels_that_share_the_scratch_follow_each_other(gpu, directed):
    """BFS over lists, BFS over tiles, components and multi-source BFS in every
    order of two on one workspace."""
    import torch
    if directed:
        r = np.random.default_rng(5)
        e = np.unique(r.integers(0, 20_000, (150_000, 2)), axis=0)
        e = e[e[:, 0] != e[:, 1]]
        csc = Csc.from_edges(20_000, e[:, 0], e[:, 1])
    else:
        csc = Csc.rmat(14, 12, seed=6, permute_seed=2)
    g = Graph(Bvss.build(csc), csc.transpose())
    ws, stream = Workspace(g), torch.cuda.Stream()
    lv = [O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s) for s in range(4)]
    cc = O.cc_csc(csc.n, csc.col_ptrs, csc.rows)
    out = torch.empty((2, csc.n), dtype=torch.int32, device="cuda")

    def bfs(test):
        def run(i):
            ws.bfs_async(i, out[0].data_ptr(), stream.cuda_stream, params=bfs_params("auto", test))
            ws.sync()
            return out[0], lv[i]
        return run

    def components(i):
        ws.cc(out[0].data_ptr(), stream=stream.cuda_stream)
        return out[0], cc

    def multi(i):
        ws.mbfs_rows([3, i], [out[1].data_ptr(), out[0].data_ptr()], stream=stream.cuda_stream)
        return out[0], lv[i]

    kinds = [bfs("cuda_core"), bfs("mma"), components, multi]
    for rep in range(3):
        for a in kinds:
            for b in kinds:
                for f in (a, b):
                    out.fill_(5)
                    torch.cuda.synchronize()
                    got, want = f(rep)
                    stream.synchronize()
                    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint32), want)
