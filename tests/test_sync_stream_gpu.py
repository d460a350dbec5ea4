"""Settling the last asynchronous call waits for its stream, work that the
caller put there after the call included."""
import numpy as np
import pytest

import oracle as O
from blest_b200 import Csc, Graph, Workspace, bfs_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("test", ["cuda_core", "mma"])
@pytest.mark.parametrize("calls", [1, 3])
def test_sync_waits_for_what_follows_the_call(gpu, test, calls):
    import torch
    csc = Csc.rmat(12, 8, seed=3, permute_seed=4)
    ws = Workspace(Graph.from_csc(csc))
    stream = torch.cuda.Stream()
    out = torch.empty(csc.n, dtype=torch.int32, device="cuda")
    host = torch.empty(csc.n, dtype=torch.int32, pin_memory=True)
    busy = torch.zeros(1 << 28, dtype=torch.int32, device="cuda")  # a pass over it takes a few hundred us
    torch.cuda.synchronize()
    for source in (0, 17, csc.n - 1):
        host.fill_(-7)
        with torch.cuda.stream(stream):
            for i in range(calls):
                ws.bfs_async(source if i == calls - 1 else i, out.data_ptr(), stream.cuda_stream,
                             params=bfs_params("auto", test))
            for _ in range(20):
                busy.add_(1)
            host.copy_(out, non_blocking=True)
        ws.sync()
        np.testing.assert_array_equal(host.numpy().view(np.uint32), O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, source))
