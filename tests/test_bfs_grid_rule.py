"""Launch size of single-source BFS over lists: the caller's blocks_per_sm and
threads_per_block are used, and the cut for small graphs counts threads."""
import ctypes
import subprocess

import numpy as np
import pytest

import oracle as O
from blest_b200 import Bvss, Csc, Graph, bfs_params
from conftest import ROOT

SMS = 148


@pytest.fixture(scope="module")
def blocks(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    (d / "rule.cpp").write_text('#include "bfs_grid.hpp"\nextern "C" int rule(uint32_t n, uint64_t nnz, int sms, int mb, '
                                'int bps, int th) { return blest::bfs_lists_blocks(n, nnz, sms, mb, bps, th); }\n')
    subprocess.run(["g++", "-std=c++20", "-shared", "-fPIC", f"-I{ROOT / 'blest_b200' / 'csrc' / 'device'}", "-o",
                    str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    f = ctypes.CDLL(str(d / "rule.so")).rule
    f.argtypes = [ctypes.c_uint32, ctypes.c_uint64] + [ctypes.c_int] * 4
    return lambda n, nnz, max_blocks, bps, threads: f(n, nnz, SMS, max_blocks, bps, threads)


@pytest.mark.parametrize("n,nnz", [(1, 0), (1024, 20_000), (1 << 19, 1 << 26), ((1 << 20) - 1, 1 << 20), (1 << 22, 1 << 27)])
def test_the_callers_blocks_per_sm_are_used(blocks, n, nnz):
    assert blocks(n, nnz, 2, 1, 512) == SMS
    assert blocks(n, nnz, 2, 2, 512) == 2 * SMS
    assert blocks(n, nnz, 8, 5, 128) == 5 * SMS
    assert blocks(n, nnz, 2, 9, 512) == 2 * SMS  # no more than are resident


@pytest.mark.parametrize("threads,max_blocks", [(32, 32), (96, 10), (128, 8), (512, 2)])
def test_the_cut_counts_threads(blocks, threads, max_blocks):
    for n, nnz in [(1, 0), (513, 100), (1024, 20_000), (1 << 16, 1 << 20), ((1 << 20) - 1, 1 << 26)]:
        want = min(max(n, nnz // 4) + 512, 512 * SMS)
        got = blocks(n, nnz, max_blocks, 0, threads) * threads
        assert want <= got < want + threads or got == max_blocks * SMS * threads
    assert blocks(1 << 20, 1 << 25, max_blocks, 0, threads) == max_blocks * SMS


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [32, 128, 512])
@pytest.mark.parametrize("bps", [0, 1, 2, 4])
def test_levels_do_not_depend_on_the_launch(gpu, threads, bps):
    for csc in (Csc.rmat(10, 8, seed=2, permute_seed=3), Csc.er(70_001, 500_000, seed=4), Csc.grid(211, 190, 0.05, 0.001, seed=1)):
        g = Graph(Bvss.build(csc), csc)
        for s in (0, csc.n // 2):
            lv, _, _ = g.bfs(s, params=bfs_params("auto", blocks_per_sm=bps, threads_per_block=threads))
            np.testing.assert_array_equal(lv, O.bfs_csc(csc.n, csc.col_ptrs, csc.rows, s))
