"""ar_sequential_impulse with more sweeps than the reference's 18: however many, they go into one
schedule (a second one would start its first level only after the first one's last), and the results
are the oracle's bit for bit, one-body contacts and contacts of one body with itself included."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_sis_scratch import _List

pytestmark = pytest.mark.gpu


def _nodes(ctx, lst, iterations):
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        lst.solve(ctx, iterations)
    count = C.c_size_t()
    cudart = C.CDLL("libcudart.so.12")
    assert cudart.cudaGraphGetNodes(C.c_void_p(graph.raw_cuda_graph()), None, C.byref(count)) == 0
    return count.value


def test_one_schedule(ctx):
    lst = _List(300, 2000, 2000)
    lst.solve(ctx, 400)  # the arena grows here
    ctx.check()
    assert _nodes(ctx, lst, 400) == _nodes(ctx, lst, 33) == _nodes(ctx, lst, 2)


@pytest.mark.parametrize("nb,count,iterations", [(2, 40, 300), (40, 600, 33), (300, 2000, 100),
                                                 (1500, 4000, 64)])
def test_many_sweeps(ctx, nb, count, iterations):
    lst = _List(nb, count, count)
    lst.solve(ctx, iterations)
    ctx.check()
    lst.check(iterations)
