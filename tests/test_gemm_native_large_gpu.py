"""Native SGEMM on its 128 x 128 tile: ragged sides and K tails that the cost model
sends there (checked on the captured launch), every storage pair, both alignments,
with the checks and the tolerance of the small tiles' test."""
import ctypes as C

import numpy as np
import pytest
import torch

import coral_b200 as cb
from test_gemm_native_gpu import OPS, check

pytestmark = pytest.mark.gpu

SHAPES = [(1409, 1535, 17), (1535, 1409, 47), (2047, 2045, 77)]


class _KernelNode(C.Structure):   # cudaKernelNodeParams
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p)]


def _launch(m, n, k):
    """Blocks and threads of the one kernel that an m x n x k call launches, from a captured graph."""
    a, b, c = (torch.zeros(s, device="cuda") for s in (m * k, k * n, m * n))
    cb.sgemm(0, 0, m, n, k, 1.0, a, m, b, k, 0.0, c, m)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        cb.sgemm(0, 0, m, n, k, 1.0, a, m, b, k, 0.0, c, m)
    rt = C.CDLL("libcudart.so.12")
    count, graph = C.c_size_t(8), C.c_void_p(g.raw_cuda_graph())
    nodes = (C.c_void_p * 8)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(count)) == 0 and count.value == 1
    p = _KernelNode()
    assert rt.cudaGraphKernelNodeGetParams(C.c_void_p(nodes[0]), C.byref(p)) == 0
    return p.grid[0] * p.grid[1] * p.grid[2], p.block[0]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_shapes_take_the_large_tile(cuda, shape):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shapes are chosen for 148 SMs")
    cb.set_gemm_mode(cb.GemmMode.NATIVE)
    m, n, k = shape
    assert _launch(m, n, k) == (-(-m // 128) * -(-n // 128), 128)
    assert _launch(513, 511, 517)[0] % 72 == 0   # 9 x 8 tiles of 64 x 64, for contrast


@pytest.mark.parametrize("ops", OPS, ids=str)
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_large_tile_edges(cuda, shape, ops):
    check(np.float32, *ops, *shape, seed=sum(shape))
