"""sp24_zero: which memory a kernel clears and which the runtime's memset does, seen in a captured graph, and that exactly the bytes asked
for become zero, captured and not."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
KERNEL, MEMSET = 0, 2          # cudaGraphNodeType


def _node_types(graph):
    rt = ctypes.CDLL("libcudart.so.12")
    g, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert rt.cudaGraphGetNodes(g, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(g, nodes, ctypes.byref(count)) == 0
    kinds = []
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    return kinds


@pytest.mark.parametrize("memory,offset,count,kind", [("device", 4, 4, KERNEL), ("device", 16, 1 << 18, KERNEL), ("device", 16, (1 << 18) + 4, MEMSET),
                                                      ("device", 2, 64, MEMSET), ("device", 4, 7, MEMSET), ("pinned", 16, 64, MEMSET)])
def test_zero(memory, offset, count, kind):
    from sparse import _ext
    size = offset + count + 16
    buf = torch.ones(size, dtype=torch.uint8, device=DEV) if memory == "device" else torch.ones(size, dtype=torch.uint8).pin_memory()
    zero = lambda: _ext.check(_ext.lib().sp24_zero(buf.data_ptr() + offset, count, _ext.stream()), "zero")

    def check():
        torch.cuda.synchronize()
        assert int(buf.sum()) == size - count and not bool(buf[offset:offset + count].any())

    zero()
    check()
    torch.cuda.synchronize()
    buf.fill_(1)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        zero()
    assert _node_types(graph) == [kind]
    graph.instantiate()
    torch.cuda.synchronize()
    graph.replay()
    check()
