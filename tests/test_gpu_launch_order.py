"""Which launches of the library may start behind the last wave of the one before (programmatic edges in a captured graph) and which go
in plain stream order: grids of long blocks that would crowd on the SMs with room."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class _Edge(ctypes.Structure):
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte), ("reserved", ctypes.c_ubyte * 5)]


def _chained(fn):
    """Of two captured calls of fn, whether the second's kernel starts early."""
    rt = ctypes.CDLL("libcudart.so.12")
    fn()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        fn()
        fn()
    g, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert rt.cudaGraphGetEdges_v2(g, None, None, None, ctypes.byref(n)) == 0 and n.value == 1
    a, b, e = (ctypes.c_void_p * 1)(), (ctypes.c_void_p * 1)(), (_Edge * 1)()
    assert rt.cudaGraphGetEdges_v2(g, a, b, e, ctypes.byref(n)) == 0
    return e[0].type == 1          # cudaGraphDependencyTypeProgrammatic


# exact MVUE of rows: blocks of 32 rows x 512 columns, three on an SM at once
@pytest.mark.parametrize("m,k,early", [(512, 2048, True), (2048, 2048, False), (8192, 4096, True)])
def test_grids_that_crowd_go_in_plain_order(m, k, early):
    from sparse import _ext
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = (m // 32) * (k // 512)
    assert early == (blocks <= sms or -(-blocks // sms) >= 3)
    x = torch.randn(m, k, device=DEV).half()
    packed, meta = torch.empty(m, k // 2, dtype=torch.float16, device=DEV), torch.empty(m, k // 16, dtype=torch.int16, device=DEV)

    def call():
        _ext.check(_ext.lib().sp24_prune_compress(x.data_ptr(), _ext.F16, m, k, k, 0, packed.data_ptr(), _ext.F16, k // 2, meta.data_ptr(),
                                                  _ext.PRUNE_MVUE, None, 0, None, 0, 1, 0, torch.cuda.current_stream().cuda_stream), "prune")
    assert _chained(call) == early
