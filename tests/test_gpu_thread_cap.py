"""LibShalom_set_thread_nums caps the CTAs resident at once: with a cap set, no
kernel of a call is placed beside the one before it (the launches of a captured
call have full dependencies), and the results are the same."""
import ctypes

import pytest

import libshalom_b200 as ls
from tests.test_gpu_capture_growth import Batch

pytestmark = pytest.mark.gpu

PROGRAMMATIC = 1  # cudaGraphDependencyTypeProgrammatic


def _edge_types(graph):
    """Types of the edges of a captured graph (cudaGraphEdgeData: from port, to
    port, type, five reserved bytes)."""
    get = ctypes.CDLL("libcudart.so.12").cudaGraphGetEdges_v2
    n = ctypes.c_size_t(0)
    handle = ctypes.c_void_p(graph.raw_cuda_graph())
    assert get(handle, None, None, None, ctypes.byref(n)) == 0
    ends = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)()
    data = (ctypes.c_ubyte * (8 * n.value))()
    assert get(handle, ends[0], ends[1], data, ctypes.byref(n)) == 0
    return [data[8 * i + 2] for i in range(n.value)]


@pytest.mark.parametrize("kind", ["fp32", "bf16x6", "fma", "dmma"])
def test_cap_keeps_kernels_apart(kind):
    import torch
    b = Batch(kind, 3_000)
    s = torch.cuda.Stream()
    ls.set_stream(s)
    ls.set_sync(False)
    try:
        b.fill(1)
        torch.cuda.synchronize()
        b.run()
        torch.cuda.synchronize()
        want = b.C.clone()
        for cap in (0, 20):
            ls.set_thread_nums(cap)
            g = torch.cuda.CUDAGraph(keep_graph=True)
            with torch.cuda.graph(g, stream=s):
                b.run()
            types = _edge_types(g)
            assert len(types) >= 3
            assert (PROGRAMMATIC in types) == (cap == 0)
            b.C.fill_(float("nan"))
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(b.C, want)
    finally:
        torch.cuda.synchronize()
        ls.set_stream(None)
