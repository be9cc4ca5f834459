"""Grouped batches captured into a caller's CUDA graph: the library's workspace
may grow inside the capture, and a graph stays valid when a later call outgrows
the workspace that it names.  Replays give the bits of direct calls."""
import numpy as np
import pytest

import libshalom_b200 as ls
from tests._util import to_dev

pytestmark = pytest.mark.gpu

# entries whose lists exceed the first workspace (1 MB)
KINDS = [("fp32", 12_000), ("bf16x6", 20_000), ("fma", 60_000), ("dmma", 60_000)]


class Batch:
    def __init__(self, kind, count):
        import torch
        double = kind in ("fma", "dmma")
        dt, size = (torch.float64, 8) if double else (torch.float32, 4)
        self.kind, self.count, self.double = kind, count, double
        self.A, self.B, self.C = (torch.empty(count * n, dtype=dt, device="cuda")
                                  for n in (5 * 3, 3 * 4, 5 * 4))
        e = np.zeros(count, ls.entry_dtypes()[double])
        e["M"], e["N"], e["K"], e["alpha"] = 5, 4, 3, 1.0
        for name, t, n in (("A", self.A, 15), ("B", self.B, 12), ("C", self.C, 20)):
            e[name] = t.data_ptr() + size * n * np.arange(count)
        self.E = to_dev(e.view(np.uint8))

    def fill(self, seed):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.A.uniform_(-1, 1, generator=g)
        self.B.uniform_(-1, 1, generator=g)
        self.C.fill_(float("nan"))

    def run(self, count=None):
        if self.double:
            ls.set_dgemm_method(ls.DGEMM_FMA if self.kind == "fma" else ls.DGEMM_DMMA)
            ls.dgemm_batched(self.E, count or self.count)
        else:
            ls.set_precision(ls.PREC_FP32 if self.kind == "fp32" else ls.PREC_BF16X6)
            ls.sgemm_batched(self.E, count or self.count)

    def check(self, graph, seed):
        import torch
        torch.cuda.synchronize()
        self.fill(seed)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        got = self.C.clone()
        assert torch.isfinite(got).all()
        self.C.fill_(float("nan"))
        torch.cuda.synchronize()
        self.run()
        torch.cuda.synchronize()
        assert torch.equal(got, self.C)


@pytest.fixture
def stream():
    import torch
    ls.finalize()
    s = torch.cuda.Stream()
    ls.set_stream(s)
    ls.set_sync(False)
    yield s
    torch.cuda.synchronize()
    ls.set_stream(None)
    ls.finalize()


def _capture(s, b):
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        b.run()
    return g


@pytest.mark.parametrize("kind,count", KINDS, ids=[k for k, _ in KINDS])
def test_workspace_grows_in_a_capture(stream, kind, count):
    b = Batch(kind, count)
    b.fill(1)
    b.run(16)  # the first workspace
    stream.synchronize()
    g = _capture(stream, b)
    for seed in (2, 3):
        b.check(g, seed)


def test_graph_keeps_its_workspace(stream):
    small = [Batch(kind, 300) for kind, _ in KINDS]
    for b in small:
        b.fill(1)
        b.run()
    stream.synchronize()
    graphs = [_capture(stream, b) for b in small]
    for kind, count in KINDS * 2:  # outgrown again and again
        big = Batch(kind, count)
        big.fill(1)
        big.run()
        stream.synchronize()
    for b, g in zip(small, graphs):
        b.check(g, 5)


def test_stack_calls_in_a_capture(stream):
    """LibShalom_dgemm_stack: the front-end buffer (72 bytes a product) grows in a
    capture, and a graph keeps the one it names."""
    import torch
    m, n, k, many = 5, 4, 3, 30_000

    def call(count):
        g = torch.Generator(device="cuda").manual_seed(count)
        A, B = (torch.rand(count * x, generator=g, device="cuda", dtype=torch.float64)
                for x in (m * k, k * n))
        C = torch.zeros(count * m * n, device="cuda", dtype=torch.float64)
        offs = [torch.arange(count, device="cuda") * x for x in (m * k, k * n, m * n)]
        ref = torch.bmm(A.view(count, m, k), B.view(count, k, n)).reshape(-1)
        return C, ref, lambda: ls.dgemm_stack(A, B, C, *offs, count, m=m, n=n, k=k), (A, B, offs)

    graphs = []
    for count in (200, many):
        C, ref, run, keep = call(count)
        torch.cuda.synchronize()
        if count == 200:
            run()
            torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            run()
        graphs.append((C, ref, g, keep))
    big = call(2 * many)  # outgrows both
    torch.cuda.synchronize()
    big[2]()
    torch.cuda.synchronize()
    for C, ref, g, _ in graphs:
        C.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        # both sides: k roundings of sums of k terms below 1
        assert torch.max(torch.abs(C - ref)) <= 2 * k * k * 2.0 ** -53
