"""Deep products captured into a graph on a stream that holds no workspace yet: nothing can be allocated
there, so they run without a K split. Entries are small integers: the result is exact either way."""
from __future__ import annotations

import pytest
import torch

from remora_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 128, 8192), (70, 9, 2100), (640, 700, 4096)])
def test_capture_of_a_deep_product(cuda, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(k)
    A = torch.randint(-4, 5, (m, k), generator=g, device="cuda").double()
    B = torch.randint(-4, 5, (k, n), generator=g, device="cuda").double()
    C = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    want = (A.cpu() @ B.cpu()).cuda()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        ops.gemm(A, B, C, 1.0, 0.0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(C, want)
    del graph
    C.zero_()
    ops.gemm(A, B, C, 1.0, 0.0)  # split, where the model says so
    assert torch.equal(C, want)
