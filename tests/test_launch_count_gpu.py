"""The count of launches against the kernels of a captured graph, where it depends on the shape: the float32 product's pieces and
the short convolution's two forms."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def counted_and_captured(fn):
    from cuda.bindings import runtime as rt
    import toyinfer_b200.kernels as K
    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        before = K.launch_count
        fn()
        counted = K.launch_count - before
    raw = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    _, _, n = rt.cudaGraphGetNodes(raw)
    _, nodes, n = rt.cudaGraphGetNodes(raw, n)
    kinds = [rt.cudaGraphNodeGetType(node)[1] for node in nodes[:n]]
    return counted, sum(k == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for k in kinds)


@pytest.mark.parametrize("M,N,Kd,kernels", [(40, 256, 64, 1), (40, 256, 2560, 2), (300, 74 * 128, 96, 1), (500, 2560, 9728, 2)])
def test_float32_product(M, N, Kd, kernels):
    import toyinfer_b200.kernels as K
    x, w = torch.randn(M, Kd, device="cuda"), torch.randn(N, Kd, device="cuda")
    assert counted_and_captured(lambda: K.linear(x, w)) == (kernels, kernels)


@pytest.mark.parametrize("taps", [1, 4, 5])
@pytest.mark.parametrize("n", [1, 16, 17, 64, 65])
@pytest.mark.parametrize("pad", [4, 3])
def test_short_conv(taps, n, pad):
    from toyinfer_b200.kernels import recurrent as KR
    C = 64
    x = torch.randn(n, C + pad, device="cuda")[:, :C]
    w, state = torch.randn(C, taps, device="cuda"), torch.zeros(1, max(4, (taps - 1) * C), device="cuda")
    batch = SimpleNamespace(cu_new=torch.tensor([0, n], dtype=torch.int32, device="cuda"), seq_slot=torch.zeros(1, dtype=torch.int32, device="cuda"),
                            n_seq=1, max_new=n)
    kernels = 2 if taps > 1 and n > (16 if taps <= 4 and pad == 4 else 64) else 1
    assert counted_and_captured(lambda: KR.short_conv(x, w, state, 0, batch)) == (kernels, kernels)
