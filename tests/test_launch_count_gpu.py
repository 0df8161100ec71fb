"""The count of launches against the kernels of a captured graph, where it depends on the shape: the float32 product's pieces, the
short convolution's two forms, the CUDA-core decode attention's ways of merging its splits."""
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


@pytest.mark.parametrize("n_seq,length,kernels", [(1, 300, 1), (1, 2000, 1), (4, 2000, 2), (64, 300, 1), (3, 7000, 2)])
def test_decode_attention_clusters_only_where_all_find_room(n_seq, length, kernels):
    """24 heads of 128 over 4 in float32: one sequence's four clusters find room, four sequences' sixteen of eight blocks do not (as
    clusters they took 27.9 us, through scratch memory 17.2); one split, and more than sixteen."""
    from toyinfer_b200.kernels import attention
    pages = -(-length // 64)
    k = torch.randn(n_seq * pages, 4, 64, 128, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    mem = SimpleNamespace(k_pages=k, v_pages=k, page_table=torch.arange(n_seq * pages, **i32).view(n_seq, pages), page_size=64, ring_rows=0, n_kv_heads=4)
    batch = SimpleNamespace(plan_len=length, n_real_seq=n_seq, seq_slot=torch.arange(n_seq, **i32), seq_len=torch.full((n_seq,), length, **i32))
    q = torch.randn(n_seq, 24, 128, device="cuda")
    out = torch.empty_like(q)
    assert counted_and_captured(lambda: attention.decode(q, mem, out, 0.1, 0, batch)) == (kernels, kernels)
