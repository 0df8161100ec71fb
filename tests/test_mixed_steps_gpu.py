"""Steps in which long and short sequences meet (kernels/recurrent.py: in_chunks): long ones go in chunks, the others token by token
beside them, and every sequence's result is what it is on its own.  And the rule that shares a step out, on the CPU."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

import test_delta_chunk_gpu as delta
import test_ssd_chunk_gpu as ssd


def test_who_goes_in_chunks():
    from toyinfer_b200.kernels.recurrent import in_chunks
    step = lambda lens, known=True: SimpleNamespace(n_seq=len(lens), max_new=max(lens, default=0), host_new=lens if known else None)
    rule = lambda lens, known=True: in_chunks(step(lens, known), 32, 128, 148)
    assert rule([]) is None and rule([31]) is None and rule([32]) == 0 and rule([32] * 50) == 0
    assert rule([64, 1]) == 0                                     # a short one costs less than a second pass
    assert rule([40] + [1] * 8) is None                           # a chain of 40 tokens beside which the others cost little
    assert rule([512] + [1] * 32) == 32 and rule([2048] + [20] * 100) == 32
    assert rule([100] + [1] * 32) is None
    assert rule([512] * 33, known=False) == 32                    # lengths not known: all but one may be short
    assert rule([700], known=False) == 0


@pytest.fixture(scope="module")
def KR():
    from toyinfer_b200.kernels import recurrent
    return recurrent


LENS = [[300, 1, 1, 40, 0, 1], [1, 5, 100, 31, 32, 33], [1, 0, 90, 0]]


@pytest.mark.gpu
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("least", [32, 33, 64])
@pytest.mark.parametrize("head", [True, False])
def test_delta(KR, monkeypatch, lens, least, head):
    args = delta.make(torch.bfloat16, head, 64, 64, 2, 1, lens, 3, True)
    want = delta.exact(*args, lens, head)
    monkeypatch.setattr(KR, "in_chunks", lambda *a: least)
    o, state = delta.run(KR, args, lens, head)
    monkeypatch.setattr(KR, "in_chunks", lambda *a: 0)
    chunks = delta.run(KR, args, lens, head)
    monkeypatch.setattr(KR, "in_chunks", lambda *a: None)
    scan = delta.run(KR, args, lens, head)
    at = 0
    for b, n in enumerate(lens):                                  # each sequence as the form it goes by makes it
        from_ = chunks if n >= least else scan
        assert torch.equal(o[at:at + n], from_[0][at:at + n]) and torch.equal(state[b], from_[1][b])
        at += n
    for got, w in zip((o, state), want):
        assert float((got.double() - w).norm() / w.norm()) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("lens", LENS)
@pytest.mark.parametrize("least", [80, 100])
def test_ssd(KR, monkeypatch, lens, least):
    H, G, N, V = 4, 2, 128, 64
    args = ssd.make(H, G, N, V, lens, 3, True)
    want = ssd.exact(args, H, G, N, V, lens)
    monkeypatch.setattr(KR, "SSD_SEGMENT", 1 << 20)               # the scan in one piece
    out = []
    for mode in (least, 0, None):
        monkeypatch.setattr(KR, "in_chunks", lambda *a: mode)
        out.append(ssd.run(KR, args, H, G, N, V, lens))
    (y, state), chunks, scan = out
    at = 0
    for b, n in enumerate(lens):
        from_ = chunks if n >= least else scan
        assert torch.equal(y[at:at + n], from_[0][at:at + n]) and torch.equal(state[b], from_[1][b])
        at += n
    for got, w in zip((y, state), want):
        assert float((got.double() - w).norm() / w.norm()) < 1e-6


@pytest.mark.gpu
def test_a_captured_step_with_other_lengths(KR):
    """What a graph was captured with says how the step is shared out, not what comes out."""
    H, d, M = 2, 64, 400
    lens = [[396, 1, 1, 2], [100, 100, 100, 100], [10, 300, 60, 30]]
    args = delta.make(torch.float32, True, d, d, H, H, [100] * 4, 9, False)
    q, k, v, decay, dt, rate, beta, state = args
    store, cu = torch.zeros(4, H * d * d, device="cuda"), torch.zeros(5, dtype=torch.int32, device="cuda")
    slots = torch.arange(4, dtype=torch.int32, device="cuda")
    fill = lambda ls: (cu.copy_(torch.tensor([0] + ls).cumsum(0)), store.copy_(state.reshape(4, -1)))
    for first in lens:
        batch = SimpleNamespace(cu_new=cu, seq_slot=slots, n_seq=4, max_new=396, host_new=first)
        step = lambda: KR.delta_rule(q, k, v, decay, dt, rate, beta, store, 0, batch, head_decay=True)
        fill(first)
        step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            o = step()
        for ls in lens:
            fill(ls)
            graph.replay()
            want, left = delta.exact(*args, ls, True)
            assert float((o.view(M, H, d).double() - want).norm() / want.norm()) < 1e-6
            assert float((store.view(left.shape).double() - left).norm() / left.norm()) < 1e-6
