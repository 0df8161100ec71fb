"""Draws over many blocks (csrc/sampling.cu): the same tokens as the form of one block per row, whatever the chunks hold, and with the
rows' keys and step counts as the launch's arguments or on the device."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rows(kind, R, V):
    g = torch.Generator(device="cuda").manual_seed(R + V)
    x = torch.randn(R, V + 5, generator=g, device="cuda")[:, :V] * 3
    if kind == "ties":                     # few distinct values: many entries reach any bound
        x = (x * 0.5).round()
    elif kind == "zeros":
        x = torch.where(x > 0, torch.zeros_like(x), -torch.zeros_like(x))
    elif kind == "masked":                 # most of a row out of the draw
        x = torch.where(torch.rand(R, V, generator=g, device="cuda") < 0.01, x, torch.full_like(x, -float("inf")))
        x[:, 0] = 1.0
    elif kind == "neighbours":             # logits a unit in the last place apart: quotients tie
        x = (1.0 + (x * 4).round() * 2.0 ** -23).contiguous()
    elif kind == "tiny":
        x = x * 1e-38
    return x


@pytest.mark.parametrize("kind", ["plain", "ties", "zeros", "masked", "neighbours", "tiny"])
@pytest.mark.parametrize("R,V", [(1, 5), (3, 4097), (64, 20000), (2, 151936)])
@pytest.mark.parametrize("top_k,top_p", [(1, 1.0), (20, 0.95), (25, 0.9), (64, 1.0), (65, 0.9), (0, 0.9), (0, 1.0)])
def test_the_same_draws(monkeypatch, kind, R, V, top_k, top_p):
    import toyinfer_b200.kernels as K
    if top_k >= V:
        pytest.skip("every entry is kept")
    x = rows(kind, R, V)
    keys, steps = np.arange(R, dtype=np.int64) * 7 - 3, np.arange(R, dtype=np.int32) % 5
    for T in (0.7, 1.0, 3.0):
        on_device = K.sample(x, T, top_k, top_p, 11, torch.from_numpy(keys).cuda(), torch.from_numpy(steps).cuda())
        by_value = K.sample_rows(x, T, top_k, top_p, 11, keys, steps)
        assert torch.equal(on_device, by_value)
        if top_k:                          # (without top_k the two forms add a row's exponentials up in another order)
            monkeypatch.setattr(K, "two_kernel_sampling", False)
            assert torch.equal(K.sample(x, T, top_k, top_p, 11, torch.from_numpy(keys).cuda(), torch.from_numpy(steps).cuda()), by_value)
            monkeypatch.setattr(K, "two_kernel_sampling", True)


def test_where_rows_do_not_go_with_the_launch():
    import toyinfer_b200.kernels as K
    x = torch.randn(300, 6000, device="cuda")
    keys, steps = np.arange(300, dtype=np.int64), np.zeros(300, dtype=np.int32)
    assert K.sample_rows(x, 1.0, 20, 0.9, 1, keys, steps) is None                    # more rows than the argument holds
    assert K.sample_rows(x[:5], 1.0, 2000, 0.9, 1, keys[:5], steps[:5]) is None      # one block per row
    K.sample_rows(x[:5], 1.0, 20, 0.9, 1, keys[:5], steps[:5])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        assert K.sample_rows(x[:5], 1.0, 20, 0.9, 1, keys[:5], steps[:5]) is None    # a capture
        x[:5] * 2


@pytest.mark.parametrize("kind", ["plain", "ties", "neighbours"])
@pytest.mark.parametrize("top_k", [32, 33, 63])
def test_merges_of_many_candidates(monkeypatch, kind, top_k):
    """Chunks enough for thousands of candidates, at the number of entries where the merge takes closer bounds."""
    import toyinfer_b200.kernels as K
    x = rows(kind, 5, 151936)
    keys, steps = np.arange(5, dtype=np.int64), np.arange(5, dtype=np.int32)
    got = K.sample_rows(x, 0.8, top_k, 0.97, 3, keys, steps)
    monkeypatch.setattr(K, "two_kernel_sampling", False)
    assert torch.equal(K.sample(x, 0.8, top_k, 0.97, 3, torch.from_numpy(keys).cuda(), torch.from_numpy(steps).cuda()), got)


@pytest.mark.parametrize("V", [1025, 4096, 4097, 8191, 20001])
@pytest.mark.parametrize("kind", ["plain", "ties", "masked"])
def test_ranks_beyond_the_first_candidates(kind, V):
    """A wide nucleus, walked tier by tier, at lengths around a turn of the block over the row: the token that the rule gives in 64 bits."""
    import toyinfer_b200.kernels as K
    x = rows(kind, 4, V) * 0.1 if kind != "masked" else rows(kind, 4, V)
    keys, steps = np.arange(4, dtype=np.int64), np.arange(4, dtype=np.int32)
    got = K.sample_rows(x, 1.0, 0, 0.97, 5, keys, steps).tolist()
    p = torch.softmax(x.double(), dim=1).cpu()
    for r in range(4):
        row = x[r].tolist()
        order = sorted(range(V), key=lambda i: (-row[i], i))
        run = torch.cumsum(p[r][order], 0)
        cut = int((run > 0.97).nonzero()[0])
        coin = K.uniform_from(5, int(keys[r]), int(steps[r])) * float(run[cut])
        at = int((run > coin).nonzero()[0])
        # (sums of up to 20,000 probabilities in 32 bits, one after another: an entry whose running sum lies within 1e-4 may be passed)
        near = {order[i] for i in range(max(0, at - 400), min(V, at + 400)) if abs(float(run[i]) - coin) < 1e-4 + float(p[r][order[i]])}
        assert got[r] in near | {order[at]}
