"""The routers of few experts (csrc/moe_router.cu) at the edges of their bounds, against a plain choice in 64 bits: the same experts,
weights within rounding, every pair once and in its expert's run; and the padded plan of the grouped product made from them."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def logits(M, E, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.randn(M, E + 3, generator=g, device="cuda")[:, :E]
    z[::7, 0] = z[::7, E - 1]                       # ties go to the lower index
    return z


def check_groups(perm, off, chosen, E):
    M, top = chosen.shape
    assert off[0] == 0 and off[-1] == M * top
    flat = chosen.reshape(-1)
    assert torch.equal(perm.sort().values, torch.arange(M * top, dtype=torch.int32, device="cuda"))
    for e in range(E):
        run = perm[int(off[e]):int(off[e + 1])].long()
        assert torch.equal(run.sort().values, (flat == e).nonzero()[:, 0])


def choose(c, top):
    """The ``top`` largest of every row, the lower index first among equals."""
    return torch.sort(c, dim=1, descending=True, stable=True).indices[:, :top]


@pytest.mark.parametrize("M,E,top", [(1, 1, 1), (5, 8, 8), (33, 9, 2), (1023, 16, 4), (1025, 17, 1), (2100, 32, 16), (64, 33, 3)])
@pytest.mark.parametrize("kind", ["softmax", "corrected", "biased", "sigmoid"])
def test_choices_and_runs(M, E, top, kind):
    from toyinfer_b200.kernels import moe as KM
    z = logits(M, E, M + E)
    g = torch.Generator(device="cuda").manual_seed(3)
    extra = 0.1 * torch.randn(E, generator=g, device="cuda")
    zz = z.double()
    if kind == "sigmoid":
        perm, off, w, w2 = KM.route_topk(z, E, top)
        chosen = choose(z, top)
        want = torch.sigmoid(zz.gather(1, chosen))
        torch.testing.assert_close(w2.view(M, top).double(), want * want, rtol=2e-6, atol=0)
    else:
        bias, corr = (extra if kind == "biased" else None), (extra if kind == "corrected" else None)
        perm, off, w = KM.route_softmax(z, corr, E, top, scale=1.5, logit_bias=bias)
        zb = z + bias if bias is not None else z
        s = torch.softmax(zb.double(), dim=1)
        # (in 32 bits, where ties are decided)
        chosen = choose(zb, top) if corr is None else choose((torch.exp(zb - zb.max(1, keepdim=True).values).double()
                                                              / torch.exp((zb - zb.max(1, keepdim=True).values).double()).sum(1, keepdim=True)).float() + corr, top)
        want = s.gather(1, chosen)
        want = 1.5 * want / want.sum(1, keepdim=True)
    got = w.view(M, top).double()
    off_by = ((got - want).abs() / want).amax(1)
    # a corrected choice may meet another rounding of its sums: a token whose order differs is one in a thousand at most
    assert (off_by > 1e-5).float().mean() <= (1e-3 if kind == "corrected" else 0.0)
    if kind != "corrected":
        check_groups(perm, off, chosen, E)


@pytest.mark.parametrize("counts", [[1], [128, 0, 129], [0, 0, 700, 1, 0], [5] * 40])
def test_padded_plan(counts):
    from toyinfer_b200.kernels import _call, _ptr, _stream
    from toyinfer_b200.kernels.moe import I, P, _fn
    E, n = len(counts), sum(counts)
    off = torch.tensor([0] + counts, device="cuda").cumsum(0).to(torch.int32)
    perm = torch.randperm(n, device="cuda").to(torch.int32)
    rows = (n + 127 * E + 127) // 128 * 128
    src, place, tile = (torch.empty(k, dtype=torch.int32, device="cuda") for k in (rows, n, rows // 128))
    _call(_fn("ti_moe_pad_plan", [P, P, I, I, I, I, P, P, P, P]), _ptr(perm), _ptr(off), E, n, 1, rows, _ptr(src), _ptr(place), _ptr(tile), _stream())
    at, want_src, want_tile = 0, torch.full((rows,), -1, dtype=torch.int32), torch.full((rows // 128,), -1, dtype=torch.int32)
    for e, c in enumerate(counts):
        want_src[at:at + c] = perm[int(off[e]):int(off[e + 1])].cpu()
        pad = (c + 127) // 128
        want_tile[at // 128:at // 128 + pad] = e
        at += 128 * pad
    assert torch.equal(src.cpu(), want_src) and torch.equal(tile.cpu(), want_tile)
    assert torch.equal(src[place.long()], torch.arange(n, dtype=torch.int32, device="cuda"))
