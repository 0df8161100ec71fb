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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,E,top,H", [(1, 1, 1, 8), (3, 8, 8, 264), (40, 9, 2, 1024), (777, 16, 2, 2048), (4099, 17, 1, 136), (600, 32, 16, 1032)])
@pytest.mark.parametrize("kind", ["plain", "biased", "corrected"])
def test_router_with_its_product(dtype, M, E, top, H, kind):
    from toyinfer_b200.kernels import moe as KM
    g = torch.Generator(device="cuda").manual_seed(M + E + H)
    x = torch.randn(M, H + 8, generator=g, device="cuda").to(dtype)[:, :H]
    w = (torch.randn(E, H, generator=g, device="cuda") / H ** 0.5).to(dtype)
    extra = 0.1 * torch.randn(E, generator=g, device="cuda")
    bias, corr = (extra if kind == "biased" else None), (extra if kind == "corrected" else None)
    z = x.double() @ w.double().T + (bias.double() if bias is not None else 0)
    s = torch.softmax(z, dim=1)
    c = s + corr if corr is not None else z
    ff = 64
    assert KM.route_rows_eligible(x, w, 0, top)
    perm, off, weight, plan = KM.route_rows(x, w, corr, top, 1.5, bias, ff)
    chosen = choose(c, top)
    want = 1.5 * s.gather(1, chosen) / s.gather(1, chosen).sum(1, keepdim=True)
    # sums of H products and an exponential in 32 bits; tokens whose choices lie within 1e-5 may fall either way
    order = torch.sort(c, dim=1, descending=True).values
    sure = (order[:, :-1] - order[:, 1:])[:, :top].amin(1) > 1e-5 if E > 1 else torch.ones(M, dtype=torch.bool, device="cuda")
    torch.testing.assert_close(weight.view(M, top).double()[sure], want[sure], rtol=1e-5, atol=0)
    assert (plan is not None) == (dtype == torch.bfloat16 and M * top >= KM.TC_MIN_GROUP * E)
    if plan is None:
        runs = perm.long(), off.long()
    else:
        pad_src, place, tile = plan
        assert torch.equal(pad_src[place.long()].long(), torch.arange(M * top, device="cuda") // top)
        assert int((pad_src >= 0).sum()) == M * top
        e_of = tile[place.long() // 128].long()
        runs = e_of.sort(stable=True).indices, torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), torch.bincount(e_of, minlength=E).cumsum(0)])
    perm, off = runs
    assert torch.equal(perm.sort().values, torch.arange(M * top, device="cuda"))
    for e in range(E):
        mine = torch.zeros(M * top, dtype=torch.bool, device="cuda")
        mine[perm[int(off[e]):int(off[e + 1])]] = True
        wrong = mine != (chosen.reshape(-1) == e)
        assert not (wrong.view(M, top) & sure[:, None]).any()


def test_router_with_its_product_not_a_number():
    """The lowest open expert is kept against every other where its score is not a number; elsewhere such a score never wins."""
    from toyinfer_b200.kernels import moe as KM
    x, w = torch.eye(8, device="cuda")[:3].contiguous(), torch.zeros(4, 8, device="cuda")
    nan = float("nan")
    w[:, 0] = torch.tensor([nan, 3.0, 2.0, 1.0])          # x = unit vectors: a row's logits are w's columns; 0 * nan reaches the others
    perm, off, _, _ = KM.route_rows(x[:1].contiguous(), w, None, 2, 1.0, None, 64)
    assert sorted(perm.tolist()) == [0, 1] and off.tolist() == [0, 1, 2, 2, 2]
    w[:, 0] = torch.tensor([0.0, nan, -0.0, -1.0])          # 0 wins over -0 as the lower index; then the lowest open one is no number
    perm, off, _, _ = KM.route_rows(x[:1].contiguous(), w, None, 2, 1.0, None, 64)
    assert off.tolist() == [0, 1, 2, 2, 2]
    w[:, 0] = torch.tensor([0.0, -1.0, nan, -0.0])          # where the lowest open one is a number, a score that is none never wins
    perm, off, _, _ = KM.route_rows(x[:1].contiguous(), w, None, 2, 1.0, None, 64)
    assert off.tolist() == [0, 1, 1, 1, 2]
    for column in w.T[:1].contiguous(), torch.tensor([[0.0, nan, -0.0, -1.0]], device="cuda"), torch.tensor([[nan, nan, 1.0, 2.0]], device="cuda"):
        w[:, 0] = column[0]
        got, want = KM.route_rows(x[:1].contiguous(), w, None, 2, 1.0, None, 64), KM.route_softmax(column, None, 4, 2)
        assert torch.equal(got[1], want[1]) and torch.equal(got[0], want[0])          # as the router of finished logits chooses


@pytest.mark.parametrize("M,E,H,takes", [(2048, 8, 4096, True), (1, 8, 4096, False), (1, 8, 2048, True), (1, 16, 4096, True), (2049, 16, 4096, False), (8192, 8, 2048, True), (8193, 8, 2048, False),
                                         (8193, 16, 2048, True), (8193, 32, 4096, True)])
def test_where_the_product_of_its_own_is_faster(M, E, H, takes):
    from toyinfer_b200.kernels import moe as KM
    x, w = torch.empty(M, H, dtype=torch.bfloat16, device="cuda"), torch.empty(E, H, dtype=torch.bfloat16, device="cuda")
    assert KM.route_rows_eligible(x, w, 0, 2) == takes
    assert KM.route_rows_eligible(x.float(), w.float(), 0, 2)
