"""The padded groups' product with its activation at the end (csrc/gemm_tcgen05_grouped.cu), against 64 bits: columns that do not fill a
tile, groups without rows, few tiles and more than the SMs hold at a time."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def places(M, E, top):
    g = torch.Generator().manual_seed(M + E)
    choice = torch.stack([torch.randperm(max(E - 1, top), generator=g)[:top] for _ in range(M)])       # (the last group is empty where it may be)
    expert = choice.reshape(-1)
    perm = torch.argsort(expert, stable=True)
    off = torch.zeros(E + 1, dtype=torch.int64)
    off[1:] = torch.bincount(expert, minlength=E).cumsum(0)
    return expert, perm.to(torch.int32).cuda(), off.to(torch.int32).cuda()


@pytest.mark.parametrize("M,E,top,H,ff", [(130, 2, 1, 64, 8), (257, 3, 2, 72, 72), (200, 4, 2, 136, 200), (700, 8, 2, 256, 1000), (900, 4, 3, 128, 64), (64, 1, 1, 64, 64), (2500, 4, 2, 1024, 256)])
@pytest.mark.parametrize("act", ["silu", "clamped", "relu2"])
def test_against_64_bits(M, E, top, H, ff, act):
    from toyinfer_b200.kernels import moe as KM, check_status
    g = torch.Generator(device="cuda").manual_seed(ff)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    x, F = r(M, H), torch.float64
    expert, perm, off = places(M, E, top)
    up = r(E, ff if act == "relu2" else 2 * ff, H) * H ** -0.5
    down = r(E, H, ff) * ff ** -0.5
    if act == "relu2":
        z, place = KM.experts_relu2(x, perm, off, up, down, top)
    else:
        limit, alpha, shift = (float("inf"), 1.0, 0.0) if act == "silu" else (0.7, 1.702, 1.0)
        z, place, padded = KM.expert_pairs(x, perm, off, up, down, top, limit, alpha, shift)
        assert padded
    check_status()
    got = z[place.long()].to(F)
    want = torch.empty(M * top, H, dtype=F, device="cuda")
    for e in range(E):
        pairs = (expert == e).nonzero().flatten().cuda()
        u = x[pairs // top].to(F) @ up[e].to(F).T
        if act == "relu2":
            y = u.clamp(min=0) ** 2
        else:
            a, b = u[:, :ff].clamp(max=limit), u[:, ff:].clamp(-limit, limit)
            y = a * torch.sigmoid(alpha * a) * (b + shift)
        want[pairs] = y @ down[e].to(F).T
    # two roundings to bfloat16, of the activation and of the result: 2^-9 each at most
    assert float((got - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("act", ["silu", "clamped"])
def test_products_are_rounded_before_the_activation(act):
    """An identity as the second matrix leaves the activated products as they are: those of products rounded to bfloat16, the values
    that groups of fewer places give."""
    from toyinfer_b200.kernels import moe as KM, check_status
    M, E, H = 300, 2, 256
    g = torch.Generator(device="cuda").manual_seed(9)
    x, F = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16), torch.float64
    expert, perm, off = places(M, E, 1)
    up = (torch.randn(E, 2 * H, H, generator=g, device="cuda") * H ** -0.5).to(torch.bfloat16)
    down = torch.eye(H, device="cuda").to(torch.bfloat16).expand(E, H, H).contiguous()
    limit, alpha, shift = (float("inf"), 1.0, 0.0) if act == "silu" else (0.7, 1.702, 1.0)

    def run(rows):
        """The pairs' rows in the tokens' order, for the first ``rows`` tokens."""
        order = perm[perm < rows].contiguous()
        at = torch.tensor([0] + torch.bincount(expert[:rows], minlength=E).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        z, place, padded = KM.expert_pairs(x[:rows], order, at, up, down, 1, limit, alpha, shift)
        assert padded == (rows == M)
        check_status()
        return z if place is None else z[place.long()]

    got = run(M)
    u = torch.stack([x[m].to(F) @ up[expert[m]].to(F).T for m in range(M)]).to(torch.bfloat16).to(F)
    a, b = u[:, :H].clamp(max=limit), u[:, H:].clamp(-limit, limit)
    want = a * torch.sigmoid(alpha * a) * (b + shift)
    # a sum in 32 bits within 2^-20 of its terms' size falls on the other side of a rounding to 8 bits in fewer than one case of a
    # hundred, for either of two products and for the result; without the rounding before the activation a third and more differ
    assert float((got != want.to(torch.bfloat16)).float().mean()) < 0.03
    few = run(40)
    assert float((got[:40] != few).float().mean()) < 0.03


def test_the_squared_relu_takes_products_in_32_bits():
    """As above for the experts whose activation is the squared ReLU: every form squares the products before they are rounded."""
    from toyinfer_b200.kernels import moe as KM, check_status
    M, E, H = 300, 2, 256
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn(M, H, generator=g, device="cuda").to(torch.bfloat16)
    expert, perm, off = places(M, E, 1)
    up = (torch.randn(E, H, H, generator=g, device="cuda") * H ** -0.5).to(torch.bfloat16)
    down = torch.eye(H, device="cuda").to(torch.bfloat16).expand(E, H, H).contiguous()
    want = torch.stack([(x[m].double() @ up[expert[m]].double().T).clamp(min=0) ** 2 for m in range(M)]).to(torch.bfloat16)
    # padded; tiles of some tens of places; from registers, several and one an expert
    for rows in (300, 90, 40, 6, 1):
        order = perm[perm < rows].contiguous()
        at = torch.tensor([0] + torch.bincount(expert[:rows], minlength=E).cumsum(0).tolist(), dtype=torch.int32, device="cuda")
        z, place = KM.experts_relu2(x[:rows], order, at, up, down, 1)
        check_status()
        got = z if place is None else z[place.long()]
        # (sums within 2^-20 fall on another side of a rounding to 8 bits in fewer than one case of a hundred)
        assert float((got != want[:rows]).float().mean()) < 0.03
