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
