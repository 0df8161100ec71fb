"""The few-row float32 product at the edges of its tiles: 1 to 16 tokens in passes of 1, 2, 4 and 8, weight rows that end inside a group of
four, contractions that end inside a warp's turn or leave slices without work, both matrix sizes, plain and gated."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 4), (2, 100), (7, 132), (386, 96), (1030, 516), (130, 4100), (6, 131072), (9730, 260)]


def operands(M, N, Kd):
    g = torch.Generator(device="cuda").manual_seed(M * N + Kd)
    x = torch.randn(M, Kd + 4, generator=g, device="cuda")[:, :Kd]
    return x, torch.randn(N, Kd + 8, generator=g, device="cuda")[:, :Kd] / Kd ** 0.5


# sums of up to 131,072 products, of which a lane adds up 512 in four chains' worth, then a tree: 32 bits
BOUND = 2e-6


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("N,Kd", SHAPES)
def test_product(M, N, Kd):
    import toyinfer_b200.kernels as K
    x, w = operands(M, N, Kd)
    out, want = K.linear(x, w).double(), x.double() @ w.double().T
    assert ((out - want).norm() <= BOUND * x.double().norm() * w.double().norm() / Kd ** 0.5)
    assert (out - want).abs().max() <= 1e-5 * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("M", [1, 2, 3, 7, 16])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clamped_swish"])
@pytest.mark.parametrize("N,Kd", [s for s in SHAPES if s[0] % 2 == 0])
def test_gated(M, N, Kd, act):
    import toyinfer_b200.kernels as K
    x, w = operands(M, N, Kd)
    got = K.linear_swiglu(x, w, act, 1.5) if act == "clamped_swish" else K.linear_swiglu(x, w, act)
    gu = x.double() @ w.double().T
    g, u = gu[:, 0::2], gu[:, 1::2]
    if act == "silu":
        want = u * g / (1 + torch.exp(-g))
    elif act == "gelu_tanh":
        want = u * torch.nn.functional.gelu(g, approximate="tanh")
    else:
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        want = g * torch.sigmoid(1.702 * g) * (u + 1)
    assert (got.double() - want).abs().max() <= 2e-5 * max(1.0, float(want.abs().max()))
