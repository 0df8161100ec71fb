"""The quotient behind sigmoids and silu (ti_over, csrc/common.cuh) through the elementwise activations: silu within 6 x 2^-24 of 64 bits
over the whole range, and the limits, signs of zeros among them, as the arithmetic of IEEE 754 gives them."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def silu(z):
    """silu(z) times one, by the elementwise activation of dense rows (gate, up)."""
    import toyinfer_b200.kernels as K
    return K.swiglu(torch.cat([z, torch.ones_like(z)], dim=1))


def test_float32_over_the_range():
    g = torch.Generator(device="cuda").manual_seed(1)
    z = torch.cat([torch.randn(1 << 20, generator=g, device="cuda") * s for s in (0.01, 1.0, 10.0, 30.0)]).clamp(-85, 300).view(-1, 64).contiguous()
    got, x = silu(z).double(), z.double()
    want = x / (1 + torch.exp(-x))
    # the exponential (two units in the last place, times at most one where it counts fully), one addition, one quotient, two products
    assert ((got - want).abs() <= 6 * 2.0 ** -24 * want.abs() + 1e-37).all()


def test_limits():
    z = torch.tensor([[float("inf"), -float("inf"), float("nan"), 0.0, -0.0, -100.0, -88.6, 3.0e38, -3.0e38, 1e-40]], device="cuda")
    got = silu(z)[0].tolist()
    assert got[0] == float("inf") and got[1] != got[1] and got[2] != got[2]
    assert got[3] == 0.0 and got[4] == 0.0 and abs(got[5]) < 1e-35 and abs(got[6]) < 1e-35 and got[7] == pytest.approx(3.0e38, rel=1e-6) and got[8] == 0.0
    assert 0 <= got[9] <= 1e-40


def test_signs_of_zeros():
    z = torch.tensor([[0.0, -0.0, -200.0, 200.0, -1e-45, 1e-45]], device="cuda")
    assert torch.signbit(silu(z)[0]).tolist() == [False, True, True, False, True, False]
