"""The grouped products from registers (csrc/moe_rows.cuh) at the edges of their tiles: groups of 0, 1, TM and TM + 1 places, more than
32 experts, contractions that end inside a lane's piece, rows off the 16-byte boundary, and the tensor-core tiles beside them."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def run(dtype, counts, H, ff, top, bound, shift=0):
    from toyinfer_b200.kernels import moe as KM
    E, pairs = len(counts), sum(counts)
    assert pairs % top == 0
    g = torch.Generator(device="cuda").manual_seed(pairs + H)
    n = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)
    x = n(pairs // top, H + 8 + shift)[:, shift:shift + H]
    w1, w2 = n(E, 2 * ff, H, std=H ** -0.5), n(E, H, ff, std=ff ** -0.5)
    perm = torch.randperm(pairs, generator=g, device="cuda").to(torch.int32)
    off = torch.tensor([0] + counts, device="cuda").cumsum(0).to(torch.int32)
    z, place, padded = KM.expert_pairs(x, perm, off, w1, w2, top, float("inf"), 1.0, 0.0)
    assert place is None and not padded
    e_of = torch.empty(pairs, dtype=torch.long, device="cuda")
    e_of[perm.long()] = torch.repeat_interleave(torch.arange(E, device="cuda"), torch.tensor(counts, device="cuda"))
    want = torch.empty(pairs, H, dtype=torch.float64, device="cuda")
    for p0 in range(0, pairs, 256):
        e = e_of[p0:p0 + 256]
        xx = x[torch.arange(p0, min(p0 + 256, pairs), device="cuda") // top].double()
        gu = torch.einsum("ph,pfh->pf", xx, w1[e].double())
        y = torch.nn.functional.silu(gu[:, :ff]) * gu[:, ff:]
        want[p0:p0 + 256] = torch.einsum("pf,phf->ph", y, w2[e].double())
    assert ((z.double() - want).norm(dim=1) <= bound * want.norm(dim=1)).all()


# 32 bits: sums of up to 2,048 products, at most 64 of which follow one another, twice, and an exponential
F32 = 2e-6
# bfloat16: gate, up, their product and the result are each rounded to 2^-9
BF16 = 1.2e-2


@pytest.mark.parametrize("counts,H,ff,top", [([1], 64, 8, 1), ([0, 8, 9, 0, 7], 264, 36, 2), ([16, 17, 1, 33, 15, 0], 1024, 392, 2),
                                             ([1] * 40 + [0] * 30 + [3, 1], 520, 100, 4), ([150, 170], 256, 260, 4)])
def test_float32(counts, H, ff, top):
    run(torch.float32, counts, H, ff, top, F32)


@pytest.mark.parametrize("counts,H,ff", [([5, 0, 12], 70, 13), ([40, 2], 264, 33)])
def test_float32_off_the_boundary(counts, H, ff):
    run(torch.float32, counts, H, ff, 1, F32, shift=1)


@pytest.mark.parametrize("counts,H,ff,top", [([1], 64, 8, 1), ([0, 8, 9, 0, 7], 264, 40, 2), ([16, 17, 1, 33, 15, 0], 1024, 392, 2),
                                             ([2] * 33, 2048, 72, 1), ([24, 26, 22], 520, 104, 3), ([31, 64, 65, 0], 136, 200, 1), ([3, 2], 8, 16, 1)])
def test_bfloat16(counts, H, ff, top):
    run(torch.bfloat16, counts, H, ff, top, BF16)


def test_bfloat16_off_the_boundary():
    run(torch.bfloat16, [5, 0, 12], 70, 13, 1, BF16, shift=1)


@pytest.mark.parametrize("counts,H,ff", [([900, 1, 0, 650, 33, 32], 70, 1003), ([1300], 513, 900)])
def test_many_places_off_the_boundary(counts, H, ff):
    """Staged tiles for the first product (more than seven blocks an SM), either form for the second."""
    run(torch.float32, counts, H, ff, 1, F32, shift=1)
    run(torch.bfloat16, counts, H, ff, 1, BF16, shift=1)
