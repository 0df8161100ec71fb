"""One token per sequence through a recurrent layer's state (csrc/state_step.cu) against 64 bits and against the scans that serve
every other step: the sizes it takes, slots out of order, heads that share queries, decays of both kinds, rows that are nobody's."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
SIZES = [(64, 64, 2, 1, 1), (64, 128, 3, 3, 5), (128, 64, 4, 2, 3), (128, 128, 16, 16, 33)]      # dim, vdim, heads, query heads, sequences


def batch_of(n, longest):
    """n sequences of a token each; ``longest`` 2 sends the step to the scan."""
    g = torch.Generator(device="cuda").manual_seed(n)
    return SimpleNamespace(cu_new=torch.arange(n + 1, dtype=torch.int32, device="cuda"), n_seq=n, n_tok=n, max_new=longest,
                           seq_slot=torch.randperm(n + 2, generator=g, device="cuda")[:n].to(torch.int32))


def rnd(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, generator=g, device="cuda")


def close(got, scan, want):
    off = lambda x: float((x.double() - want).norm() / want.norm())
    assert off(got) <= max(1.5 * off(scan), 2e-7), (off(got), off(scan))      # the same sums in another order


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,dv,H,G,n", SIZES)
@pytest.mark.parametrize("act,k_scale", [("silu", 1.0), ("none", 0.25)])
def test_lightning(dtype, d, dv, H, G, n, act, k_scale):
    from toyinfer_b200.kernels import lightning as KS
    r = rnd(d + dv + n)
    rows = r(n, H * (2 * d + dv)).to(dtype)
    q, k, v = rows[:, :H * d].view(n, H, d), rows[:, H * d:2 * H * d].view(n, H, d), rows[:, 2 * H * d:].view(n, H, dv)
    decay, state = torch.rand(H, device="cuda"), r(n + 3, H, d, dv)
    at = batch_of(n, 1).seq_slot.long()
    f = (lambda x: x.double() / (1 + torch.exp(-x.double()))) if act == "silu" else (lambda x: x.double())
    S = decay.double()[:, None, None] * state[at].double() + (f(k) * k_scale)[..., None] * f(v)[:, :, None]
    o = torch.einsum("nhdv,nhd->nhv", S, f(q)).reshape(n, -1)
    out = []
    for longest in (1, 2):
        st = state.clone()
        out.append((KS.mix(q, k, v, st, decay, batch_of(n, longest), act=act, k_scale=k_scale), st))
    close(out[0][0], out[1][0], o)
    close(out[0][1][at], out[1][1][at], S)
    rest = torch.ones(n + 3, dtype=torch.bool)
    rest[at.cpu()] = False
    assert torch.equal(out[0][1][rest], state[rest])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d,dv,H,G,n", SIZES)
@pytest.mark.parametrize("head", [True, False])
def test_delta(dtype, d, dv, H, G, n, head):
    from toyinfer_b200.kernels import recurrent as KR
    r = rnd(d + dv + n + 1)
    M = n + 3                                                # the last rows are nobody's
    rows = r(M, 2 * G * d + H * dv + 8).to(dtype)
    q, k, v = rows[:, :G * d].view(M, G, d), rows[:, G * d:2 * G * d].view(M, G, d), rows[:, 2 * G * d:2 * G * d + H * dv].view(M, H, dv)
    decay = r(M, H).to(dtype) if head else r(M, H * d)
    decay[0] = 2000.0                                        # one sequence forgets everything
    dt, rate, beta = r(H if head else H * d) - 2.0, torch.exp(0.5 * r(H)), r(M, H).to(dtype)
    state = r(n + 3, 4 + H * d * dv)
    at = batch_of(n, 1).seq_slot.long()
    unit = lambda x: (x[:n].double() / torch.sqrt((x[:n].double() ** 2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    soft = torch.nn.functional.softplus(decay[:n].double() + dt.double(), threshold=100)
    g = torch.exp(-rate.double()[:, None] * (soft[:, :, None].expand(-1, H, d) if head else soft.view(n, H, d)))
    S = g[..., None] * state[at, 4:].double().view(n, H, d, dv)
    e = torch.sigmoid(beta[:n].double())[..., None] * (v[:n].double() - torch.einsum("nhdv,nhd->nhv", S, unit(k)))
    S = S + unit(k)[..., None] * e[:, :, None]
    o = torch.einsum("nhdv,nhd->nhv", S, unit(q) * d ** -0.5).reshape(n, -1)
    out = []
    for longest in (1, 2):
        st = state.clone()
        out.append((KR.delta_rule(q, k, v, decay, dt, rate, beta, st, 4, batch_of(n, longest), head_decay=head), st))
    close(out[0][0][:n], out[1][0][:n], o)
    close(out[0][1][at, 4:].view(S.shape), out[1][1][at, 4:].view(S.shape), S)
    assert not out[0][0][n:].any() and torch.equal(out[0][1][:, :4], state[:, :4])


@pytest.mark.parametrize("longest", [0, 1, 100])
def test_a_step_of_no_sequences(longest):
    """Rows that are nobody's are zero though no kernel runs."""
    from toyinfer_b200.kernels import recurrent as KR
    batch = SimpleNamespace(cu_new=torch.zeros(1, dtype=torch.int32, device="cuda"), seq_slot=torch.zeros(0, dtype=torch.int32, device="cuda"),
                            n_seq=0, n_tok=0, max_new=longest)
    r = rnd(1)
    state = torch.zeros(2, 2 * 64 * 64, device="cuda")

    def call(fn, shape, dtype):
        poison = torch.full(shape, float("nan"), dtype=dtype, device="cuda")       # what the result's memory holds before
        del poison
        y = fn()
        assert y.shape == shape and not y.any()

    call(lambda: KR.short_conv(r(5, 128).to(torch.bfloat16), r(128, 4), state, 0, batch), (5, 128), torch.bfloat16)
    call(lambda: KR.delta_rule(r(5, 2, 64), r(5, 2, 64), r(5, 2, 64), r(5, 2), r(2), r(2), r(5, 2), state, 0, batch, head_decay=True), (5, 128), torch.float32)
    call(lambda: KR.ssd_scan(r(5, 128 + 128).to(torch.bfloat16), r(5, 2).to(torch.bfloat16), r(2), r(2), None, 2, 1, 64, 64, state, 0, batch), (5, 128),
         torch.float32)
