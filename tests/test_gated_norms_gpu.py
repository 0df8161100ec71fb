"""The gated norms' wide forms (a thread holds eight values of its row) and the widths and strides that take the general form, against
64 bits: csrc/lightning.cu, csrc/delta_rule.cu, csrc/ssd_scan.cu.  And the short convolution's (csrc/short_conv.cu), against its own
general form on rows that are not aligned."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DT = [torch.float32, torch.bfloat16]


def rnd(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda")


def strided(x, dtype, extra):
    """``x`` as columns of wider rows: with ``extra`` a multiple of 8 they stay aligned, else not."""
    wide = torch.zeros(x.shape[0], x.shape[1] + extra, dtype=dtype, device="cuda")
    wide[:, :x.shape[1]] = x
    return wide[:, :x.shape[1]]


def close(got, want, dtype):
    # float32: a few roundings of some 20 operations; bfloat16: the result's own rounding
    tol = dict(rtol=4e-6, atol=1e-6) if dtype == torch.float32 else dict(rtol=2.0 ** -8, atol=1e-6)
    torch.testing.assert_close(got.double(), want, **tol)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("extra", [8, 3])
@pytest.mark.parametrize("M,N", [(1, 256), (33, 2048), (3, 8192), (5, 8448), (7, 1000)])
def test_gated_rmsnorm(dtype, M, N, extra):
    from toyinfer_b200.kernels import lightning as KS
    o, g, w = rnd(M, N), strided(rnd(M, N, seed=1) * 3, dtype, extra), rnd(N, seed=2)
    want = o.double() / torch.sqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(g.double())
    close(KS.gated_rmsnorm(o, g, w, 1e-5), want, dtype)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("extra", [8, 3])
@pytest.mark.parametrize("M,H,V", [(1, 1, 8), (5, 3, 64), (33, 16, 128), (2, 7, 256), (9, 2, 96), (3, 2, 512)])
@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_head_gated_rmsnorm(dtype, M, H, V, extra, act):
    from toyinfer_b200.kernels import recurrent as KR
    o, g, w = rnd(M, H * V), strided(rnd(M, H * V, seed=1) * 3, dtype, extra), rnd(V, seed=2)
    x = o.double().view(M, H, V)
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()
    gate = torch.sigmoid(g.double()) * (g.double() if act == "silu" else 1.0)
    close(KR.head_gated_rmsnorm(o, g, w, H, 1e-5, gate_act=act), y.reshape(M, -1) * gate, dtype)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("extra", [8, 3])
@pytest.mark.parametrize("M,parts,size", [(1, 1, 256), (5, 8, 512), (33, 3, 2048), (2, 1, 8192), (3, 2, 8448), (7, 4, 100)])
def test_gate_group_rmsnorm(dtype, M, parts, size, extra):
    from toyinfer_b200.kernels import recurrent as KR
    N = parts * size
    y, z, w = rnd(M, N), strided(rnd(M, N, seed=1) * 3, dtype, extra), rnd(N, seed=2)
    u = (y.double() * z.double() * torch.sigmoid(z.double())).view(M, parts, size)
    want = (u / torch.sqrt((u * u).mean(-1, keepdim=True) + 1e-5)).reshape(M, N) * w.double()
    close(KR.gate_group_rmsnorm(y, z, w, parts, 1e-5), want, dtype)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("taps", [1, 2, 4])
@pytest.mark.parametrize("C,lens", [(4, [1, 2, 3]), (520, [16, 17, 1]), (1028, [100, 33])])
def test_short_conv(dtype, taps, C, lens):
    from toyinfer_b200.kernels import recurrent as KR
    n, M = len(lens), sum(lens) + 2                          # two rows are nobody's
    x, w, ib, ob = rnd(M, C), rnd(C, taps, seed=1), rnd(C, seed=2), rnd(C, seed=3)
    x = x.to(dtype)
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_new=cu, seq_slot=torch.arange(n, dtype=torch.int32, device="cuda"), n_seq=n, max_new=max(lens))
    state = rnd(n + 1, (taps - 1) * C + 4, seed=4)
    out = []
    for extra, offset in ((8, 4), (3, 0)):
        st = state.clone() if offset else torch.cat([state[:, 4:], state[:, :4]], 1).contiguous()
        out.append((KR.short_conv(strided(x, dtype, extra), w, st, offset, batch, in_bias=ib, out_bias=ob, act="silu"), st[:, offset:offset + (taps - 1) * C]))
    (a, sa), (b, sb) = out
    assert torch.equal(sa, sb) and not a[sum(lens):].any() and not b[sum(lens):].any()
    assert torch.equal(a, b)


FAR = [-88.5, -88.0, -87.5, -87.0, -40.0, 0.0, 40.0, 88.0]        # exp(-z) up to the end of float32's range


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("extra", [8, 3])
def test_gates_far_out(dtype, extra):
    """Whatever form a row takes: the exact quotient, also where exp(-z) is close to the largest float32."""
    from toyinfer_b200.kernels import lightning as KS, recurrent as KR
    M, V = 3, 256
    z = torch.tensor(FAR, device="cuda").repeat(M, V // len(FAR))
    gate, o, w = strided(z, dtype, extra), rnd(M, V).abs() + 0.1, torch.ones(V, device="cuda")
    zz = gate.double()
    silu, sigmoid = zz * torch.sigmoid(zz), torch.sigmoid(zz)
    rms = lambda x: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5)
    near = lambda got, want: torch.testing.assert_close(got.double(), want, rtol=2e-6 if dtype == torch.float32 else 2.0 ** -8, atol=3e-38)
    near(KR.head_gated_rmsnorm(o, gate, w, 1, 1e-5, gate_act="silu"), rms(o.double()) * silu)
    near(KR.head_gated_rmsnorm(o, gate, w, 1, 1e-5), rms(o.double()) * sigmoid)
    near(KR.gate_group_rmsnorm(o, gate, w, 1, 1e-5), rms(o.double() * silu))
    near(KS.gated_rmsnorm(o, gate, w, 1e-5), rms(o.double()) * sigmoid)
    cu = torch.tensor([0, M], dtype=torch.int32, device="cuda")
    batch = SimpleNamespace(cu_new=cu, seq_slot=torch.zeros(1, dtype=torch.int32, device="cuda"), n_seq=1, max_new=M)
    near(KR.short_conv(gate, torch.ones(V, 1, device="cuda"), torch.zeros(1, 4, device="cuda"), 0, batch, act="silu"), silu)
