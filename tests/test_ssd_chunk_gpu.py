"""The Mamba-2 recurrence in chunks (csrc/ssd_chunk.cu) against 64 bits and against the token-by-token scan: at edges of its
chunks and tiles, several sequences, strided rows, decays from none to total and states that are not zero."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def KR():
    from toyinfer_b200.kernels import recurrent
    return recurrent


def make(H, G, N, V, lens, seed, strong=False):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    M = sum(lens)
    rows = r(M, H * V + 2 * G * N + H + (-H % 8)).to(torch.bfloat16)       # as the projection leaves them, the step sizes beside
    xbc, dt = rows[:, :H * V + 2 * G * N], rows[:, H * V + 2 * G * N:H * V + 2 * G * N + H]
    if strong:
        dt[5::17], dt[9::23] = 5000.0, -60.0        # some tokens forget everything, some write nothing and forget nothing
    bias, rate, skip = r(H) * 0.5 - 1.0, torch.exp(r(H)), 1.0 + 0.2 * r(H)
    return xbc, dt, bias, rate, skip, r(len(lens), H, V, N)


def exact(args, H, G, N, V, lens):
    xbc, dt, bias, rate, skip, state = (t.double() for t in args)
    d = torch.nn.functional.softplus(dt + bias, threshold=100)
    a = torch.exp(-rate * d)
    x = xbc[:, :H * V].view(-1, H, V)
    B, C = (xbc[:, H * V + i * G * N:H * V + (i + 1) * G * N].view(-1, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    out, left, t = [], [], 0
    for b, n in enumerate(lens):
        S = state[b].clone()
        for _ in range(n):
            S = a[t, :, None, None] * S + (d[t, :, None] * x[t])[:, :, None] * B[t, :, None]
            out.append(torch.einsum("hvn,hn->hv", S, C[t]) + skip[:, None] * x[t])
            t += 1
        left.append(S)
    return torch.stack(out), torch.stack(left)


def run(KR, args, H, G, N, V, lens):
    xbc, dt, bias, rate, skip, state = args
    n = len(lens)
    store = torch.zeros(n + 1, H * N * V + 3, device="cuda")
    store[:n, 3:] = state.reshape(n, -1)
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_new=cu, seq_slot=torch.arange(n, dtype=torch.int32, device="cuda"), n_seq=n, max_new=max(lens))
    y = KR.ssd_scan(xbc, dt, bias, rate, skip, H, G, N, V, store, 3, batch)
    return y.view(-1, H, V), store[:n, 3:].view(n, H, V, N)


@pytest.mark.parametrize("H,G,N,V,lens,strong", [(2, 1, 64, 32, [80], False), (4, 2, 128, 64, [127, 1, 129], False), (8, 8, 128, 64, [16, 128, 17], True),
                                                 (6, 1, 64, 64, [300], True), (24, 2, 128, 32, [256, 5], False), (3, 3, 128, 64, [600], False)])
def test_against_the_scan(KR, monkeypatch, H, G, N, V, lens, strong):
    args = make(H, G, N, V, lens, H + N + V + sum(lens), strong)
    want = exact(args, H, G, N, V, lens)
    assert KR.ssd_chunked(args[0], H, N, V, SimpleNamespace(max_new=max(lens), n_seq=len(lens)))
    got = run(KR, args, H, G, N, V, lens)
    monkeypatch.setattr(KR, "SSD_CHUNKED_FROM", 1 << 30)
    scan = run(KR, args, H, G, N, V, lens)
    for g, s, w in zip(got, scan, want):
        off = lambda x: float((x.double() - w).norm() / w.norm())
        # no further off than the scan (a tenth for one draw's spread), or as good as a sum of two roundings can be expected to be
        assert off(g) <= max(1.1 * off(s), 1.2e-7), (off(g), off(s))
        print(f"{off(g):.2e} against the scan's {off(s):.2e}")
        assert ((g.double() - w).abs().max() / w.abs().max()) <= 4e-6


def test_rows_that_are_not_aligned_take_the_scan(KR):
    args = list(make(2, 1, 64, 32, [90], 3))
    wide = torch.zeros(90, args[0].shape[1] + 1, dtype=torch.bfloat16, device="cuda")
    wide[:, 1:] = args[0]
    args[0] = wide[:, 1:]
    assert KR.ssd_chunked(args[0], 2, 64, 32, SimpleNamespace(max_new=90, n_seq=1)) == 0
    want = exact(args, 2, 1, 64, 32, [90])
    for g, w in zip(run(KR, args, 2, 1, 64, 32, [90]), want):
        assert float((g.double() - w).norm() / w.norm()) < 1e-6


@pytest.mark.parametrize("H,G,N,V,lens", [(4, 2, 128, 64, [700]), (8, 2, 64, 32, [300, 90]), (4, 4, 128, 32, [256])])
@pytest.mark.parametrize("kind", ["silu", "positive"])
def test_no_further_off_than_the_scan(KR, monkeypatch, H, G, N, V, lens, kind):
    """x, B and C as they come from silu, and of one sign with a state of the same, where truncated sums all err the same way."""
    off = []
    for seed in range(6):
        xbc, dt, bias, rate, skip, state = make(H, G, N, V, lens, seed)
        x = torch.nn.functional.silu(xbc.float()) if kind == "silu" else xbc.float().abs()
        args = (x.to(torch.bfloat16), dt, bias, rate, skip, state if kind == "silu" else state.abs())
        want = exact(args, H, G, N, V, lens)
        both = []
        for least in (KR.SSD_CHUNKED_FROM, 1 << 30):
            with monkeypatch.context() as m:
                m.setattr(KR, "SSD_CHUNKED_FROM", least)
                both += [float((g.double() - w).norm() / w.norm()) for g, w in zip(run(KR, args, H, G, N, V, lens), want)]
        off.append(both)
    y, S, y_scan, S_scan = torch.tensor(off).mean(0).tolist()
    print(f"{kind}: y {y:.2e} against the scan's {y_scan:.2e}, state {S:.2e} against {S_scan:.2e}")
    # A product of 16 is truncated once, 2^-24 of it at most and 0.36 of 2^-23 on average; C . B and the product with x are one
    # each, so that outputs of one sign lose 8.6e-8 at most.  Else no further off than the scan (a tenth for six draws' spread).
    slack = 0.0 if kind == "silu" else 4e-8
    assert y <= 1.1 * y_scan + slack and S <= 1.1 * S_scan


@pytest.mark.parametrize("lens", [[0, 90, 0, 130], [100, 0]])
def test_empty_sequences_and_rows_that_are_nobodys(KR, lens):
    args = make(4, 2, 64, 32, lens, 7)
    xbc, dt, bias, rate, skip, state = args
    M, H, N, V = sum(lens) + 3, 4, 64, 32
    wide = lambda t: torch.cat([t, torch.ones(3, t.shape[1], dtype=t.dtype, device="cuda")])
    xbc, dt = wide(xbc), wide(dt)
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    batch = SimpleNamespace(cu_new=cu, seq_slot=torch.arange(len(lens), dtype=torch.int32, device="cuda"), n_seq=len(lens), max_new=max(lens))
    store = state.reshape(len(lens), -1).clone()
    poison = torch.full((M, H * V), float("nan"), device="cuda")         # what the result's memory holds before
    del poison
    y = KR.ssd_scan(xbc, dt, bias, rate, skip, H, 2, N, V, store, 0, batch)
    want, left = exact(args, 4, 2, 64, 32, lens)
    assert not y[sum(lens):].any()
    assert float((y[:sum(lens)].view(-1, H, V).double() - want).norm() / want.norm()) < 1e-6
    assert float((store.view(left.shape).double() - left).norm() / left.norm()) < 1e-6


@pytest.mark.parametrize("V", [32, 64])
@pytest.mark.parametrize("what", ["x nan", "x inf", "B", "C", "dt"])
def test_a_token_that_is_not_finite_spoils_none_before_it(KR, V, what):
    H, G, N, lens, bad = 4, 2, 64, [300, 90], 200                # the token in the first sequence's second chunk, amid a tile
    args = make(H, G, N, V, lens, 3)
    clean, left = (t.clone() for t in run(KR, args, H, G, N, V, lens))
    xbc, dt = args[:2]
    at = {"x nan": slice(V, V + 5), "x inf": slice(V, V + 5), "B": slice(H * V, H * V + N), "C": slice(H * V + G * N, H * V + G * N + N)}
    if what == "dt":
        dt[bad] = float("nan")
    else:
        xbc[bad, at[what]] = float("inf" if what == "x inf" else "nan")
    y, state = run(KR, args, H, G, N, V, lens)
    keep = torch.ones(sum(lens), dtype=torch.bool, device="cuda")
    keep[bad:lens[0]] = False
    assert torch.equal(y[keep], clean[keep]) and torch.equal(state[1], left[1])
    if what[0] == "x":                                           # five channels of the second head, from the token on
        assert not y[bad:lens[0], 1, :5].isfinite().any() and not state[0, 1, :5].isfinite().any()
        y[:, 1, :5], clean[:, 1, :5], state[0, 1, :5], left[0, 1, :5] = 0, 0, 0, 0
        assert torch.equal(y, clean) and torch.equal(state, left)
    elif what == "C":
        keep[bad + 1:lens[0]] = True
        assert torch.equal(y[keep], clean[keep]) and y[bad, :2].isnan().all() and torch.equal(state, left)
    else:
        assert y[bad:lens[0], :2].isnan().all() and state[0, :2].isnan().all()
