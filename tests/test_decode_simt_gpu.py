"""The CUDA-core decode attention at the sizes where its split of the work changes: 8, 16 and 32 lanes a key and one, two or four
runs of four elements each, one to six query heads a block and chunks of them, lengths around a warp's batch and a page, rows off
the 16-byte boundary, and splits that write directly, merge as a cluster (up to 16) or through scratch memory."""
from __future__ import annotations

import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [1, 7, 8, 33, 63, 64, 65, 129, 1300]


def paged(lens, nkv, hd, dtype, window, seed, offset=0):
    """Caches of random pages (every line that no sequence owns is NaN), and keys and values by sequence."""
    ring = -(-window // 64) * 64 if window else 0
    need = [-(-(min(n, ring) if ring else n) // 64) for n in lens]
    g = torch.Generator("cuda").manual_seed(seed)
    order = torch.randperm(sum(need), generator=g, device="cuda").tolist()
    stores = [torch.full((sum(need) * nkv * 64 * hd + offset,), float("nan"), dtype=dtype, device="cuda")[offset:].view(-1, nkv, 64, hd) for _ in range(2)]
    table = torch.zeros((len(lens), max(need)), dtype=torch.int32, device="cuda")
    rows = []
    for s, n in enumerate(lens):
        pages = [order.pop() for _ in range(need[s])]
        table[s, :len(pages)] = torch.tensor(pages, dtype=torch.int32)
        kv = [torch.randn((n, nkv, hd), generator=g, device="cuda").to(dtype) for _ in range(2)]
        for p in range(max(0, n - ring) if ring else 0, n):
            r = p % ring if ring else p
            for store, x in zip(stores, kv):
                store[pages[r // 64], :, r % 64] = x[p]
        rows.append(kv)
    mem = SimpleNamespace(k_pages=stores[0], v_pages=stores[1], page_table=table, page_size=64, ring_rows=ring, n_kv_heads=nkv)
    return mem, rows


def exact(q, rows, scale, window):
    out = []
    for x, (k, v) in zip(q.double(), rows):
        lo = max(0, k.shape[0] - window) if window else 0
        k, v = (a[lo:].double().repeat_interleave(x.shape[0] // a.shape[1], dim=1) for a in (k, v))
        p = torch.softmax(torch.einsum("hd,phd->hp", x, k) * scale, dim=1)
        out.append(torch.einsum("hp,phd->hd", p, v))
    return torch.stack(out)


def run(monkeypatch, dtype, nh, nkv, hd, window, splits, offset=0, lens=LENS):
    from toyinfer_b200.kernels import attention
    mem, rows = paged(lens, nkv, hd, dtype, window, nh * hd, offset)
    g = torch.Generator("cuda").manual_seed(5)
    q = torch.randn((len(lens), nh * hd + 3), generator=g, device="cuda").to(dtype)[:, 3:].view(len(lens), nh, hd)
    batch = SimpleNamespace(plan_len=max(lens), n_real_seq=len(lens), seq_slot=torch.arange(len(lens), dtype=torch.int32, device="cuda"),
                            seq_len=torch.tensor(lens, dtype=torch.int32, device="cuda"))
    monkeypatch.setattr(attention, "decode_plan", lambda *a: (splits, 0))
    out = torch.full((len(lens), nh, hd), float("nan"), dtype=dtype, device="cuda")
    scale = 1 / math.sqrt(hd)
    attention.decode(q, mem, out, scale, window, batch)
    want = exact(q, rows, scale, window)
    # 32 bits: sums of up to 1,300 terms of which no more than 170 follow one another, and an exponential of two
    # units in the last place; bfloat16: the result's rounding
    bound = 2e-6 if dtype == torch.float32 else 4e-3
    assert ((out.double() - want).norm(dim=2) <= bound * want.norm(dim=2)).all()


@pytest.mark.parametrize("splits", [1, 2, 7, 16, 17])
@pytest.mark.parametrize("nh,nkv,hd,window", [(3, 3, 4, 0), (4, 2, 32, 0), (6, 2, 32, 100), (5, 1, 36, 0), (16, 2, 64, 0), (4, 4, 72, 0),
                                              (12, 2, 128, 0), (8, 2, 128, 64), (10, 1, 128, 0), (4, 2, 160, 0), (2, 2, 256, 130)])
def test_float32(monkeypatch, nh, nkv, hd, window, splits):
    run(monkeypatch, torch.float32, nh, nkv, hd, window, splits)


@pytest.mark.parametrize("splits", [1, 5])
@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 32, 0), (5, 1, 48, 40), (6, 6, 96, 0), (4, 1, 256, 0)])
def test_bfloat16(monkeypatch, nh, nkv, hd, window, splits):
    run(monkeypatch, torch.bfloat16, nh, nkv, hd, window, splits)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd", [32, 68, 160])
def test_pages_off_the_boundary(monkeypatch, dtype, hd):
    run(monkeypatch, dtype, 4, 2, hd, 0, 3, offset=1)


@pytest.mark.parametrize("dtype,offset", [(torch.float32, 0), (torch.float32, 1), (torch.bfloat16, 0), (torch.bfloat16, 1)])
@pytest.mark.parametrize("nh,nkv,hd,splits", [(4, 2, 260, 1), (3, 1, 384, 7), (2, 2, 448, 17), (2, 1, 401, 2)])
def test_heads_of_four_runs(monkeypatch, dtype, offset, nh, nkv, hd, splits):
    """Wider than any layer's (kernels/attention.py stops at 256): the C entry's own range."""
    run(monkeypatch, dtype, nh, nkv, hd, 0, splits, offset=offset)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("splits", [8, 9, 16])
@pytest.mark.parametrize("nh,nkv,hd", [(6, 1, 32), (5, 1, 96), (2, 2, 256)])
def test_clusters(monkeypatch, dtype, nh, nkv, hd, splits):
    """Two sequences, whose clusters find room (more of them meet through scratch memory): splits with and without keys."""
    run(monkeypatch, dtype, nh, nkv, hd, 0, splits, lens=[1300, 70])
