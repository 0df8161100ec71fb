"""Single tokens over a cached latent (csrc/attn_latent.cu, kernels/latent.py) at the edges of what they take, against 64 bits: rows so
wide that one tile of keys fits beside the queries, long heads, float32 at its own number of splits.  And that number's rule."""
from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

PAGE = 64


def test_float32_rows_take_a_second_round_only_where_tiles_are_left():
    from toyinfer_b200.kernels.latent import decode_splits as splits
    assert splits(4, 8, 8, 2000, 148) == 64                       # tensor cores: all blocks run at once
    assert splits(4, 8, 8, 2000, 148, 576) == 37                  # one block an SM; a second round would leave a tile each
    assert splits(16, 8, 8, 2000, 148, 576) == 16 and splits(16, 8, 8, 2000, 148, 288) == 18
    assert splits(64, 16, 16, 2000, 148, 576) == 4
    for n in (1, 3, 16, 64, 500):
        for heads, hb in ((8, 8), (16, 16), (32, 32), (40, 32)):
            for span in (1, 31, 200, 4000, 100000):
                for row in (64, 424, 425, 576, 890):
                    one = max(1, min(148 // (n * -(-heads // hb)), span // 32 + 2, 64))
                    assert one <= splits(n, heads, hb, span, 148, row) <= splits(n, heads, hb, span, 148)


def layer(dtype, n_heads, plain, rot, rank, vdim, held, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n, W = len(held), rank + rot
    need = [-(-(h + 1) // PAGE) for h in held]
    table = torch.full((n, max(need)), -1, dtype=torch.int32)
    at = 0
    for b, k in enumerate(need):
        table[b, :k] = torch.arange(at, at + k)
        at += k
    pages = r(at, 1, PAGE, W).to(dtype)
    mem = SimpleNamespace(k_pages=pages, page_table=table.cuda(), page_size=PAGE, ring_rows=0, n_kv_heads=1, head_dim=W)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    batch = SimpleNamespace(mode="extend", n_seq=n, n_tok=n, max_new=1, max_pos_after=max(held) + 1, plan_len=max(held) + 1, tok_pos=i32(held),
                            tok_seq=i32(list(range(n))), seq_slot=i32(list(range(n))), seq_start=i32(held), seq_len=i32([h + 1 for h in held]),
                            cu_new=i32(list(range(n + 1))))
    angle = torch.arange(max(held) + 1, device="cuda")[:, None] * 0.01 * torch.arange(1, rot // 2 + 1, device="cuda")[None]
    tables = (angle.cos().float().contiguous(), angle.sin().float().contiguous(), rot)
    d, q = r(n, W).to(dtype), (r(n, n_heads, plain + rot) * 0.3).to(dtype)
    uk, uv = ((r(n_heads * k, rank) * rank ** -0.5).to(dtype) for k in (plain, vdim))
    return d, q, 1.0 + 0.1 * r(rank), tables, uk, uv, batch, mem


def exact(d, q, norm_w, tables, uk, uv, batch, mem, rank, scale):
    F = torch.float64
    n, H, hd = q.shape
    cos, sin, rot = tables
    plain = hd - rot
    pos = batch.tok_pos.long()
    rounded = lambda x: x.to(d.dtype).to(F)                       # what the cache holds and the tensor cores multiply

    def turn(x):
        u, v = x[..., :rot // 2], x[..., rot // 2:]
        c, s = (t[pos].to(F).view(n, *([1] * (x.dim() - 2)), rot // 2) for t in (cos, sin))
        return torch.cat([u * c - v * s, v * c + u * s], -1)

    c = d[:, :rank].to(F)
    row = rounded(torch.cat([c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-6) * norm_w.to(F), turn(d[:, rank:].to(F))], -1))
    uk, uv = uk.to(F).view(H, plain, rank), uv.to(F).view(H, -1, rank)
    qa = torch.cat([torch.einsum("nhp,hpr->nhr", q[..., :plain].to(F), uk), rounded(turn(q[..., plain:].to(F)))], -1)
    out = []
    for b in range(n):
        held = int(pos[b])
        keys = torch.cat([mem.k_pages[mem.page_table[b].clamp(min=0).long()].reshape(-1, row.shape[1])[:held].to(F), row[b:b + 1]])
        p = torch.softmax(qa[b] @ keys.T * scale, -1)
        out.append(torch.einsum("hr,hvr->hv", p @ keys[:, :rank], uv).reshape(-1))
    return torch.stack(out)


# rows of 1,200 elements over 20 heads and of 1,456 over 8: one tile; of 1,168: the widest of two; a head of 9,000 unrotated elements
@pytest.mark.gpu
@pytest.mark.parametrize("H,plain,rot,rank", [(20, 64, 688, 512), (8, 64, 944, 512), (20, 64, 656, 512), (16, 32, 32, 128), (1, 9000, 32, 64)])
def test_single_tokens(H, plain, rot, rank):
    from toyinfer_b200.kernels import latent as KL, check_status
    scale = (plain + rot) ** -0.5
    d, q, norm_w, tables, uk, uv, batch, mem = layer(torch.bfloat16, H, plain, rot, rank, 48, [0, 31, 32, 200, 1000])
    want = exact(d, q, norm_w, tables, uk, uv, batch, mem, rank, scale)
    got = KL.attention_single(d, q, rank, rot, norm_w, 1e-6, tables, uk, uv, 48, scale, 0, None, batch, mem)
    check_status()
    # queries in the latent space and softmax weights are rounded to bfloat16 (2^-9 each), the result too
    assert float((got.double() - want).norm() / want.norm()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("n,H,rank,rot", [(4, 8, 512, 64), (16, 8, 256, 32), (20, 16, 512, 64), (1, 3, 64, 16)])
def test_float32_single_tokens(n, H, rank, rot):
    from toyinfer_b200.kernels import latent as KL
    scale = (64 + rot) ** -0.5
    held = [(i * 613) % 1900 for i in range(n)]
    d, q, norm_w, tables, uk, uv, batch, mem = layer(torch.float32, H, 64, rot, rank, 64, held)
    want = exact(d, q, norm_w, tables, uk, uv, batch, mem, rank, scale)
    lat = KL.prep(d, q, rank, rot, norm_w, 1e-6, tables, batch, mem)
    got = KL.attention(q, lat, uk, uv, 64, rank, rot, scale, 0, None, batch, mem)
    assert float((got.double() - want).norm() / want.norm()) < 2e-6      # sums of some 600 products and of 2,000 positions in 32 bits
