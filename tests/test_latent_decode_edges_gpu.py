"""Single tokens over a cached latent (csrc/attn_latent.cu) where a tile of keys cannot be brought as usual, against 64 bits: the
widest rows (no byte of shared memory is left beside them), pages whose length is no multiple of a tile, windows, rings."""
from __future__ import annotations

import pytest
import torch

import test_latent_sizes_gpu as sizes


def exact(d, q, norm_w, tables, uk, uv, batch, mem, rank, scale, window):
    """As sizes.exact, over the positions a window leaves and through the cache's ring."""
    F = torch.float64
    n, H, hd = q.shape
    cos, sin, rot = tables
    pos = batch.tok_pos.long()
    rounded = lambda x: x.to(d.dtype).to(F)

    def turn(x):
        u, v = x[..., :rot // 2], x[..., rot // 2:]
        c, s = (t[pos].to(F).view(n, *([1] * (x.dim() - 2)), rot // 2) for t in (cos, sin))
        return torch.cat([u * c - v * s, v * c + u * s], -1)

    c = d[:, :rank].to(F)
    row = rounded(torch.cat([c / torch.sqrt((c * c).mean(-1, keepdim=True) + 1e-6) * norm_w.to(F), turn(d[:, rank:].to(F))], -1))
    qa = torch.cat([torch.einsum("nhp,hpr->nhr", q[..., :hd - rot].to(F), uk.to(F).view(H, hd - rot, rank)), rounded(turn(q[..., hd - rot:].to(F)))], -1)
    out = []
    for b in range(n):
        at = int(pos[b])
        p = torch.arange(max(0, at - window + 1) if window else 0, at, device=d.device)
        r = p % mem.ring_rows if mem.ring_rows else p
        keys = mem.k_pages[mem.page_table[b].long()[r // mem.page_size], 0, r % mem.page_size].to(F)
        keys = torch.cat([keys, row[b:b + 1]])
        w = torch.softmax(qa[b] @ keys.T * scale, -1)
        out.append(torch.einsum("hr,hvr->hv", w @ keys[:, :rank], uv.to(F).view(H, -1, rank)).reshape(-1))
    return torch.stack(out)


# 2,384 and 1,776 elements: the widest rows with up to 16 heads a block and with 32; 640 | 656: with the queries in registers | not
@pytest.mark.gpu
@pytest.mark.parametrize("H,rank,rot,page,window,ring", [
    (8, 512, 1872, 64, 0, 0), (20, 512, 1264, 64, 0, 0), (16, 512, 128, 64, 0, 0), (16, 512, 144, 64, 0, 0),
    (16, 512, 64, 24, 0, 0), (20, 256, 32, 5, 0, 0), (16, 512, 64, 64, 100, 0), (16, 512, 64, 24, 33, 0),
    (8, 256, 64, 64, 100, 192), (20, 512, 64, 24, 90, 120)])
def test_single_tokens(monkeypatch, H, rank, rot, page, window, ring):
    from toyinfer_b200.kernels import latent as KL, check_status
    monkeypatch.setattr(sizes, "PAGE", page)
    scale = (64 + rot) ** -0.5
    d, q, norm_w, tables, uk, uv, batch, mem = sizes.layer(torch.bfloat16, H, 64, rot, rank, 48, [0, 31, 32, 200, 1000, 95])
    mem.ring_rows = ring
    want = exact(d, q, norm_w, tables, uk, uv, batch, mem, rank, scale, window)
    got = KL.attention_single(d, q, rank, rot, norm_w, 1e-6, tables, uk, uv, 48, scale, window, None, batch, mem)
    check_status()
    # queries in the latent space and softmax weights are rounded to bfloat16 (2^-9 each), the result too
    assert float((got.double() - want).norm() / want.norm()) < 1e-2


@pytest.mark.gpu
@pytest.mark.parametrize("H,rank", [(8, 256), (16, 512), (20, 256)])
def test_a_sequence_does_not_depend_on_the_others(H, rank):
    """The same bits whatever the lengths of the sequences beside it: the step is planned for its longest, and a split is a part of
    the sequence's own keys."""
    from toyinfer_b200.kernels import latent as KL, check_status
    longest = [1000, 3000, 2900, 1700, 2000, 2500]
    d, q, norm_w, tables, uk, uv, batch, mem = sizes.layer(torch.bfloat16, H, 64, 64, rank, 48, longest)
    got = []
    for held in (longest, [1000, 3000, 40, 70, 0, 31]):
        batch.tok_pos, batch.seq_start = (torch.tensor(held, dtype=torch.int32, device="cuda") for _ in range(2))
        batch.seq_len = batch.seq_start + 1
        got.append(KL.attention_single(d, q, rank, 64, norm_w, 1e-6, tables, uk, uv, 48, 128 ** -0.5, 0, None, batch, mem))
    check_status()
    assert torch.equal(got[0][:2], got[1][:2])
