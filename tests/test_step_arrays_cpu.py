"""A step's arrays where only part of them is written anew (engine/batch.py), and page tables that go to the device by runs of rows
(cache/manager.py): the same as with everything written."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from toyinfer_b200.cache.manager import CacheManager
from toyinfer_b200.engine.batch import BatchBuffers, fill_batch
from toyinfer_b200.parts.base import KVRequest


@pytest.mark.parametrize("seed", range(8))
def test_a_buffer_used_again_holds_what_a_new_one_would(seed):
    rng = np.random.default_rng(seed)
    used = BatchBuffers(9, 12, "cpu")
    for _ in range(40):
        n = int(rng.integers(1, 5))
        kind = rng.choice(["single", "single", "single", "runs", "spare"])
        pad = int(rng.integers(0, 3)) if kind == "single" else 0
        slots = [int(s) for s in rng.permutation(8)[:n]]
        starts = [int(s) for s in rng.integers(0, 500, n)]
        new = [1] * n if kind != "runs" else [int(k) for k in rng.integers(1, 4, n)]
        tokens = [[int(t) for t in rng.integers(0, 1000, k)] for k in new]
        mode = "mixed" if kind == "runs" else "extend"
        total = 8 if kind == "spare" else None
        scratch = int(rng.choice([8, 9]))
        got = fill_batch(used, mode, slots, starts, tokens, scratch, 600, pad_seqs=pad, total_tok=total)
        fresh = BatchBuffers(9, 12, "cpu")
        want = fill_batch(fresh, mode, slots, starts, tokens, scratch, 600, pad_seqs=pad, total_tok=total)
        assert torch.equal(used.dev, fresh.dev)
        for name in BatchBuffers.FIELDS:
            assert torch.equal(getattr(got, name), getattr(want, name)), name
        assert (got.n_seq, got.n_tok, got.max_new, got.max_pos_after, got.host_slots, got.host_starts, got.host_new) == \
            (want.n_seq, want.n_tok, want.max_new, want.max_pos_after, want.host_slots, want.host_starts, want.host_new)


@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("max_len", [300, 200000])       # rows short enough to go together, and long ones
def test_page_tables_reach_the_device(window, max_len):
    cache = CacheManager([KVRequest(1, 8, window)], 64 * 60, 6, max_len, torch.float32, "cpu")
    rng = np.random.default_rng(max_len + window)
    live = []
    for _ in range(80):
        if len(live) < 6 and rng.random() < 0.5:
            live.append(cache.allocate_slot())
        for slot in live:
            if rng.random() < 0.5 and cache.length[slot] < 200:
                n = cache.length[slot] + int(rng.integers(1, 90))
                cache.reserve(slot, n)
                cache.commit(slot, n)
        if live and rng.random() < 0.2:
            cache.release(live.pop(int(rng.integers(len(live)))))
        cache.flush()
        for g in cache.kv_groups:
            for slot in live:
                held = g.slot_pages.get(slot, [])
                assert g.table[slot, :len(held)].tolist() == held
