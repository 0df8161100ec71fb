"""A step's arrays through the two pinned host buffers of a GPU (engine/batch.py): bursts of steps written while the stream is still busy
with what came before, so that a buffer is filled while the other's upload waits, each holding its own last layout.  What every step
finds on the device is what a new buffer would have brought."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from toyinfer_b200.engine.batch import BatchBuffers, fill_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(4))
def test_bursts_behind_a_busy_stream(seed):
    rng = np.random.default_rng(seed)
    used, got, want = BatchBuffers(9, 12, "cuda"), [], []
    for _ in range(20):
        torch.cuda._sleep(2_000_000)                     # about a millisecond: longer than the burst takes to write
        for _ in range(int(rng.integers(1, 6))):
            n = int(rng.integers(1, 5))
            kind = rng.choice(["single", "single", "single", "runs", "spare"])
            pad = int(rng.integers(0, 3)) if kind == "single" else 0
            slots = [int(s) for s in rng.permutation(8)[:n]]
            starts = [int(s) for s in rng.integers(0, 500, n)]
            new = [1] * n if kind != "runs" else [int(k) for k in rng.integers(1, 4, n)]
            tokens = [[int(t) for t in rng.integers(0, 1000, k)] for k in new]
            step = ("mixed" if kind == "runs" else "extend", slots, starts, tokens, int(rng.choice([8, 9])), 600)
            more = dict(pad_seqs=pad, total_tok=8 if kind == "spare" else None)
            views = fill_batch(used, *step, **more)
            got.append([used.dev.clone()] + [getattr(views, name).clone() for name in BatchBuffers.FIELDS])
            fresh = BatchBuffers(9, 12, "cpu")
            views = fill_batch(fresh, *step, **more)
            want.append([fresh.dev.clone()] + [getattr(views, name).clone() for name in BatchBuffers.FIELDS])
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert all(torch.equal(x.cpu(), y) for x, y in zip(a, b))
