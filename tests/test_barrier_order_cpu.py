"""Shared-memory barriers (mbarriers) are set up by one thread; no other may wait on one before the block has met.  Looked for in the
kernels' text: between the last set-up of a kernel and the first wait after it stands a barrier of the block or the cluster."""
from __future__ import annotations

import os
import re

import pytest

import toyinfer_b200

CSRC = os.path.join(os.path.dirname(toyinfer_b200.__file__), "csrc")
FILES = sorted(n for n in os.listdir(CSRC) if n.endswith((".cu", ".cuh")) and n != "tma.cuh")      # (tma.cuh defines the calls themselves)
MEETS = re.compile(r"__syncthreads\(\)|cluster_sync\w*\(\)|cluster\.sync\(\)|cluster_wait\w*\(\)")


def unordered(text):
    """Lines of the first waits that no meeting of the block separates from the barriers' set-up."""
    text = re.sub(r"//[^\n]*", "", text)
    found, at = [], 0
    while (first := text.find("mbar_init(", at)) >= 0:
        wait = text.find("mbar_wait(", first)
        if wait < 0:
            return found
        last = text.rfind("mbar_init(", 0, wait)
        if not MEETS.search(text, last, wait):
            found.append(text.count("\n", 0, wait) + 1)
        at = wait
    return found


@pytest.mark.parametrize("name", FILES)
def test_the_block_meets_between_set_up_and_wait(name):
    with open(os.path.join(CSRC, name)) as f:
        assert unordered(f.read()) == []


def test_the_search_itself():
    assert unordered("if (t == 0) mbar_init(&b, 1);\nmbar_wait(&b, 0);") == [2]
    assert unordered("mbar_init(&b, 1);\n__syncthreads();\nmbar_wait(&b, 0);") == []
    assert unordered("mbar_init(&b, 1);\n// __syncthreads();\nmbar_wait(&b, 0);") == [3]
