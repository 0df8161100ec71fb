"""Which form the experts' bfloat16 product takes (csrc/moe_grouped.cu): the register form up to eight places an expert and
wherever the experts are few, shared-memory tiles where the register form's repeated reads of the weights were measured to take longer.
Needs nvcc to build the library, no GPU."""
from __future__ import annotations

import shutil

import pytest

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None, reason="the kernel library cannot be built without nvcc")


def tiles(E, places, N, K, pair):
    from toyinfer_b200.kernels.lib import library
    return library().ti_moe_skinny_tiles(E, E * places, N, K, int(pair), 148)


# (experts, places, weight rows, contraction, pair): us from registers / in tiles, measured
SLOWER_FROM_REGISTERS = [(32, 16, 1024, 2048, True),      # 80 / 59
                         (32, 12, 1024, 2048, True),      # 66 / 59
                         (64, 24, 1280, 2048, True),      # 268 / 150
                         (64, 20, 256, 1024, True),       # 36 / 32
                         (32, 16, 2048, 1024, False),     # 52 / 36
                         (64, 12, 2048, 1280, False),     # 111 / 78
                         (16, 16, 4096, 1536, False)]     # 73 / 50
FASTER_FROM_REGISTERS = [(8, 24, 1024, 2048, True),       # 30 / 54
                         (16, 20, 1024, 2048, True),      # 51 / 59
                         (16, 24, 640, 1024, True),       # 25 / 29
                         (8, 24, 2048, 1024, False),      # 18 / 26
                         (16, 16, 2048, 1280, False),     # 34 / 40
                         (64, 8, 1280, 2048, True)]       # both products 232 / 247


@pytest.mark.parametrize("E,places,N,K,pair", SLOWER_FROM_REGISTERS)
def test_tiles_where_they_are_faster(E, places, N, K, pair):
    assert tiles(E, places, N, K, pair) == 0


@pytest.mark.parametrize("E,places,N,K,pair", FASTER_FROM_REGISTERS)
def test_registers_where_they_are_faster(E, places, N, K, pair):
    assert tiles(E, places, N, K, pair) > 0


def test_limits():
    for E in (1, 2, 8, 33, 100, 512):
        for N in (8, 100, 1024, 100000):
            for K in (8, 640, 1032, 8192):
                for pair in (False, True):
                    got = [tiles(E, p, N, K, pair) for p in range(1, 30)]
                    assert got[:4] == [1] * 4 and got[4:8] == [2] * 4 and set(got[8:18]) <= {0, 2} and set(got[18:24]) <= {0, 4}
                    assert got[24:] == [0] * 5
                    assert not any(a == 0 and b > 0 for a, b in zip(got, got[1:]))       # once in tiles, always in tiles


# rows off the 16-byte boundary: us from registers / in staged tiles
@pytest.mark.parametrize("E,places,N,pair,staged", [(16, 80, 1023, True, True),       # 942 / 799
                                                    (16, 320, 391, True, True),       # 676 / 403
                                                    (4, 320, 1023, True, True),       # 860 / 567
                                                    (16, 80, 2047, False, True),      # 495 / 428
                                                    (16, 40, 1023, True, False),      # 503 / 606
                                                    (16, 80, 391, True, False),       # 176 / 230
                                                    (4, 160, 2047, False, False),     # 219 / 277
                                                    (32, 2, 4096, True, False)])
def test_rows_off_the_boundary(E, places, N, pair, staged):
    from toyinfer_b200.kernels.lib import library
    assert bool(library().ti_moe_staged_tiles(E, E * places, N, int(pair), 148)) == staged
