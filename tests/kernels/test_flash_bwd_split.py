"""How many CTAs share a key tile in the attention backward: the launcher's rule at grids that were timed with one, two and four. Host
arithmetic of the built library, no GPU."""

import ctypes

import pytest

from nanonemo_b200.csrc import build

# head_dim, batch, heads, KV heads, T: whole backward, us, with one / two / four CTAs a key tile on 148 SMs
TIMED = [
    (64, 1, 8, 8, 64, 16.4, 18.4, 18.4), (64, 8, 8, 8, 64, 16.4, 20.5, 28.7), (64, 10, 8, 8, 64, 16.4, 28.7, 36.9), (64, 14, 8, 8, 128, 20.5, 32.7, 51.2),
    (64, 36, 8, 8, 128, 30.7, 57.3, 106.4), (64, 4, 8, 8, 200, 18.6, 22.4, 30.7), (64, 8, 8, 8, 256, 22.5, 34.8, 53.2), (64, 4, 8, 8, 512, 26.6, 36.8, 53.2),
    (64, 25, 12, 4, 64, 24.5, 34.8, 49.1), (64, 14, 12, 4, 128, 24.5, 26.6, 32.7), (64, 14, 12, 4, 256, 32.8, 43.0, 59.4), (64, 10, 12, 4, 512, 47.1, 63.5, 79.8),
    (64, 1, 12, 4, 512, 36.8, 28.7, 22.5), (64, 1, 12, 4, 1024, 57.3, 40.9, 30.7), (64, 4, 12, 4, 1024, 65.5, 59.4, 77.8), (64, 8, 12, 4, 1024, 79.8, 104.4, 143.3),
    (64, 2, 12, 4, 2048, 104.4, 75.8, 98.2), (64, 4, 12, 4, 2048, 116.7, 139.3, 182.2), (64, 18, 16, 4, 256, 43.0, 51.0, 73.7), (64, 2, 16, 4, 2048, 135.1, 90.1, 112.5),
    (128, 8, 8, 8, 128, 20.4, 26.6, 38.9), (128, 14, 8, 8, 128, 24.5, 40.9, 65.5), (128, 25, 12, 4, 128, 36.8, 53.2, 75.7), (128, 14, 16, 4, 256, 55.2, 67.5, 88.0),
    (128, 10, 16, 4, 512, 88.0, 104.4, 128.8), (128, 4, 16, 4, 512, 71.7, 55.3, 57.3), (128, 1, 16, 4, 2048, 208.8, 127.6, 94.2), (128, 8, 6, 1, 2048, 320.5, 196.6, 235.3),
    (128, 36, 6, 1, 512, 118.8, 112.1, 149.5), (128, 1, 6, 1, 64, 22.5, 24.4, 22.4),
    (64, 5, 12, 4, 1024, 67.6, 73.7, 92.1), (64, 24, 6, 1, 1024, 120.8, 124.9, 155.6), (64, 100, 64, 1, 64, 208.9, 231.4, 231.4), (64, 5, 6, 1, 4096, 354.3, 247.2, 280.6),
    (128, 5, 12, 4, 1024, 104.4, 108.5, 135.2), (128, 3, 12, 4, 1024, 96.2, 69.4, 88.0), (128, 2, 6, 1, 4096, 561.4, 321.3, 192.5),
]


@pytest.fixture(scope="module")
def split():
    if not build.LIB.exists():
        pytest.skip("kernel library not built")
    lib = ctypes.CDLL(str(build.LIB))
    lib.nnb_flash_bwd_split.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    return lambda hd, B, H, KVH, T, sms=148: lib.nnb_flash_bwd_split(T, 128 if hd == 64 else 64, B * KVH, H // KVH, sms)


@pytest.mark.parametrize("hd,B,H,KVH,T,one,two,four", TIMED)
def test_no_timed_grid_gets_slower_by_sharing(split, hd, B, H, KVH, T, one, two, four):
    us = {1: one, 2: two, 4: four}
    chosen = us[split(hd, B, H, KVH, T)]
    assert chosen <= 1.02 * one  # (the timer's steps are 2 us)
    assert chosen <= 1.12 * min(us.values())


@pytest.mark.parametrize("hd", [64, 128])
def test_no_more_ctas_than_visits_and_none_shared_in_full_grids(split, hd):
    for H, KVH in ((1, 1), (8, 8), (12, 4), (6, 1), (64, 1)):
        for T in (1, 2, 63, 64, 65, 127, 128, 129, 200, 333, 1024, 4096, 131072):
            for B in (1, 2, 3, 7, 40, 150, 1000):
                s = split(hd, B, H, KVH, T)
                assert s in (1, 2, 4)
                assert s <= -(-T // (128 if hd == 64 else 64)) * (H // KVH)
                if B * KVH * -(-T // 128) >= 2 * 148:
                    assert s == 1
