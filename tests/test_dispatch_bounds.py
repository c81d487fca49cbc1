"""Bounds of the batch kernels' dispatch rules, called in the built library without a device."""
from __future__ import annotations

import ctypes

import pytest

UNIT_BYTES = {1: 144, 5: 272, 6: 84, 7: 110, 8: 144, 9: 176, 10: 210, 15: 66, 20: 54}      # Q4_0 Q8_0 Q2_K Q3_K Q4_K Q5_K Q6_K IQ2_XXS TQ1_0


class TileArgs(ctypes.Structure):               # weft::TileArgs of csrc/kernels.h
    _fields_ = [("fmt", ctypes.c_int)] + [(name, ctypes.c_void_p) for name in ("w", "x", "xq", "grid", "signs", "powers", "y")] + \
               [(name, ctypes.c_longlong) for name in ("n", "k", "m", "ldy")] + [("most_blocks", ctypes.c_int)]


def library():
    from weft_b200.build import ensure_built

    return ctypes.CDLL(str(ensure_built()))


@pytest.fixture(scope="module")
def tile_supported():
    rule = library()["_ZN4weft14tile_supportedERKNS_8TileArgsE"]
    rule.restype, rule.argtypes = ctypes.c_bool, [ctypes.POINTER(TileArgs)]
    return lambda fmt, m, n, k, w=1 << 20: rule(TileArgs(fmt, w, 1, 1, 1, 1, 1, 1, n, k, m, n))


@pytest.mark.parametrize("fmt", UNIT_BYTES)
def test_tile_rows_keep_to_32_bit_offsets(tile_supported, fmt):
    """A warp reaches its 32 rows and the 16-byte window around the last record of each by 32-bit offsets."""
    assert tile_supported(fmt, 3, 64, 256 * 1024)
    for blocks in sorted({1 << shift for shift in range(24)} | {(1 << 32) // 32 // UNIT_BYTES[fmt] + step for step in (-2, -1, 0, 1)}):
        fits = 32 * blocks * UNIT_BYTES[fmt] + 32 <= 1 << 32
        assert fits or not tile_supported(fmt, 3, 64, 256 * blocks), blocks
    assert tile_supported(fmt, 3, 64, 256 * min(1 << 20, (1 << 32) // 32 // UNIT_BYTES[fmt] - 1))
    assert not tile_supported(fmt, 3, 64, 256 * ((1 << 20) + 1))


@pytest.mark.parametrize("fmt", UNIT_BYTES)
def test_small_batches_go_by_token_rows(tile_supported, fmt):
    """Up to a number of products, except rows too long for some GEMV, and Q4_K up to 2048 results."""
    line = {6: 8.4e6, 15: 8.4e6, 20: 8.4e6, 5: 2.5e6}.get(fmt, 4.2e6)
    for m, n, k in [(3, 1, 256), (3, 1, 16384), (8, 256, 1024), (8, 257, 1024), (4, 512, 2048), (16, 128, 2048), (32, 64, 2048), (3, 3000, 512)]:
        assert tile_supported(fmt, m, n, k) == (m * n * k > line or (fmt == 8 and m * n > 2048)), (m, n, k)
    assert tile_supported(fmt, 3, 1, 16640)


def test_tile_sizes_that_are_left_to_others(tile_supported):
    assert not tile_supported(8, 2, 64, 4096) and not tile_supported(8, 3, 64, 4096 + 32) and not tile_supported(8, 3, 64, 4096, w=(1 << 20) + 8)


@pytest.fixture(scope="module")
def pair_supported():
    rule = library()["_ZN4weft14pair_supportedERKNS_8TileArgsEi"]
    rule.restype, rule.argtypes = ctypes.c_bool, [ctypes.POINTER(TileArgs), ctypes.c_int]
    return lambda fmt, m, n, k, w=1 << 20, sms=148: rule(TileArgs(fmt, w, 1, 1, 1, 1, 1, 1, n, k, m, n), sms)


PAIR_FORMATS = [1, 5, 8, 9, 10, 20]


@pytest.mark.parametrize("fmt", PAIR_FORMATS)
def test_pairs_take_whole_aligned_matrices(pair_supported, fmt):
    """Larger batches of whole 256-element blocks in a 16-byte aligned matrix; sums of a block's index stay in 32 bits."""
    assert pair_supported(fmt, 512, 14336, 4096)
    assert not pair_supported(fmt, 512, 14336, 4096 + 32) and not pair_supported(fmt, 512, 14336, 4096, w=(1 << 20) + 8)
    assert not pair_supported(fmt, 32, 14336, 4096) and not pair_supported(fmt, 512, 1024, 1024)
    assert not pair_supported(fmt, 1 << 19, 1 << 20, 4096)
    for m, n, k in [(1 << 20, 4096, 2048), ((1 << 20) + 3, 5, 2048), (129, 9, (1 << 22) + 2048)]:
        assert pair_supported(fmt, m, n, k) == (fmt == 20)                 # the only kernel for them, of this format alone
    assert not pair_supported(fmt, 1 << 30, 8, 2048) and not pair_supported(fmt, 4096, 5, 1 << 20)


@pytest.mark.parametrize("fmt", [1, 5])
def test_pair_plans_are_made_for_the_devices_sms(pair_supported, fmt):
    """With half a tile a pair and more, a third of the SMs takes three times as long, where the register tiles' estimate stays."""
    assert pair_supported(fmt, 128, 4096, 4096) and not pair_supported(fmt, 128, 4096, 4096, sms=48)


@pytest.mark.parametrize("fmt, m, n, k, pairs", [(5, 128, 4096, 4096, True), (5, 160, 4096, 4096, False), (5, 455, 4689, 768, False), (5, 181, 11200, 768, False),
                                                 (5, 512, 14336, 4096, True), (1, 128, 4096, 4096, True), (1, 177, 7387, 1280, False), (1, 317, 14656, 512, False),
                                                 (1, 570, 8000, 512, False), (1, 512, 4096, 14336, True), (20, 50, 4722, 5888, False), (20, 40, 8192, 8192, False),
                                                 (20, 38, 8512, 5376, False), (20, 40, 14336, 4096, True), (20, 384, 1024, 4096, True), (20, 512, 28672, 8192, True),
                                                 (9, 40, 8192, 8192, False), (9, 40, 14336, 4096, True)])
def test_pairs_and_register_tiles_by_what_was_measured(pair_supported, fmt, m, n, k, pairs):
    """Sizes at which one of the two is quicker by 5 % and more."""
    assert pair_supported(fmt, m, n, k) == pairs
