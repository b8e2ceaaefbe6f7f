"""What the packed prompt call asks its caller to allocate: the exact size for a number of experts never exceeds the one that covers any
number, short calls hold no tile images, and long ones the images of the SwiGLU rows alone, as tiles (a rank that holds an eighth of the
experts too: its call may get every row)."""
import ctypes as C
import random

import pytest

from basalt_b200 import capi, moe
from oracle import oracle as O


def sizes(H, I, tokens, rows, experts, held):
    L = moe.native_expert_layout(O.T_NVFP4, O.T_NVFP4, H, I)
    lb = capi.lib()
    return (lb.bsx_experts_prefill_packed_scratch_bytes(C.byref(L), tokens, rows),
            lb.bsx_experts_prefill_packed_held_scratch_bytes(C.byref(L), tokens, rows, experts, held))


def test_any_number_of_experts_is_covered(lib):
    rng = random.Random(1)
    for _ in range(3000):
        T, k, E = int(2 ** rng.uniform(0, 17)), rng.randint(1, 12), rng.randint(1, 1100)
        any_number, exact = sizes(256 * rng.randint(1, 28), 256 * rng.randint(1, 9), T, T * k, E, E)
        assert 0 < exact <= any_number, (T, k, E)


@pytest.mark.parametrize("T", [65, 256, 1300])
def test_short_calls_hold_rows_not_images_of_tiles(lib, T):
    H, I, rows = 7168, 2048, 9 * T
    _, exact = sizes(H, I, T, rows, 257, 257)
    row_buffers = T * (2.25 * H + 4) + rows * (4 * I + 2.25 * I + 4)          # FP4 terms of x, fp32 h and its FP4 terms
    lists = (rows + 1025) * 64 + 128 * I * 4                                  # pass and tile records; the rows past the last tile
    assert exact <= row_buffers + lists + 16 * 256


def test_long_call_and_a_rank_with_an_eighth(lib):
    H, I, T, k, E = 7168, 2048, 8192, 8, 256
    rows = 8 * T * k
    _, whole = sizes(H, I, 8 * T, rows, E, E)
    _, eighth = sizes(H, I, 8 * T, rows, E, E // 8)
    fixed = 8 * T * (2.25 * H + 4) + (rows + 128) * (4 * I + 8)                # FP4 terms of x, fp32 h
    images = 2.25 * I                                                          # of a SwiGLU row; a tile's: up to 24 rows more than its rows
    lists = (rows // 128 + E) * 32 + 16 * 256
    assert whole <= fixed + (rows + 24 * (rows // 128 + E)) * images + lists
    assert eighth <= fixed + (rows + 24 * (rows // 128 + E // 8)) * images + lists
    assert sizes(H, I, T, T, 8, 9)[1] == 0 and sizes(H, I, T, T, 0, 0)[1] == 0


@pytest.mark.parametrize("I,most", [(256, 38), (512, 29), (2304, 29)])
def test_rows_an_expert_up_to_which_a_call_is_short(lib, I, most):
    """A short call's scratch has pass records and few tile records, a longer one's tile records alone."""
    H, E = 2048, 64
    up = lambda n: (n + 255) // 256 * 256

    def size(T, rows, recs, passes):
        return sum(map(up, (T * 2 * H, T * H // 4, T * 4, (rows + 128) * I * 4, rows * 2 * I, rows * I // 4, (rows + 128) * 4, recs * 32, 12, passes * 16, 4)))
    for per, short in ((most, True), (most + 1, False)):
        rows = per * E
        tiles = rows // 128 + E
        want = size(rows, rows, min(tiles, rows // 65 + 1), rows // 8 + tiles) if short else size(rows, rows, tiles, 0)
        assert sizes(H, I, rows, rows, E, E)[1] == want, (per, want)


def test_scratch_of_the_largest_call_covers_the_smaller(lib):
    """around the numbers of rows where the route changes, at each of which the buffers differ"""
    rng = random.Random(3)
    for _ in range(150):
        H, I, E, k = 256 * rng.randint(1, 28), 256 * rng.choice([1, 1, 2, 3, 9]), rng.choice([1, 3, 8, 64, 257, 513, 1025]), rng.randint(1, 10)
        held = rng.choice([E, max(1, E // 8)])
        last = (0, 0)
        for T in sorted({max(1, r * E // k + d) for r in (1, 4, 28, 29, 30, 37, 38, 39, 48, 49, 60) for d in (-1, 0, 1)}):
            now = sizes(H, I, T, T * k, E, held)
            assert now[0] >= last[0] and now[1] >= last[1], (H, I, E, k, held, T)
            last = now
