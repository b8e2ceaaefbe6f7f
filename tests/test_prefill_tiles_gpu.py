"""Packed prompt experts at the row counts where a 128-row tile's image changes its length (whole groups of eight rows, one more,
one less, one row, two tiles), at one and several chunks of either product, and with an output that is only 16-byte aligned; and at
the row counts where the short-prompt route's passes fill; and with experts that another device holds, whose rows stay as they are.
Bound 7e-4: four times the four-term FP4 error of a row (1.8e-4)."""
import ctypes as C

import numpy as np
import pytest
import torch

from basalt_b200 import capi, moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_experts_gpu import dev

pytestmark = pytest.mark.gpu


TILES = [1, 0, 7, 8, 9, 127, 128, 129, 0, 260]                                    # 67 rows an expert: tiles
SHORT16 = [0, 1, 8, 9, 15, 16, 17, 0, 130, 32, 33, 0, 0, 2, 0, 0]                # 16 an expert: the decode stream, passes of 16
SHORT8 = [0, 1, 7, 8, 9, 0, 17, 0, 0, 0, 0, 0, 0, 1, 0, 0]                       # 3 an expert: passes of 8


def run(H, I, shift, counts, held_elsewhere=(), n_held=None):
    """n_held: through the entry that is told the number of experts held here, whose scratch is exact"""
    rng = np.random.default_rng(H * 3 + I)
    E = len(counts)
    Lo, blobs = make_expert_blobs(rng, min(E, 10), O.T_NVFP4, O.T_NVFP4, H, I)
    L = moe.native_expert_layout(O.T_NVFP4, O.T_NVFP4, H, I)
    packed = moe.pack_experts(L, dev(stack_blobs(blobs)))
    n, T = sum(counts), 300
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    src = rng.integers(0, T, n).astype(np.int32)
    tiles = np.array([(e, off[e] + 128 * i) for e in range(E) for i in range((counts[e] + 127) // 128)], np.int32)
    x = rng.standard_normal((T, H)).astype(np.float32)
    table = packed.data_ptr() + torch.arange(E, dtype=torch.int64, device="cuda") % len(blobs) * packed.shape[1]
    table[list(held_elsewhere)] = 0
    lb = capi.lib()
    size = (lb.bsx_experts_prefill_packed_scratch_bytes(C.byref(L), T, n) if n_held is None
            else lb.bsx_experts_prefill_packed_held_scratch_bytes(C.byref(L), T, n, E, n_held))
    scratch = torch.full((size + 4096,), 0xFF, dtype=torch.uint8, device="cuda")
    raw = torch.full((n * H * 4 + 256,), 0xFF, dtype=torch.uint8, device="cuda")
    dm = raw[shift:shift + n * H * 4].view(torch.float32).view(n, H)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    o, s, t, nt, xd = dev(off), dev(src), dev(tiles), dev(np.array([len(tiles)], np.int32)), dev(x)
    stream = moe._stream(None)
    torch.cuda.synchronize()
    for _ in range(2):          # again over the scratch that the first call left
        args = (C.byref(L), table.data_ptr(), o.data_ptr(), s.data_ptr(), t.data_ptr(), nt.data_ptr(), len(tiles), n, xd.data_ptr(), capi.X_F32, T, E)
        rest = (scratch.data_ptr(), dm.data_ptr(), status.data_ptr(), stream)
        capi.check("prefill packed", lb.bsx_experts_prefill_packed(*args, *rest) if n_held is None else lb.bsx_experts_prefill_packed_held(*args, n_held, *rest))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    got = dm.cpu().numpy()
    assert (raw[:shift] == 0xFF).all() and (raw[shift + n * H * 4:] == 0xFF).all() and (scratch[size:] == 0xFF).all()
    for e in range(E):
        rows = got[off[e]:off[e + 1]]
        if e in held_elsewhere:
            assert (rows.view(np.uint32) == 0xFFFFFFFF).all(), e
        elif counts[e]:
            want = O.expert_forward(Lo, blobs[e % len(blobs)], x[src[off[e]:off[e + 1]]], dtype=np.float64)
            assert rel_l2(rows, want) < 7e-4, (e, counts[e], rel_l2(rows, want))


@pytest.mark.parametrize("H,I,shift,counts", [(256, 256, 0, TILES), (512, 512, 16, TILES), (768, 768, 0, TILES), (256, 1024, 16, TILES), (2048, 512, 0, TILES),
                                              (256, 256, 16, SHORT16), (2048, 512, 0, SHORT16), (768, 1280, 0, SHORT16), (512, 512, 0, SHORT8), (768, 768, 16, SHORT8)])
def test_tile_row_counts(lib, cuda, H, I, shift, counts):
    run(H, I, shift, counts)


MANY = [130, 500, 257] * 17                                                       # more tiles than an SM each


@pytest.mark.parametrize("H,I,counts,away", [(256, 256, TILES, (0, 4, 9)), (512, 512, TILES, (9,)), (768, 768, TILES, (0, 1, 2, 3)), (256, 512, MANY, range(0, 51, 3)),
                                             (256, 768, MANY, range(1, 51, 2)), (512, 512, SHORT16, (1, 8, 13)), (768, 2304, SHORT16, (8, 9)),
                                             (512, 256, SHORT8, (1, 6, 13)), (768, 768, SHORT8, (4,)), (256, 256, SHORT8, range(16)), (256, 256, TILES, range(10))])
def test_experts_held_elsewhere(lib, cuda, H, I, counts, away):
    run(H, I, 0, counts, tuple(away))


@pytest.mark.parametrize("H,I,counts,here", [(256, 256, TILES, (9,)), (512, 768, TILES, (9,)), (256, 512, TILES, (7, 9)), (512, 256, TILES, range(10)), (256, 768, MANY, range(34, 51)),
                                             (256, 512, MANY, (50,)), (256, 256, MANY, range(51)), (512, 512, SHORT16, (8,)), (768, 768, SHORT8, (6, 8)), (256, 256, [49], (0,)),
                                             (256, 512, [1, 120], (1,))])
def test_rounds_over_the_room_of_an_even_share(lib, cuda, H, I, counts, here):
    """rows that crowd onto the experts held here, more than twice an even share: the exact scratch for these few holds all their images"""
    run(H, I, 0, counts, tuple(e for e in range(len(counts)) if e not in here), len(tuple(here)))


# short calls by their average whose rows crowd onto few experts: full tiles and remainders above and below the 65 rows from which a
# tile stays one, over enough items that the call takes them (22 tiles x 6 or more), with passes of 16 and of 8 beside them
CROWD = [1000, 3, 0, 1000, 64, 65, 0, 700] + [0] * 55 + [9]


@pytest.mark.parametrize("H,I,shift,counts,away", [(256, 768, 0, CROWD, ()), (512, 1280, 16, CROWD, ()), (768, 2304, 0, CROWD, (1, 4)), (2048, 768, 0, CROWD, ()),
                                                   (256, 512, 16, CROWD * 2, ()), (512, 256, 0, CROWD * 5, (0, 64)), (256, 768, 0, CROWD + [0] * 700, ()),
                                                   (256, 768, 0, CROWD, (0, 3, 7))])
def test_crowded_short_calls(lib, cuda, H, I, shift, counts, away):
    run(H, I, shift, counts, away)
    run(H, I, shift, counts, away, len(counts))


# 34 rows an expert: tiles whose SwiGLU rows are gathered from row images
MID = [40, 1, 16, 17, 33, 129, 8, 64, 0, 31]
MID256 = [40, 1, 16, 17, 33, 129, 8, 64, 0, 120]                                 # 43 an expert: n_ff 256 is short up to 38


@pytest.mark.parametrize("H,I,shift,counts,away", [(256, 256, 0, MID, ()), (768, 512, 16, MID, ()), (512, 1280, 0, MID, (0, 5)), (2048, 2304, 0, MID, ()), (256, 512, 0, MID * 12, ()),
                                                   (768, 256, 0, TILES * 12, ()), (1280, 768, 0, TILES, (1, 9)), (256, 256, 0, MID256, ()), (2048, 256, 16, MID256 * 12, (3,))])
def test_tiles_of_gathered_rows(lib, cuda, H, I, shift, counts, away):
    """Every number of columns modulo 16 on either side of a pair's halves, one and two accumulators an item, few and many items a pair."""
    run(H, I, shift, counts, away)
    run(H, I, shift, counts, away, len(counts))
