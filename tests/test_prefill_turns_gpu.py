"""NVFP4 prompt rows in place whose contraction has an odd number of 128-column pairs: the two decoder groups take turns from one work item
to the next, over several items a CTA; with one pair a group has no part in every other item.  Bound 9e-4: four times the fp16 rounding of
weights and SwiGLU rows (2.1e-4 measured)."""
import numpy as np
import pytest
import torch

from basalt_b200 import moe
from oracle import oracle as O
from tests.helpers import make_expert_blobs, rel_l2, stack_blobs
from tests.test_prefill_gpu import run_prefill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,T,E", [(2560, 320, 100, 60), (2560, 64, 100, 60), (2560, 640, 100, 40), (2560, 256, 100, 40)])
def test_odd_pair_counts(lib, cuda, H, I, T, E):
    rng = np.random.default_rng(H + I)
    Lo, blobs = make_expert_blobs(rng, E, O.T_NVFP4, O.T_NVFP4, H, I)
    L = moe.native_expert_layout(O.T_NVFP4, O.T_NVFP4, H, I)
    ids = rng.integers(0, E, (T, 1)).astype(np.int32)
    xd = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).cuda().bfloat16()
    x = xd.float().cpu().numpy()
    dm, cnt, off, src, _ = run_prefill(L, torch.from_numpy(stack_blobs(blobs)).cuda(), ids, 1, E, xd)
    for e in range(E):
        if cnt[e]:
            want = O.expert_forward(Lo, blobs[e], x[src[off[e]:off[e + 1]]], dtype=np.float64)
            assert rel_l2(dm[off[e]:off[e + 1]], want) < 9e-4, (e, rel_l2(dm[off[e]:off[e + 1]], want))
